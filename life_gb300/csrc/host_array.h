// Which host arrays a kernel may write to.
#pragma once
#include <cstddef>
#include <cstdint>

namespace life {

// The allocation or registration that a host pointer belongs to, as the driver
// reports it: the address range it covers on the host, the device's address of
// the pointer, and whether the device may write there.
struct HostRange {
    bool locked = false;  // page-locked host memory
    bool writable = false;
    std::uintptr_t start = 0, device = 0;
    std::size_t size = 0;
};

// Whether [p, p + bytes) lies in the range, to its last byte: a registration
// may cover only the start of the array it was given.
inline bool host_range_covers(const HostRange& r, const void* p, std::size_t bytes) {
    const std::uintptr_t a = reinterpret_cast<std::uintptr_t>(p);
    return r.locked && a >= r.start && a - r.start <= r.size && bytes <= r.size - (a - r.start);
}

// The device's address of the array, if a kernel can write all of it in
// elements of `align` bytes; 0 otherwise (the array is then staged).
inline std::uintptr_t kernel_target(const HostRange& r, const void* p, std::size_t bytes, std::size_t align) {
    if (!host_range_covers(r, p, bytes) || !r.writable || r.device == 0 || r.device % align != 0) return 0;
    return r.device;
}

}  // namespace life
