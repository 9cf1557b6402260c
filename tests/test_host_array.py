"""Which host arrays the export kernel may write to (``host_array.h``, compiled here
for the host): only those that one page-locked, device-writable range covers from
the first byte to the last. A range that ends inside the array, starts inside it,
is read-only or has no device address leaves the array to the staged copies."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "life_gb300", "csrc")

DRIVER = r"""
#include "host_array.h"
#include <cstdio>
#include <cstdlib>
int main(int argc, char** argv) {
    // locked writable start size device | pointer bytes align
    unsigned long long v[8];
    for (int k = 0; k < 8; k++) v[k] = strtoull(argv[k + 1], nullptr, 0);
    life::HostRange r;
    r.locked = v[0]; r.writable = v[1]; r.start = v[2]; r.size = v[3]; r.device = v[4];
    const void* p = reinterpret_cast<const void*>(static_cast<std::uintptr_t>(v[5]));
    printf("%d %llx\n", (int)life::host_range_covers(r, p, v[6]), (unsigned long long)life::kernel_target(r, p, v[6], v[7]));
    return 0;
}
"""

A, N = 0x7F0000010000, 1 << 20


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("host_array")
    src, exe = d / "host_array.cpp", d / "host_array"
    src.write_text(DRIVER)
    subprocess.run([cxx, "-O1", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return str(exe)


def ask(driver, locked=1, writable=1, start=A, size=N, device=A, p=A, nbytes=N, align=16):
    args = [locked, writable, start, size, device, p, nbytes, align]
    out = subprocess.run([driver] + [hex(int(a)) for a in args], capture_output=True, text=True, check=True).stdout.split()
    return bool(int(out[0])), int(out[1], 16)


@pytest.mark.parametrize("kw,covers,target", [
    (dict(), True, A),                                                  # the whole array, exactly
    (dict(size=2 * N), True, A),                                        # more than the array
    (dict(p=A + 4096, nbytes=N - 4096, device=A + 4096), True, A + 4096),   # its tail, to the last byte
    (dict(size=N - 1), False, 0),                                       # one byte short
    (dict(size=N // 2), False, 0),                                      # only the first half registered
    (dict(size=4096), False, 0),                                        # only the first page
    (dict(p=A + 4096, device=A + 4096), False, 0),                      # runs out of the range
    (dict(start=A + 4096), False, 0),                                   # the range starts inside the array
    (dict(p=A + N, device=A + N, nbytes=8), False, 0),                  # just past the range
    (dict(nbytes=2 ** 64 - 16), False, 0),                              # (no wrap-around)
    (dict(locked=0), False, 0),
    (dict(writable=0), True, 0),                                        # registered read-only
    (dict(device=0), True, 0),
    (dict(device=0x200000000), True, 0x200000000),                      # another address on the device
    (dict(device=A + 8), True, 0),                                      # not aligned for pairs
    (dict(device=A + 8, align=8), True, A + 8),
])
def test_kernel_target(driver, kw, covers, target):
    assert ask(driver, **kw) == (covers, target)
