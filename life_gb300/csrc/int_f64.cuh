// FP64 arithmetic on the integer units, rounded as IEEE round to nearest even.
//
// The SM's FP64 unit takes 64 cycles of a sub-partition per warp instruction
// (2 lanes per cycle and SM) and the FP64 lattice kernels keep it busy all the
// time while more than 90 % of the issue slots are free. A product formed from
// integer instructions (a 53 x 53 bit multiplication of the significands, one
// normalising shift, rounding) takes some 50 cycles of issue slots and none
// of the FP64 unit, and runs beside it at no cost to it (measured: a loop of
// four FP64 additions takes 307 cycles alone and with two integer additions
// beside them, 388 with two additions and two products).
//
// The operands are zero or normal and the product is zero or normal: the
// callers check the range of a site's values once, not per operation.
#pragma once
#include <cuda_runtime.h>

#include <cstring>

#include "div_rn.cuh"

namespace life {

__host__ __device__ __forceinline__ double bits_double(unsigned long long u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double d;
    std::memcpy(&d, &u, sizeof d);
    return d;
#endif
}

// a * b.
//   kNonZero   neither operand is zero
//   kZeroA     a may be zero (the product is then +0, whatever the signs)
//   kZeroAny   either may be zero (a zero product has its sign)
enum { kNonZero, kZeroA, kZeroAny };
template <int ZERO = kZeroA>
__host__ __device__ __forceinline__ double mul_int(double a, double b) {
    const unsigned long long ua = div_bits(a), ub = div_bits(b);
    const unsigned ah = (unsigned)(ua >> 32), bh = (unsigned)(ub >> 32);
    // 53-bit significands; b's shifted up to bit 63, so the product's high 64
    // bits hold the result's significand with its leading bit at 51 or 52 and
    // the low 64 bits the fraction that is rounded off
    const unsigned a1 = (ah & 0xfffffu) | 0x100000u, b1s = (bh & 0xfffffu) | 0x100000u;
    const unsigned a0 = (unsigned)ua;
    const unsigned long long mb = (((unsigned long long)b1s << 32) | (unsigned)ub) << 11;
    const unsigned b1 = (unsigned)(mb >> 32), b0 = (unsigned)mb;
    // ah - a1 is the sign and the exponent less one; adding the two adds the
    // exponents and multiplies the signs (the carry out of bit 31 is lost)
    const unsigned e = (ah - a1) + (bh - b1s) - (1021u << 20);
    unsigned r1, r0;
    const unsigned long long p00 = (unsigned long long)a0 * b0;
    const unsigned long long t = (unsigned long long)a0 * b1 + (p00 >> 32);
    const unsigned long long u = (unsigned long long)a1 * b0 + (unsigned)t;
    const unsigned long long hi = (unsigned long long)a1 * b1 + (t >> 32) + (u >> 32);
    const unsigned long long lo = (u << 32) | (unsigned)p00;
    const unsigned lead = (unsigned)(hi >> 32) & 0x100000u;  // leading bit at 52
    const unsigned up = lead ? 0u : 1u;
#ifdef __CUDA_ARCH__
    const unsigned lo1 = (unsigned)(lo >> 32), lo0 = (unsigned)lo, hi1 = (unsigned)(hi >> 32), hi0 = (unsigned)hi;
    const unsigned f0 = lo0 << up, f1 = __funnelshift_l(lo0, lo1, up);
    const unsigned s0 = __funnelshift_l(lo1, hi0, up), s1 = __funnelshift_l(hi0, hi1, up);
    const unsigned odd = s0 & 1u;
    // round to nearest even: add half less one, plus one for an odd significand
    asm("{\n\t.reg .u32 t;\n\t"
        "add.cc.u32 t, %2, %3;\n\t"
        "addc.cc.u32 t, %4, %5;\n\t"
        "addc.cc.u32 %0, %6, 0;\n\t"
        "addc.u32 %1, %7, %8;\n\t}"
        : "=r"(r0), "=r"(r1)
        : "r"(f0), "r"(odd - 1u), "r"(f1), "r"(odd + 0x7fffffffu), "r"(s0), "r"(s1), "r"(e + lead - 0x100000u));
#else
    const unsigned long long sig = (hi << up) | (up ? lo >> 63 : 0), frac = lo << up;
    const unsigned long long half = 0x7fffffffffffffffull + (sig & 1u);
    const unsigned long long r = sig + (frac + half < frac ? 1u : 0u) + ((unsigned long long)(e + lead - 0x100000u) << 32);
    r1 = (unsigned)(r >> 32);
    r0 = (unsigned)r;
#endif
    if (ZERO == kZeroA && (ah & 0x7ff00000u) == 0u) r1 = r0 = 0u;
    if (ZERO == kZeroAny && ((ah & 0x7ff00000u) == 0u || (bh & 0x7ff00000u) == 0u)) {
        r1 = (ah ^ bh) & 0x80000000u;
        r0 = 0u;
    }
    return bits_double(((unsigned long long)r1 << 32) | r0);
}

__host__ __device__ __forceinline__ int leading_zeros(unsigned long long x) {
#ifdef __CUDA_ARCH__
    return __clzll((long long)x);
#else
    return x ? __builtin_clzll(x) : 64;
#endif
}
// shifts whose counts may pass 63 (the result is then 0)
__host__ __device__ __forceinline__ unsigned long long shift_right(unsigned long long x, unsigned d) {
#ifdef __CUDA_ARCH__
    unsigned long long r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(d));
    return r;
#else
    return d > 63 ? 0 : x >> d;
#endif
}
__host__ __device__ __forceinline__ unsigned long long shift_left(unsigned long long x, unsigned d) {
#ifdef __CUDA_ARCH__
    unsigned long long r;
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(d));
    return r;
#else
    return d > 63 ? 0 : x << d;
#endif
}

// 2^E + x for |x| < 2^E: fixed point with 2^E at bit 62. Bits of x below the
// unit (only where |x| < 2^(E-10), so the sum keeps its leading bit to within
// one place) fold into the lowest bit.
template <int E>
__host__ __device__ __forceinline__ double add_pow2_int(double x) {
    const unsigned long long u = div_bits(x);
    const unsigned h = (unsigned)(u >> 32);
    const unsigned long long m = (((unsigned long long)((h & 0xfffffu) | 0x100000u) << 32) | (unsigned)u) << 10;
    const unsigned d = (unsigned)(1023 + E) - ((h >> 20) & 0x7ffu);
    unsigned long long a = shift_right(m, d);
    if (shift_left(a, d) != m) a |= 1;
    unsigned long long s = (1ull << 62) + ((int)h < 0 ? 0ull - a : a);
    const int lz = leading_zeros(s);
    s = shift_left(s, (unsigned)(lz - 1));
    s += 0x1ff + ((unsigned)(s >> 10) & 1u);
    return bits_double((s >> 10) + ((unsigned long long)(unsigned)(1023 + E - lz) << 52));
}

// The density and momentum sums of moment_sums() for populations in [2^-8, 1):
// every population is a multiple of 2^-60, so the running sums are 64-bit
// integers in that unit, rounded to 53 significant bits after each addition.
// The density may reach 9, which needs all 64 bits, unsigned; the momenta stay
// below 3 in magnitude. About 25 issue cycles an addition.
__host__ __device__ __forceinline__ long long round53(long long s) {
    const unsigned long long z = (unsigned long long)(s ^ (s >> 63));
    int p = 11 - leading_zeros(z);  // bits below the 53 significant ones
    p = p > 0 ? p : 0;
    const unsigned lo = (unsigned)s, below = (1u << p) - 1u;
    s += (below >> 1) + ((lo >> p) & (p > 0 ? 1u : 0u));
    return s & ~(long long)below;
}
__host__ __device__ __forceinline__ unsigned long long unit60_bits(unsigned long long a) {  // a 2^-60, a of 53 bits, not 0
    const int lz = leading_zeros(a);
    return (shift_left(a, (unsigned)lz) >> 11) + ((unsigned long long)(unsigned)(1025 - lz) << 52);
}
__host__ __device__ __forceinline__ double unit60(long long s) {  // s 2^-60, |s| of 53 bits at most
    const unsigned long long a = s < 0 ? 0ull - (unsigned long long)s : (unsigned long long)s;
    return bits_double(a == 0 ? 0ull : unit60_bits(a) | ((unsigned long long)s & 0x8000000000000000ull));
}
__host__ __device__ __forceinline__ void moment_sums_int(const double f[9], double& r, double& mx, double& my) {
    long long x[9];
#pragma unroll
    for (int v = 0; v < 9; v++) {
        const unsigned long long u = div_bits(f[v]);
        const unsigned h = (unsigned)(u >> 32);
        const unsigned long long m = ((unsigned long long)((h & 0xfffffu) | 0x100000u) << 32) | (unsigned)u;
        x[v] = (long long)(m << ((h >> 20) - 1015u));
    }
    unsigned long long s = (unsigned long long)x[0];
#pragma unroll
    for (int v = 1; v < 9; v++) {
        s += (unsigned long long)x[v];  // at least 2^53: something to round every time
        const int p = 11 - leading_zeros(s);
        const unsigned below = (1u << p) - 1u;
        s += (below >> 1) + (((unsigned)s >> p) & 1u);
        s &= ~(unsigned long long)below;
    }
    r = bits_double(unit60_bits(s));
    mx = unit60(round53(round53(round53(round53(round53(x[1] - x[2]) + x[5]) - x[6]) + x[7]) - x[8]));
    my = unit60(round53(round53(round53(round53(round53(x[3] - x[4]) + x[5]) - x[6]) - x[7]) + x[8]));
}

// x 2^e for a non-zero x (the exponent field moved by e).
__host__ __device__ __forceinline__ double scale2_nz(double x, int e) {
    return bits_double(div_bits(x) + ((unsigned long long)(long long)e << 52));
}

}  // namespace life
