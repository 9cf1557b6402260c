// Correctly rounded FP64 division through a reciprocal, shared by the lattice
// kernels (the velocity of every site) and the FEM band solve.
#pragma once
#include <cuda_runtime.h>

#include <cstring>

namespace life {

// the bits of a double (device intrinsic, or a copy on the host)
__host__ __device__ __forceinline__ unsigned long long div_bits(double x) {
#ifdef __CUDA_ARCH__
    return (unsigned long long)__double_as_longlong(x);
#else
    unsigned long long u;
    std::memcpy(&u, &x, sizeof u);
    return u;
#endif
}

// a / b correctly rounded (round to nearest), given y = RN(1/b): Markstein's
// method (P. Markstein, IBM J. Res. Dev. 34(1), 1990; Muller et al.,
// Handbook of Floating-Point Arithmetic, "Markstein's theorem"): q0 = RN(a y)
// is within 1.5 ulp of a/b, one correction q1 = RN(q0 + RN(a - b q0) y)
// brings it within one ulp, and then the residual a - b q1 is exact and
// RN(q1 + (a - b q1) y) = RN(a/b). The theorem needs the intermediates in the
// normal range, so operands outside a safe exponent window (tested on the
// bits, with integer operations) take the hardware division.
// life_selftest_division checks this function against a / b on the device,
// and the host build of the same function is checked against IEEE division
// by the CPU tests.
__host__ __device__ __forceinline__ double div_rn_recip(double a, double b, double y) {
    const unsigned long long ba = div_bits(a);
    const unsigned long long bb = div_bits(b);
    const int ea = (int)(ba >> 52) & 0x7ff, eb = (int)(bb >> 52) & 0x7ff;
    // a zero numerator runs the same steps (every intermediate is a zero) and
    // then takes q0 = a * y, the signed zero a / b (y has the sign of b): the
    // cost of a site does not depend on its velocity being zero
    const bool a_zero = (ba << 1) == 0ull;
    const bool a_ok = a_zero || (ea > 200 && ea < 1800 && ea - eb > -700 && ea - eb < 700);
    const bool b_ok = eb > 200 && eb < 1800;
    if (!(a_ok && b_ok)) return a / b;
    const double q0 = a * y;
    const double r0 = fma(-b, q0, a);
    const double q1 = fma(r0, y, q0);
    const double r1 = fma(-b, q1, a);
    const double q = fma(r1, y, q1);
    return a_zero ? q0 : q;
}

#ifdef __CUDACC__
// Reciprocal and quotient with a short latency, for chains of a few lanes: an
// FP64 instruction takes 64 cycles however few lanes need it, and a correctly
// rounded reciprocal of them 351 cycles; the integer steps below take 174.
//
// recip64: X near 2^64 / s, s in (1, 2) the significand of b (a multiple of
// 2^-52), from the hardware's FP32 approximation y of 1/s (of s cut to 24 bits):
// with the residual e = 1 - s y, |e| < 2^-21, X = 2^64 y (1 + e + e^2). The
// cut terms are e^3 < 2^-63 and a few units of the integer arithmetic: X is
// within 8 of 2^64 / s. Returns whether b is normal, not a power of two, and X
// lies in range. (A published scheme: Newton's reciprocal iteration with its
// second-order term.)
__device__ __forceinline__ bool recip64(double b, unsigned long long& X) {
    const unsigned long long u = div_bits(b);
    const unsigned h = (unsigned)(u >> 32), e = (h >> 20) & 0x7ffu;
    const unsigned long long B = (((unsigned long long)((h & 0xfffffu) | 0x100000u) << 32) | (unsigned)u) << 11;
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(0x3f800000u | ((unsigned)(B >> 40) & 0x7fffffu))));
    const unsigned yb = __float_as_uint(y), m = (yb & 0x7fffffu) | 0x800000u;  // y in units of 2^-24
    // R = 2^63 e, rounded down: 2^87 - B m in units of 2^24
    const unsigned long long lo = (unsigned long long)(unsigned)B * m;
    const unsigned long long T = (unsigned long long)(unsigned)(B >> 32) * m + (lo >> 32);
    const long long R = ((long long)((1ull << 55) - T) << 8) - (long long)((unsigned)lo >> 24);
    const int es = (int)(R >> 14);
    const long long S = R + (((long long)es * es) >> 35);  // 2^63 (e + e^2)
    X = ((unsigned long long)m << 40) +
        (unsigned long long)((long long)m * (S >> 23) + (((long long)m * (long long)(S & 0x7fffff)) >> 23));
    return (yb >> 23) == 126u && e - 200u < 1600u && (long long)X < 0;
}

// RN(1/b) from recip64's X; false where X does not decide the rounding.
__device__ __forceinline__ bool recip_round(double b, unsigned long long X, double& r) {
    const unsigned h = (unsigned)(div_bits(b) >> 32), e = (h >> 20) & 0x7ffu;
    const unsigned long long q = ((X + 0x400u) >> 11) + ((unsigned long long)(2044u - e) << 52);
    r = __longlong_as_double((long long)(q | ((unsigned long long)(h & 0x80000000u) << 32)));
    return ((unsigned)X & 0x7ffu) - 0x3f0u > 0x20u;
}

// RN(a/b) from recip64's X of b; false where it does not decide the rounding,
// or a is zero or outside div_rn_recip's window (b is inside it).
__device__ __forceinline__ bool quotient_round(double a, double b, unsigned long long X, double& q) {
    const unsigned long long ua = div_bits(a);
    const unsigned ah = (unsigned)(ua >> 32), bh = (unsigned)(div_bits(b) >> 32);
    const int ea = (int)((ah >> 20) & 0x7ffu), eb = (int)((bh >> 20) & 0x7ffu);
    const unsigned long long A = (((unsigned long long)((ah & 0xfffffu) | 0x100000u) << 32) | (unsigned)ua) << 11;
    unsigned long long p = __umul64hi(A, X);  // 2^63 a'/b', a' and b' the significands, within 10
    const unsigned up = (unsigned)(p >> 63) ^ 1u;
    p <<= up;
    // (equal significands: p ends just below 2^64 and the rounding would carry
    // out; not decided here)
    const bool fits = (long long)(p + 0x400u) < 0;
    const unsigned long long r = ((p + 0x400u) >> 11) + ((unsigned long long)(unsigned)(ea - eb + 1022 - (int)up) << 52);
    q = __longlong_as_double((long long)(r | ((unsigned long long)((ah ^ bh) & 0x80000000u) << 32)));
    return fits && ((unsigned)p & 0x7ffu) - 0x3e0u > 0x40u && (unsigned)(ea - 200) < 1600u && (unsigned)(ea - eb + 699) < 1399u;
}
#endif

}  // namespace life
