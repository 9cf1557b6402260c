// Central-moments collision in FP64 (De Rosis 2019), the reference's
// CENTRAL_MOMENTS branch of GridClass::streamCollide.
#pragma once
#include "int_f64.cuh"
#include "lbm_device.cuh"

namespace life {

// Inverse central-moment transform (De Rosis 2019), term order as in the
// reference (src/Grid.cpp:109-223); FP64 parity depends on that order.
template <bool UNF>
__host__ __device__ __forceinline__ void collide_cm(const double f[9], double rho, double ux, double uy, double Fx, double Fy,
                           double omega, double cs, double fs[9]) {
    // the two sums start at their first term rather than at +0 (see
    // moment_sums: equal up to the sign of a zero, which pos_zero restores)
    double k4Pre, k5Pre;
#pragma unroll
    for (int v = 0; v < 9; v++) {
        double cx = cx_of(v) - ux;
        double cy = cy_of(v) - uy;
        const double t4 = f[v] * (LSQ(cx) - LSQ(cy)), t5 = f[v] * cx * cy;
        k4Pre = v == 0 ? t4 : k4Pre + t4;
        k5Pre = v == 0 ? t5 : k5Pre + t5;
    }
    k4Pre = pos_zero(k4Pre);
    k5Pre = pos_zero(k5Pre);
    const double k0 = rho;
    const double k1 = 0.5 * Fx;
    const double k2 = 0.5 * Fy;
    const double k3 = 2.0 * rho * LSQ(cs);
    const double k4 = (1.0 - omega) * k4Pre;
    const double k5 = (1.0 - omega) * k5Pre;
    const double k6 = 0.5 * Fy * LSQ(cs);
    const double k7 = 0.5 * Fx * LSQ(cs);
    const double k8 = rho * LQU(cs);
    const double X2 = LSQ(ux), Y2 = LSQ(uy);
    // The force moments k1, k2, k6, k7 are exact zeros when Fx = Fy = 0 (a
    // value the whole launch shares); their terms are then not formed, and
    // every other term is added in the reference's order.
    const bool forced = !UNF && (Fx != 0.0 || Fy != 0.0);
    {
        double a = (X2 * Y2 - X2 - Y2 + 1.0) * k0;
        if (forced) a = a + ((2.0 * ux * Y2 - 2.0 * ux) * k1);
        if (forced) a = a + ((2.0 * uy * X2 - 2.0 * uy) * k2);
        a = a + ((0.5 * X2 + 0.5 * Y2 - 1.0) * k3);
        a = a + ((0.5 * Y2 - 0.5 * X2) * k4);
        a = a + (4.0 * ux * uy * k5);
        if (forced) a = a + (2.0 * uy * k6);
        if (forced) a = a + (2.0 * ux * k7);
        a = a + (k8);
        fs[0] = a;
    }
    {
        double a = (0.5 * X2 - 0.5 * (X2 * Y2) - 0.5 * (ux * Y2) + 0.5 * ux) * k0;
        if (forced) a = a + ((ux - ux * Y2 - 0.5 * Y2 + 0.5) * k1);
        if (forced) a = a + ((-uy * X2 - uy * ux) * k2);
        a = a + ((-0.25 * X2 - 0.25 * ux - 0.25 * Y2 + 0.25) * k3);
        a = a + ((0.25 * X2 + 0.25 * ux - 0.25 * Y2 + 0.25) * k4);
        a = a + ((-uy - 2.0 * ux * uy) * k5);
        if (forced) a = a + ((-uy) * k6);
        if (forced) a = a + ((-ux - 0.5) * k7);
        a = a - (0.5 * k8);
        fs[1] = a;
    }
    {
        double a = (-0.5 * (X2 * Y2) + 0.5 * X2 + 0.5 * (ux * Y2) - 0.5 * ux) * k0;
        if (forced) a = a + ((ux - ux * Y2 + 0.5 * Y2 - 0.5) * k1);
        if (forced) a = a + ((-uy * X2 + uy * ux) * k2);
        a = a + ((-0.25 * X2 + 0.25 * ux - 0.25 * Y2 + 0.25) * k3);
        a = a + ((0.25 * X2 - 0.25 * ux - 0.25 * Y2 + 0.25) * k4);
        a = a + ((uy - 2.0 * ux * uy) * k5);
        if (forced) a = a + ((-uy) * k6);
        if (forced) a = a + ((0.5 - ux) * k7);
        a = a - (0.5 * k8);
        fs[2] = a;
    }
    {
        double a = (0.5 * Y2 - 0.5 * (X2 * uy) - 0.5 * (X2 * Y2) + 0.5 * uy) * k0;
        if (forced) a = a + ((-ux * Y2 - ux * uy) * k1);
        if (forced) a = a + ((uy - X2 * uy - 0.5 * X2 + 0.5) * k2);
        a = a + ((-0.25 * X2 - 0.25 * Y2 - 0.25 * uy + 0.25) * k3);
        a = a + ((0.25 * X2 - 0.25 * Y2 - 0.25 * uy - 0.25) * k4);
        a = a + ((-ux - 2.0 * ux * uy) * k5);
        if (forced) a = a + ((-uy - 0.5) * k6);
        if (forced) a = a + ((-ux) * k7);
        a = a - (0.5 * k8);
        fs[3] = a;
    }
    {
        double a = (-0.5 * (X2 * Y2) + 0.5 * (X2 * uy) + 0.5 * Y2 - 0.5 * uy) * k0;
        if (forced) a = a + ((-ux * Y2 + ux * uy) * k1);
        if (forced) a = a + ((uy - X2 * uy + 0.5 * X2 - 0.5) * k2);
        a = a + ((-0.25 * X2 - 0.25 * Y2 + 0.25 * uy + 0.25) * k3);
        a = a + ((0.25 * X2 - 0.25 * Y2 + 0.25 * uy - 0.25) * k4);
        a = a + ((ux - 2.0 * ux * uy) * k5);
        if (forced) a = a + ((0.5 - uy) * k6);
        if (forced) a = a + ((-ux) * k7);
        a = a - (0.5 * k8);
        fs[4] = a;
    }
    {
        double a = (0.25 * (X2 * Y2) + 0.25 * (X2 * uy) + 0.25 * (ux * Y2) + 0.25 * (ux * uy)) * k0;
        if (forced) a = a + ((0.25 * uy + 0.5 * (ux * uy) + 0.5 * (ux * Y2) + 0.25 * Y2) * k1);
        if (forced) a = a + ((0.25 * ux + 0.5 * (ux * uy) + 0.5 * (X2 * uy) + 0.25 * X2) * k2);
        a = a + ((0.125 * X2 + 0.125 * ux + 0.125 * Y2 + 0.125 * uy) * k3);
        a = a + ((-0.125 * X2 - 0.125 * ux + 0.125 * Y2 + 0.125 * uy) * k4);
        a = a + ((0.5 * ux + 0.5 * uy + ux * uy + 0.25) * k5);
        if (forced) a = a + ((0.5 * uy + 0.25) * k6);
        if (forced) a = a + ((0.5 * ux + 0.25) * k7);
        a = a + (0.25 * k8);
        fs[5] = a;
    }
    {
        double a = (0.25 * (X2 * Y2) - 0.25 * (X2 * uy) - 0.25 * (ux * Y2) + 0.25 * (ux * uy)) * k0;
        if (forced) a = a + ((0.25 * uy - 0.5 * (ux * uy) + 0.5 * (ux * Y2) - 0.25 * Y2) * k1);
        if (forced) a = a + ((0.25 * ux - 0.5 * (ux * uy) + 0.5 * (X2 * uy) - 0.25 * X2) * k2);
        a = a + ((0.125 * X2 - 0.125 * ux + 0.125 * Y2 - 0.125 * uy) * k3);
        a = a + ((-0.125 * X2 + 0.125 * ux + 0.125 * Y2 - 0.125 * uy) * k4);
        a = a + ((ux * uy - 0.5 * uy - 0.5 * ux + 0.25) * k5);
        if (forced) a = a + ((0.5 * uy - 0.25) * k6);
        if (forced) a = a + ((0.5 * ux - 0.25) * k7);
        a = a + (0.25 * k8);
        fs[6] = a;
    }
    {
        double a = (0.25 * (X2 * Y2) - 0.25 * (X2 * uy) + 0.25 * (ux * Y2) - 0.25 * (ux * uy)) * k0;
        if (forced) a = a + ((0.5 * (ux * Y2) - 0.5 * (ux * uy) - 0.25 * uy + 0.25 * Y2) * k1);
        if (forced) a = a + ((0.5 * (ux * uy) - 0.25 * ux + 0.5 * (X2 * uy) - 0.25 * X2) * k2);
        a = a + ((0.125 * X2 + 0.125 * ux + 0.125 * Y2 - 0.125 * uy) * k3);
        a = a + ((-0.125 * X2 - 0.125 * ux + 0.125 * Y2 - 0.125 * uy) * k4);
        a = a + ((0.5 * uy - 0.5 * ux + ux * uy - 0.25) * k5);
        if (forced) a = a + ((0.5 * uy - 0.25) * k6);
        if (forced) a = a + ((0.5 * ux + 0.25) * k7);
        a = a + (0.25 * k8);
        fs[7] = a;
    }
    {
        double a = (0.25 * (X2 * Y2) + 0.25 * (X2 * uy) - 0.25 * (ux * Y2) - 0.25 * (ux * uy)) * k0;
        if (forced) a = a + ((0.5 * (ux * uy) - 0.25 * uy + 0.5 * (ux * Y2) - 0.25 * Y2) * k1);
        if (forced) a = a + ((0.5 * (X2 * uy) - 0.5 * (ux * uy) - 0.25 * ux + 0.25 * X2) * k2);
        a = a + ((0.125 * X2 - 0.125 * ux + 0.125 * Y2 + 0.125 * uy) * k3);
        a = a + ((-0.125 * X2 + 0.125 * ux + 0.125 * Y2 + 0.125 * uy) * k4);
        a = a + ((0.5 * ux - 0.5 * uy + ux * uy - 0.25) * k5);
        if (forced) a = a + ((0.5 * uy + 0.25) * k6);
        if (forced) a = a + ((0.5 * ux - 0.25) * k7);
        a = a + (0.25 * k8);
        fs[8] = a;
    }
}

// ---- one population of the central-moment collision ----------------------
//
// collide_cm's expressions with their power-of-two coefficients taken out:
// scaling by a power of two commutes with round-to-nearest while nothing
// leaves the normal range, so (0.25 a + 0.25 b) k is 0.25 ((a + b) k), and
// every moment k enters as (poly) (scale k), the scaled moment formed once.
// Without the factors each polynomial is at most four terms, and the terms
// of all nine populations are the same few products with a sign, so ONE
// instruction stream serves any population: a warp whose lanes hold the nine
// populations of a site runs 20 FP64 instructions (36 with a force) where
// the nine written-out polynomials take about 220 (320). The sums keep the
// reference's order. cm_factored_ok() tells whether the values are in the
// range where the scalings are exact; otherwise the written-out form runs.
struct CmSite {
    double ux, uy;              // velocity
    double X2, Y2, XY, W;       // ux^2, uy^2, ux uy, 2 ux uy
    double X2Y2, uxY2, X2uy;
    double k0, k3, k4, k5, k8;  // moments after relaxation (k1, k2, k6, k7: force)
    double k1, k2, k6, k7;
};

// x with its sign flipped when the integer c is negative / multiplied by 2^e
// (the exponent field moved by e; x zero or well inside the normal range).
__host__ __device__ __forceinline__ double sgn_c(int c, double x) {
    return bits_double(div_bits(x) ^ ((unsigned long long)((unsigned)c & 0x80000000u) << 32));
}
__host__ __device__ __forceinline__ double scale2(double x, int e) {
    const unsigned long long u = div_bits(x);
    return (u << 1) == 0ull ? x : bits_double(u + ((unsigned long long)(long long)e << 52));
}

// Zero, or a magnitude in [2^lo, 2^hi).
__host__ __device__ __forceinline__ bool exp_within(double x, int lo, int hi) {
    const unsigned long long u = div_bits(x);
    const int e = (int)(u >> 52) & 0x7ff;
    return (u << 1) == 0ull || (e >= 1023 + lo && e < 1023 + hi);
}
// With |u| in [2^-60, 2^60) or zero, every product of the polynomials is zero
// or above 2^-240, every non-zero sum of two of their terms above 2^-350 (a
// difference of two doubles is zero or at least an ulp of the smaller), and
// with the moments in [2^-300, 2^300) or zero no scaled product leaves the
// normal range.
__host__ __device__ __forceinline__ bool cm_factored_ok(const CmSite& c) {
    return exp_within(c.ux, -60, 60) && exp_within(c.uy, -60, 60) && exp_within(c.k0, -300, 300) &&
           exp_within(c.k4, -300, 300) && exp_within(c.k5, -300, 300) && exp_within(c.k1, -300, 300) &&
           exp_within(c.k2, -300, 300);
}

template <bool UNF>
__host__ __device__ __forceinline__ void cm_site(CmSite& c, double rho, double ux, double uy, double Fx, double Fy,
                                                 double k4Pre, double k5Pre, double omega, double cs) {
    c.ux = ux;
    c.uy = uy;
    c.X2 = LSQ(ux);
    c.Y2 = LSQ(uy);
    c.XY = ux * uy;
    c.W = scale2(c.XY, 1);
    c.X2Y2 = c.X2 * c.Y2;
    c.uxY2 = ux * c.Y2;
    c.X2uy = c.X2 * uy;
    c.k0 = rho;
    c.k3 = 2.0 * rho * LSQ(cs);
    c.k4 = (1.0 - omega) * k4Pre;
    c.k5 = (1.0 - omega) * k5Pre;
    c.k8 = rho * LQU(cs);
    c.k1 = UNF ? 0.0 : 0.5 * Fx;
    c.k2 = UNF ? 0.0 : 0.5 * Fy;
    c.k6 = UNF ? 0.0 : 0.5 * Fy * LSQ(cs);
    c.k7 = UNF ? 0.0 : 0.5 * Fx * LSQ(cs);
}

// Post-collision population v (components cx, cy) of site c. `forced`: the
// force moments enter (they are exact zeros otherwise).
__host__ __device__ __forceinline__ double cm_population(int cx, int cy, const CmSite& c, bool forced) {
    const bool rest = cx == 0 && cy == 0, xax = cx != 0 && cy == 0, yax = cx == 0 && cy != 0;
    const bool diag = cx != 0 && cy != 0, up = cy > 0, same = cx == cy;
    const int cc = cx * cy;
    const double one = 1.0;
    // powers of two taken out of the coefficients of k0, k3, k4, k5, k8
    const int s0 = rest ? 0 : (diag ? -2 : -1), s3 = rest ? -1 : (diag ? -3 : -2);
    const int s5 = rest ? 2 : (diag ? -1 : 0);
    double a0, b0, c0, d0;
    if (rest) { a0 = c.X2Y2; b0 = -c.X2; c0 = -c.Y2; d0 = one; }
    else if (xax) { a0 = c.X2; b0 = -c.X2Y2; c0 = sgn_c(-cx, c.uxY2); d0 = sgn_c(cx, c.ux); }
    else if (yax) { a0 = up ? c.Y2 : c.X2uy; b0 = up ? -c.X2uy : -c.X2Y2; c0 = up ? -c.X2Y2 : c.Y2; d0 = sgn_c(cy, c.uy); }
    else { a0 = c.X2Y2; b0 = sgn_c(cy, c.X2uy); c0 = sgn_c(cx, c.uxY2); d0 = sgn_c(cc, c.XY); }
    double a3, b3, c3, d3;
    if (rest) { a3 = c.X2; b3 = c.Y2; c3 = -2.0; d3 = 0.0; }
    else if (xax) { a3 = -c.X2; b3 = sgn_c(-cx, c.ux); c3 = -c.Y2; d3 = one; }
    else if (yax) { a3 = -c.X2; b3 = -c.Y2; c3 = sgn_c(-cy, c.uy); d3 = one; }
    else { a3 = c.X2; b3 = sgn_c(cx, c.ux); c3 = c.Y2; d3 = sgn_c(cy, c.uy); }
    double a4, b4, c4, d4;
    if (rest) { a4 = c.Y2; b4 = -c.X2; c4 = 0.0; d4 = 0.0; }
    else if (xax) { a4 = c.X2; b4 = sgn_c(cx, c.ux); c4 = -c.Y2; d4 = one; }
    else if (yax) { a4 = c.X2; b4 = -c.Y2; c4 = sgn_c(-cy, c.uy); d4 = -one; }
    else { a4 = -c.X2; b4 = sgn_c(-cx, c.ux); c4 = c.Y2; d4 = sgn_c(cy, c.uy); }
    double a5, b5, c5, d5;
    if (rest) { a5 = c.XY; b5 = 0.0; c5 = 0.0; d5 = 0.0; }
    else if (xax) { a5 = sgn_c(-cx, c.uy); b5 = -c.W; c5 = 0.0; d5 = 0.0; }
    else if (yax) { a5 = sgn_c(-cy, c.ux); b5 = -c.W; c5 = 0.0; d5 = 0.0; }
    else if (same) { a5 = up ? c.ux : c.W; b5 = up ? c.uy : -c.uy; c5 = up ? c.W : -c.ux; d5 = 0.5; }
    else { a5 = up ? c.ux : c.uy; b5 = up ? -c.uy : -c.ux; c5 = c.W; d5 = -0.5; }
    double a = (((a0 + b0) + c0) + d0) * scale2(c.k0, s0);
    if (forced) {
        double a1, b1, c1, d1, a2, b2, c2, d2;
        int s1, s2;
        const double Z = scale2(c.uxY2, 1), V = scale2(c.X2uy, 1);
        if (rest) { a1 = c.uxY2; b1 = -c.ux; c1 = 0.0; d1 = 0.0; s1 = 1; }
        else if (xax) { a1 = scale2(c.ux, 1); b1 = -Z; c1 = sgn_c(-cx, c.Y2); d1 = sgn_c(cx, one); s1 = -1; }
        else if (yax) { a1 = -c.uxY2; b1 = sgn_c(-cy, c.XY); c1 = 0.0; d1 = 0.0; s1 = 0; }
        else {
            a1 = same ? c.uy : (up ? c.W : Z);
            b1 = same ? sgn_c(cc * cy, c.W) : (up ? -c.uy : -c.W);
            c1 = same || up ? Z : -c.uy;
            d1 = same ? sgn_c(cy, c.Y2) : (up ? -c.Y2 : c.Y2);
            s1 = -2;
        }
        if (rest) { a2 = c.X2uy; b2 = -c.uy; c2 = 0.0; d2 = 0.0; s2 = 1; }
        else if (xax) { a2 = -c.X2uy; b2 = sgn_c(-cx, c.XY); c2 = 0.0; d2 = 0.0; s2 = 0; }
        else if (yax) { a2 = scale2(c.uy, 1); b2 = -V; c2 = sgn_c(-cy, c.X2); d2 = sgn_c(cy, one); s2 = -1; }
        else {
            a2 = same ? c.ux : (up ? V : c.W);
            b2 = same ? sgn_c(cy, c.W) : (up ? -c.W : -c.ux);
            c2 = same || !up ? V : -c.ux;
            d2 = same ? sgn_c(cy, c.X2) : (up ? c.X2 : -c.X2);
            s2 = -2;
        }
        a = a + (((a1 + b1) + c1) + d1) * scale2(c.k1, s1);
        a = a + (((a2 + b2) + c2) + d2) * scale2(c.k2, s2);
    }
    a = a + (((a3 + b3) + c3) + d3) * scale2(c.k3, s3);
    a = a + (((a4 + b4) + c4) + d4) * scale2(c.k4, s3);
    a = a + (((a5 + b5) + c5) + d5) * scale2(c.k5, s5);
    if (forced) {
        const double e6 = cy == 0 ? 0.0 : (diag ? sgn_c(cy, 0.5) : sgn_c(-cy, 0.5));
        const double e7 = cx == 0 ? 0.0 : (diag ? sgn_c(cx, 0.5) : sgn_c(-cx, 0.5));
        const double g6 = (rest || diag ? c.uy : -c.uy) + e6, g7 = (rest || diag ? c.ux : -c.ux) + e7;
        a = a + g6 * scale2(c.k6, rest ? 1 : (diag ? -1 : 0));
        a = a + g7 * scale2(c.k7, rest ? 1 : (diag ? -1 : 0));
    }
    const double k8 = scale2(c.k8, rest ? 0 : (diag ? -2 : -1));
    return rest || diag ? a + k8 : a - k8;
}


// ---- whole sites with the products on the integer units -------------------
//
// collide_bgk<UNF = true> and collide_cm<UNF = true> for a site whose values
// lie in the range populations_in_range() and site_range_ok() test: the same
// operations on the same operands. The products and the sums with a power of
// two are formed by the integer units (int_f64.cuh), the other sums by the FP64
// unit; for the central moments the power-of-two factors are taken out (as in
// cm_population) and the partial sums that directions share, up to their sign,
// formed once: 144 FP64 instructions a site where the written-out form takes
// about 310. Measured (1536 x 1536, central moments): 1.36 -> 0.68 ms a step,
// the FP64 unit busy 82 % of the time and the integer unit 53 %; with the
// products on the FP64 unit as well the shared sums alone would leave 240.

// The populations are in [2^-8, 1), so the density is in [2^-5, 9), and each
// velocity component is zero or in [2^-60, 2^-3): then every product of the two
// collisions is zero or in the normal range (cm_factored_ok's bounds), and what 1/2, 1 and 2 are added to
// is smaller than they are (3 |ux + uy| < 3/4, |ux + uy + 2 ux uy| < 1/2).
__host__ __device__ __forceinline__ bool populations_in_range(const double f[9]) {
    unsigned worst = 0;
#pragma unroll
    for (int v = 0; v < 9; v++) {
        const unsigned d = (unsigned)(div_bits(f[v]) >> 32) - ((1023u - 8u) << 20);
        worst = d > worst ? d : worst;
    }
    return worst < (8u << 20);
}
__host__ __device__ __forceinline__ bool velocity_in_range(double u) {
    const unsigned long long b = div_bits(u) << 1;
    return b == 0ull || (unsigned)(b >> 53) - (1023u - 60u) < 57u;
}
__host__ __device__ __forceinline__ bool site_range_ok(double ux, double uy, double omega) {
    const unsigned w = (unsigned)(div_bits(omega) >> 52);  // omega in [2^-50, 4)
    return velocity_in_range(ux) && velocity_in_range(uy) && w - (1023u - 50u) < 52u;
}

// A product, or 1/2, 1 or 2 plus x, by the integer units or (INT = false) by the FP64
// unit: the same values (but for the sign of a zero product). Where the FP64
// unit is busy the integer form is free; on a lone warp, whose time is a chain,
// an FP64 product is the shorter one.
template <bool INT, int ZERO = kZeroA>
__host__ __device__ __forceinline__ double prod(double a, double b) {
    return INT ? mul_int<ZERO>(a, b) : a * b;
}
template <bool INT>
__host__ __device__ __forceinline__ double half_plus(double x) {
    return INT ? add_pow2_int<-1>(x) : 0.5 + x;
}
template <bool INT>
__host__ __device__ __forceinline__ double one_plus(double x) {
    return INT ? add_pow2_int<0>(x) : 1.0 + x;
}
template <bool INT>
__host__ __device__ __forceinline__ double two_plus(double x) {
    return INT ? add_pow2_int<1>(x) : 2.0 + x;
}

// equilibrium<false>() and equilibrium<true>() of all nine directions (rho in
// [2^-5, 9), velocity_in_range), the products that directions share formed
// once.
template <bool INT = true>
__host__ __device__ __forceinline__ void equilibria_bgk_int(double rho, double ux, double uy, double feq[9]) {
    const double px = prod<INT>(ux, 3.0), py = prod<INT>(uy, 3.0);
    const double pa = prod<INT>(ux + uy, 3.0), pb = prod<INT>(ux - uy, 3.0);
    const double d9 = prod<INT, kZeroAny>(prod<INT>(ux, 9.0), uy);
    const double X2 = prod<INT>(ux, ux), Y2 = prod<INT>(uy, uy);
    constexpr double c0 = 0.0 - 1.0 / 3.0, c1 = 1.0 - 1.0 / 3.0;
    const double x0 = prod<INT>(X2, c0), x1 = prod<INT>(X2, c1), y0 = prod<INT>(Y2, c0), y1 = prod<INT>(Y2, c1);
    const double h00 = prod<INT>(x0 + y0, 4.5), h10 = prod<INT>(x1 + y0, 4.5);
    const double h01 = prod<INT>(x0 + y1, 4.5), h11 = prod<INT>(x1 + y1, 4.5);
    const double r0 = prod<INT, kNonZero>(rho, 4.0 / 9.0), r1 = prod<INT, kNonZero>(rho, 1.0 / 9.0);
    const double r2 = prod<INT, kNonZero>(rho, 1.0 / 36.0);
    feq[0] = prod<INT, kNonZero>(one_plus<INT>(h00), r0);
    feq[1] = prod<INT, kNonZero>(one_plus<INT>(px) + h10, r1);
    feq[2] = prod<INT, kNonZero>(one_plus<INT>(-px) + h10, r1);
    feq[3] = prod<INT, kNonZero>(one_plus<INT>(py) + h01, r1);
    feq[4] = prod<INT, kNonZero>(one_plus<INT>(-py) + h01, r1);
    feq[5] = prod<INT, kNonZero>((one_plus<INT>(pa) + h11) + d9, r2);
    feq[6] = prod<INT, kNonZero>((one_plus<INT>(-pa) + h11) + d9, r2);
    feq[7] = prod<INT, kNonZero>((one_plus<INT>(pb) + h11) + -d9, r2);
    feq[8] = prod<INT, kNonZero>((one_plus<INT>(-pb) + h11) + -d9, r2);
}
template <bool INT = true>
__host__ __device__ __forceinline__ void equilibria_cm_int(double rho, double ux, double uy, double feq[9]) {
    // per axis 2 - 3 u^2 and ((9 u^2 +- 6 u) - 3 u^2) + 2
    const double X2 = prod<INT>(ux, ux), Y2 = prod<INT>(uy, uy);
    const double x3 = prod<INT>(X2, 3.0), x9 = prod<INT>(X2, 9.0), x6 = prod<INT>(ux, 6.0);
    const double y3 = prod<INT>(Y2, 3.0), y9 = prod<INT>(Y2, 9.0), y6 = prod<INT>(uy, 6.0);
    const double ax = two_plus<INT>(-x3), axp = two_plus<INT>((x9 + x6) - x3), axm = two_plus<INT>((x9 - x6) - x3);
    const double ay = two_plus<INT>(-y3), ayp = two_plus<INT>((y9 + y6) - y3), aym = two_plus<INT>((y9 - y6) - y3);
    const double rq = scale2_nz(rho, -2);
    const double r0 = prod<INT, kNonZero>(rq, 4.0 / 9.0), r1 = prod<INT, kNonZero>(rq, 1.0 / 9.0);
    const double r2 = prod<INT, kNonZero>(rq, 1.0 / 36.0);
    const double c = prod<INT, kNonZero>(r1, ax), p = prod<INT, kNonZero>(r2, axp), m = prod<INT, kNonZero>(r2, axm);
    feq[0] = prod<INT, kNonZero>(prod<INT, kNonZero>(r0, ax), ay);
    feq[1] = prod<INT, kNonZero>(prod<INT, kNonZero>(r1, axp), ay);
    feq[2] = prod<INT, kNonZero>(prod<INT, kNonZero>(r1, axm), ay);
    feq[3] = prod<INT, kNonZero>(c, ayp);
    feq[4] = prod<INT, kNonZero>(c, aym);
    feq[5] = prod<INT, kNonZero>(p, ayp);
    feq[6] = prod<INT, kNonZero>(m, aym);
    feq[7] = prod<INT, kNonZero>(p, aym);
    feq[8] = prod<INT, kNonZero>(m, ayp);
}

template <bool INT = true>
__host__ __device__ __forceinline__ void collide_bgk_int(const double f[9], double rho, double ux, double uy,
                                                         double omega, double fs[9]) {
    double feq[9];
    equilibria_bgk_int<INT>(rho, ux, uy, feq);
#pragma unroll
    for (int v = 0; v < 9; v++) fs[v] = f[v] + prod<INT>(feq[v] - f[v], omega);
}

// om = 1 - omega, cs2 = cs^2, cs4 = cs^4 in the written-out form's operations.
template <bool INT = true>
__host__ __device__ __forceinline__ void collide_cm_int(const double f[9], double rho, double ux, double uy,
                                                        double om, double cs2, double cs4, double fs[9]) {
    const double X2 = prod<INT>(ux, ux), Y2 = prod<INT>(uy, uy);
    const double xm = one_plus<INT>(-ux), xq = one_plus<INT>(ux);
    const double ym = one_plus<INT>(-uy), yq = one_plus<INT>(uy);
    const double D = X2 - Y2;
    double k4Pre, k5Pre;
    {
        // f (cx^2 - cy^2) and (f cx) cy with cx = c - ux: the components of
        // c = 0 and -1 are -ux and -(1 + ux); signs go into the sums
        const double sxm = prod<INT, kNonZero>(xm, xm), sxq = prod<INT, kNonZero>(xq, xq);
        const double sym = prod<INT, kNonZero>(ym, ym), syq = prod<INT, kNonZero>(yq, yq);
        k4Pre = prod<INT>(D, f[0]);
        k4Pre = k4Pre + prod<INT>(sxm - Y2, f[1]);
        k4Pre = k4Pre + prod<INT>(sxq - Y2, f[2]);
        k4Pre = k4Pre + prod<INT>(X2 - sym, f[3]);
        k4Pre = k4Pre + prod<INT>(X2 - syq, f[4]);
        k4Pre = k4Pre + prod<INT>(sxm - sym, f[5]);
        k4Pre = k4Pre + prod<INT>(sxq - syq, f[6]);
        k4Pre = k4Pre + prod<INT>(sxm - syq, f[7]);
        k4Pre = k4Pre + prod<INT>(sxq - sym, f[8]);
        k5Pre = prod<INT, kZeroAny>(prod<INT>(ux, f[0]), uy);
        k5Pre = k5Pre - prod<INT>(uy, prod<INT, kNonZero>(xm, f[1]));
        k5Pre = k5Pre + prod<INT>(uy, prod<INT, kNonZero>(xq, f[2]));
        k5Pre = k5Pre - prod<INT>(prod<INT>(ux, f[3]), ym);
        k5Pre = k5Pre + prod<INT>(prod<INT>(ux, f[4]), yq);
        k5Pre = k5Pre + prod<INT, kNonZero>(ym, prod<INT, kNonZero>(xm, f[5]));
        k5Pre = k5Pre + prod<INT, kNonZero>(yq, prod<INT, kNonZero>(xq, f[6]));
        k5Pre = k5Pre - prod<INT, kNonZero>(yq, prod<INT, kNonZero>(xm, f[7]));
        k5Pre = k5Pre - prod<INT, kNonZero>(ym, prod<INT, kNonZero>(xq, f[8]));
    }
    const double k4 = prod<INT, kZeroAny>(om, pos_zero(k4Pre)), k5 = prod<INT, kZeroAny>(om, pos_zero(k5Pre));
    const double k3 = scale2_nz(prod<INT, kNonZero>(rho, cs2), 1), k8 = prod<INT, kNonZero>(rho, cs4);
    const double XY = prod<INT, kZeroAny>(ux, uy), W = scale2(XY, 1);
    const double X2Y2 = prod<INT, kZeroAny>(X2, Y2), uxY2 = prod<INT, kZeroAny>(ux, Y2);
    const double X2uy = prod<INT, kZeroAny>(X2, uy);
    const double A = X2 - X2Y2, Bq = X2uy - X2Y2, Sp = X2Y2 + X2uy;
    const double S = X2 + Y2, Qp = X2 + ux, Qm = X2 - ux, QpY = Qp + Y2, QmY = Qm + Y2, Rp = Qp - Y2, Rm = Qm - Y2;
    const double uyW = uy - W, dxy = ux - uy;
    // population: (((p0 k0 + p3 k3) + p4 k4) + p5 k5) +- k8, the moments scaled
    // by the powers of two of its class (Z3: whether p3 may be zero)
#define LIFE_CM_POP(v, Z3, p0, p3, p4, p5, K0, K3, K4, K5, K8) \
    fs[v] = (((prod<INT>(p0, K0) + prod<INT, Z3>(p3, K3)) + prod<INT, kZeroAny>(p4, K4)) + prod<INT, kZeroAny>(p5, K5)) + (K8)
    LIFE_CM_POP(0, kNonZero, one_plus<INT>(-A - Y2), -two_plus<INT>(-S), Y2 - X2, XY, rho, scale2_nz(k3, -1), scale2(k4, -1), scale2(k5, 2), k8);
    {
        const double K0 = scale2_nz(rho, -1), K3 = scale2_nz(k3, -2), K4 = scale2(k4, -2), K8 = -scale2_nz(k8, -1);
        LIFE_CM_POP(1, kNonZero, (A - uxY2) + ux, one_plus<INT>(-QpY), one_plus<INT>(Rp), -(uy + W), K0, K3, K4, k5, K8);
        LIFE_CM_POP(2, kNonZero, (A + uxY2) - ux, one_plus<INT>(-QmY), one_plus<INT>(Rm), uyW, K0, K3, K4, k5, K8);
        LIFE_CM_POP(3, kNonZero, ((Y2 - X2uy) - X2Y2) + uy, one_plus<INT>(-(S + uy)), -one_plus<INT>(uy - D), -(ux + W), K0, K3, K4, k5, K8);
        LIFE_CM_POP(4, kNonZero, (Bq + Y2) - uy, one_plus<INT>(-(S - uy)), -one_plus<INT>(-(D + uy)), ux - W, K0, K3, K4, k5, K8);
    }
    {
        const double K0 = scale2_nz(rho, -2), K3 = scale2_nz(k3, -3), K4 = scale2(k4, -3), K5 = scale2(k5, -1);
        const double K8 = scale2_nz(k8, -2);
        LIFE_CM_POP(5, kZeroA, (Sp + uxY2) + XY, QpY + uy, uy - Rp, half_plus<INT>((ux + uy) + W), K0, K3, K4, K5, K8);
        LIFE_CM_POP(6, kZeroA, XY - (Bq + uxY2), QmY - uy, -(Rm + uy), half_plus<INT>(-(uyW + ux)), K0, K3, K4, K5, K8);
        LIFE_CM_POP(7, kZeroA, (uxY2 - Bq) - XY, QpY - uy, -(Rp + uy), -half_plus<INT>(dxy - W), K0, K3, K4, K5, K8);
        LIFE_CM_POP(8, kZeroA, (Sp - uxY2) - XY, QmY + uy, uy - Rm, -half_plus<INT>(-(dxy + W)), K0, K3, K4, K5, K8);
    }
#undef LIFE_CM_POP
}

}  // namespace life
