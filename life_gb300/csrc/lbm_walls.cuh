// The boundary-condition sites of a step.
//
// Straight stretches of no-slip and velocity walls and of the convective outlet
// take one thread a site, 32 sites a warp (wall_site), with what directions
// share formed once: about 200 FP64 instructions of the warp (BGK), 6 a site.
// Corners, pressure and free-slip walls, which extrapolate from the fluid, and
// cases with a force take nine lanes a site (lbm_lanes.cuh: 95 to 130 FP64
// instructions for three sites, 38 a site, a shorter chain), and with many such
// sites one thread a site, every direction written out (boundary_site: 700 to 900
// for 32 sites). wall_plan.h has the lines between them. (Products from the integer
// units, as in the interior, make the warp's chain longer: 15.6 -> 18.4 us at
// 256 x 256, no gain in a batch.) A thread whose values leave the range that
// moment_sums_int takes runs the general code of boundary_site(). All of them
// form every value with the operations and in the order of site_state() and
// collide().
#pragma once
#include "lbm_lanes.cuh"
#include "wall_plan.h"

namespace life {

static_assert(kLaneSites == 3, "wall_plan.h counts three sites a warp");

// div_rn_recip for a zero numerator or operands within its window.
__device__ __forceinline__ double quotient_in_range(double a, double b, double y) {
    const double q0 = mul_int<kZeroAny>(a, y);
    const double r0 = fma(-b, q0, a);
    const double q1 = fma(r0, y, q0);
    const double r1 = fma(-b, q1, a);
    const double q = fma(r1, y, q1);
    return (div_bits(a) << 1) == 0ull ? q0 : q;
}

// Whether rho lies in the range of the equilibria: [2^-5, 2^3).
__device__ __forceinline__ bool density_in_range(double rho) {
    return (unsigned)(div_bits(rho) >> 32) - ((1023u - 5u) << 20) < (8u << 20);
}

template <bool CM, class S>
static __device__ __noinline__ void boundary_site_call(const typename S::T* __restrict__ A, typename S::T* __restrict__ B,
                                                       const LatDev& L, int t, int i, int j, double dU0, double dU1) {
    const double dU[2] = {dU0, dU1};
    boundary_site<CM, S>(A, B, L, t, i, j, dU);
}

// Site (i, j) of a straight stretch of edge (nd, nn): its inward normal has the
// component nn along x (nd = 0) or y (nd = 1). type: LIFE_WALL, LIFE_VELOCITY or
// LIFE_CONVECTIVE (with the outlet's speed term dU). The case has no force.
// Returns false, with nothing written, where a value is out of range.
template <bool CM, class S>
__device__ __forceinline__ bool wall_site(const typename S::T* __restrict__ A, typename S::T* __restrict__ B,
                                          const LatDev& L, int t, int i, int j, int type, int nd, int nn, double dU0,
                                          double dU1) {
    double f[9];
    gather<S>(A, L, i, j, f);
    if (type == LIFE_CONVECTIVE) {
        const double* fp = L.outlet_f_prev + (size_t)j * 3;
        f[2] = fp[0] + 3.0 * wgt(2) * (dU0 * -1.0 + dU1 * 0.0);
        f[6] = fp[1] + 3.0 * wgt(6) * (dU0 * -1.0 + dU1 * -1.0);
        f[8] = fp[2] + 3.0 * wgt(8) * (dU0 * -1.0 + dU1 * 1.0);
        if (!populations_in_range(f)) return false;
    } else {
        if (!populations_in_range(f)) return false;
        double un[2] = {0.0, 0.0};
        if (type == LIFE_VELOCITY) {
            const double ramp = L.steps[t % L.steps_cap].ramp;
            un[0] = L.u_in[j * 2 + 0] * ramp;
            un[1] = L.u_in[j * 2 + 1] * ramp;
        }
        // the populations that leave through the wall and along it, in order
        const bool pos = nn > 0;
        double a, b, c, d, e;
        if (nd == 0) {
            a = pos ? f[2] : f[1];
            b = pos ? f[6] : f[5];
            c = pos ? f[8] : f[7];
            d = f[3];
            e = f[4];
        } else {
            a = pos ? f[4] : f[3];
            b = pos ? f[6] : f[5];
            c = pos ? f[7] : f[8];
            d = f[1];
            e = f[2];
        }
        const double num = scale2_nz((a + b) + c, 1) + ((f[0] + d) + e);
        const double den = 1.0 - sgn_c(nn, nd == 0 ? un[0] : un[1]);
        const double rn = div_bits(den) == 0x3ff0000000000000ull ? num : div_rn_recip(num, den, __drcp_rn(den));
        if (!density_in_range(rn) || !site_range_ok(un[0], un[1], L.omega)) return false;
        double feq[9], fneq[9];
        if (CM) equilibria_cm_int<false>(rn, un[0], un[1], feq);
        else equilibria_bgk_int<false>(rn, un[0], un[1], feq);
        // (in order: an opposite population of an unknown one is a known one)
#pragma unroll
        for (int v = 0; v < 9; v++) {
            double h = f[v];
            if (v > 0 && (nd == 0 ? cx_of(v) : cy_of(v)) == nn) h = feq[v] + (f[opp_of(v)] - feq[opp_of(v)]);
            fneq[v] = h - feq[v];
        }
        double Sxx = 0.0, Syy = 0.0, Sxy = 0.0;
        bool hx = false, hy = false, hxy = false;
#pragma unroll
        for (int v = 1; v < 9; v++) {
            if (cx_of(v) != 0) { Sxx = hx ? Sxx + fneq[v] : fneq[v]; hx = true; }
            if (cy_of(v) != 0) { Syy = hy ? Syy + fneq[v] : fneq[v]; hy = true; }
            const int cc = cx_of(v) * cy_of(v);
            if (cc != 0) { Sxy = hxy ? (cc > 0 ? Sxy + fneq[v] : Sxy - fneq[v]) : (cc > 0 ? fneq[v] : -fneq[v]); hxy = true; }
        }
        const double x0 = prod<false>(Sxx, 0.0 - L.cs2), x1 = prod<false>(Sxx, 1.0 - L.cs2);
        const double y0 = prod<false>(Syy, 0.0 - L.cs2), y1 = prod<false>(Syy, 1.0 - L.cs2);
        const double s2 = scale2(Sxy, 1), diag = x1 + y1;
        f[0] = feq[0] + prod<false>(x0 + y0, L.wreg[0]);
        const double ex = prod<false>(x1 + y0, L.wreg[1]), ey = prod<false>(x0 + y1, L.wreg[1]);
        f[1] = feq[1] + ex;
        f[2] = feq[2] + ex;
        f[3] = feq[3] + ey;
        f[4] = feq[4] + ey;
        const double dp = prod<false>(diag + s2, L.wreg[2]), dm = prod<false>(diag - s2, L.wreg[2]);
        f[5] = feq[5] + dp;
        f[6] = feq[6] + dp;
        f[7] = feq[7] + dm;
        f[8] = feq[8] + dm;
        if (!populations_in_range(f)) return false;
    }
    double rho, mx, my, fs[9];
    moment_sums_int(f, rho, mx, my);
    const double y = __drcp_rn(rho);
    const double ux = quotient_in_range(mx, rho, y), uy = quotient_in_range(my, rho, y);
    if (!site_range_ok(ux, uy, L.omega)) return false;
    outlet_outputs(L, i, j, f, ux, uy);
    if (CM) collide_cm_int<false>(f, rho, ux, uy, L.om1, L.cs2, L.cs4, fs);
    else collide_bgk_int<false>(f, rho, ux, uy, L.omega, fs);
    const size_t s = (size_t)j * L.pitch + i;
#pragma unroll
    for (int v = 0; v < 9; v++) B[(size_t)v * L.S + s] = S::save(fs[v], v);
    return true;
}

__device__ __forceinline__ void edge_ij(const LatDev& L, int e, int q, int& i, int& j) {
    if (e < 2) {
        i = 1 + q;
        j = e == 0 ? 0 : L.Ny - 1;
    } else {
        i = e == 2 ? 0 : L.Nx - 1;
        j = 1 + q;
    }
}

template <bool CM, class S>
__device__ __forceinline__ void walls_warp(const typename S::T* __restrict__ A, typename S::T* __restrict__ B,
                                           const LatDev& L, int t, const WallPlan& plan, int warp) {
    if (warp < plan.lane_warps) {
        const int slot = site_lane().slot;
        int q = kLaneSites * warp + slot, i = 0, j = 0;
        bool site = q < plan.lane_sites;
        if (q < 4) {
            i = (q & 1) ? L.Nx - 1 : 0;
            j = (q & 2) ? L.Ny - 1 : 0;
        } else {
            q -= 4;
            for (int e = 0; e < 4 && site; e++) {
                if (!((plan.lanes >> e) & 1)) continue;
                if (q < edge_sites(L, e)) {
                    edge_ij(L, e, q, i, j);
                    break;
                }
                q -= edge_sites(L, e);
            }
        }
        lanes_boundary<CM, S>(A, B, L, t, site, i, j);
        return;
    }
    int q = 32 * (warp - plan.lane_warps) + ((int)threadIdx.x & 31);
    for (int e = 0; e < 4; e++) {
        if (!((plan.straight >> e) & 1)) continue;
        const int n = edge_sites(L, e), padded = (n + 31) / 32 * 32;
        if (q >= padded) {
            q -= padded;
            continue;
        }
        const int type = edge_type(L, e);
        int i, j;
        edge_ij(L, e, q, i, j);
        double dU0 = 0.0, dU1 = 0.0;
        if (type == LIFE_CONVECTIVE) {  // (the same for the whole warp)
            const double uOut = lanes_outlet_mean<S::prec == LIFE_PREC_F64>(L);
            if (q < n) {
                outlet_term(L, uOut, j, dU0, dU1);
                L.delU[j * 2 + 0] = dU0;
                L.delU[j * 2 + 1] = dU1;
            }
        }
        if (q >= n) return;
        if (!wall_site<CM, S>(A, B, L, t, i, j, type, e < 2 ? 1 : 0, e == 0 || e == 2 ? 1 : -1, dU0, dU1))
            boundary_site_call<CM, S>(A, B, L, t, i, j, dU0, dU1);
        return;
    }
}

// One warp a block: a site is a long chain, spread over as many SMs as possible.
template <bool CM, class S>
__global__ void __launch_bounds__(32) k_perimeter(const typename S::T* __restrict__ A, typename S::T* __restrict__ B,
                                                  LatDev L, int t, WallPlan plan) {
    walls_warp<CM, S>(A, B, L, step_t(L, t), plan, blockIdx.x);
}

// One thread a site, every direction written out, around the whole perimeter
// (perimeter_ij's order). The outlet's mean is formed by the warps that hold outlet
// sites.
template <bool CM, class S>
__global__ void __launch_bounds__(32) k_perimeter_general(const typename S::T* __restrict__ A,
                                                          typename S::T* __restrict__ B, LatDev L, int t) {
    int i = 0, j = 0;
    const bool on = perimeter_ij(L, 32 * (int)blockIdx.x + (int)threadIdx.x, i, j);
    const int type = on ? site_type(L, i, j) : LIFE_FLUID;
    const bool form = L.convective && L.outlet_form == kOutletSites;
    double dU[2] = {0.0, 0.0};
    if (form && __any_sync(kAllLanes, type == LIFE_CONVECTIVE)) {
        const double uOut = lanes_outlet_mean<S::prec == LIFE_PREC_F64>(L);
        if (type == LIFE_CONVECTIVE) {
            outlet_term(L, uOut, j, dU[0], dU[1]);
            L.delU[j * 2 + 0] = dU[0];
            L.delU[j * 2 + 1] = dU[1];
        }
    }
    if (type != LIFE_FLUID) boundary_site<CM, S>(A, B, L, step_t(L, t), i, j, form ? dU : nullptr);
}

template <class S>
static void launch_walls(const void* A, void* B, const LatDev& L, int t, cudaStream_t s) {
    const WallPlan plan = wall_plan(L);
    const typename S::T* a = (const typename S::T*)A;
    typename S::T* b = (typename S::T*)B;
    if (plan.general) {
        if (L.cm) k_perimeter_general<true, S><<<plan.warps, 32, 0, s>>>(a, b, L, t);
        else k_perimeter_general<false, S><<<plan.warps, 32, 0, s>>>(a, b, L, t);
        return;
    }
    if (L.cm) k_perimeter<true, S><<<plan.warps, 32, 0, s>>>(a, b, L, t, plan);
    else k_perimeter<false, S><<<plan.warps, 32, 0, s>>>(a, b, L, t, plan);
}

}  // namespace life
