// FP64 site arithmetic with a site's nine populations on nine lanes.
//
// An FP64 instruction occupies its sub-partition's unit for 64 cycles whether
// one lane or all 32 are active (2 FP64 lanes per cycle and SM). With one
// thread per site a boundary or support site is a chain of 700-900 such
// instructions (every direction written out): 28 us for one wall row, however
// short. Here a warp takes three sites, nine lanes each: what differs by
// direction runs once for all of a site's directions, the ordered sums of the
// reference (density, both momenta; the three stress sums) run side by side
// on different lanes in the same instructions, and a wall site is about 95
// instructions (BGK) or 130 (central moments). The boundary kernel of a
// 1000 x 400 channel went from 30.0 to 17.4 us (central moments, FP32 storage),
// that of a 256^2 FP64 cavity from 28 to 10.8 us (cold, under ncu). Per site
// the FP64 unit is busy as long as before (three sites share 95 instructions,
// where 32 shared 800); where many sites step together, straight walls take one
// thread a site with the shared products formed once (lbm_walls.cuh, 200 for
// 32 sites). Every value is formed with
// the operations and in the order of site_state() / collide() in
// lbm_device.cuh, so the results are the same bits.
//
// Every function below is called by whole warps. Lanes 27-31 repeat the first
// five directions of the third site and never store.
#pragma once
#include "collide_cm.cuh"
#include "lbm_device.cuh"

namespace life {

constexpr unsigned kAllLanes = 0xffffffffu;
constexpr int kLaneSites = 3;  // sites per warp

struct SiteLane {
    int base;    // first lane of the site's nine
    int slot;    // which of the warp's sites (0..2)
    int v;       // direction of this lane
    int cx, cy;
    int opp;     // lane holding the opposite direction
    int role;    // v % 3: which of three ordered sums this lane forms
    bool store;  // false on the spare lanes
};

__device__ __forceinline__ SiteLane site_lane() {
    SiteLane g;
    const int lane = (int)threadIdx.x & 31;
    g.slot = lane < 9 ? 0 : (lane < 18 ? 1 : 2);
    g.base = 9 * g.slot;
    g.store = lane < 27;
    g.v = g.store ? lane - g.base : lane - 27;
    g.cx = cx_of(g.v);
    g.cy = cy_of(g.v);
    g.opp = g.base + opp_of(g.v);
    g.role = g.v % 3;
    return g;
}

__device__ __forceinline__ double lane_get(double x, int lane) { return __shfl_sync(kAllLanes, x, lane); }
__device__ __forceinline__ double sel(bool c, double a, double b) { return c ? a : b; }

template <class S>
__device__ __forceinline__ double lanes_gather(const typename S::T* __restrict__ P, const LatDev& L, const SiteLane& g,
                                               int i, int j) {
    int si = i - g.cx, sj = j - g.cy;
    si = si < 0 ? si + L.Nx : (si >= L.Nx ? si - L.Nx : si);
    sj = sj < 0 ? sj + L.Ny : (sj >= L.Ny ? sj - L.Ny : sj);
    return S::load(P[(size_t)g.v * L.S + (size_t)sj * L.pitch + si], g.v);
}

// moment_sums() on lanes: role 0 adds up the density (f0..f8), role 1 the x
// momentum (f1 -f2 +f5 -f6 +f7 -f8), role 2 the y momentum (f3 -f4 +f5 -f6
// -f7 +f8), each in its order and started at its first term. A finished sum
// adds +0 (pos_zero clears a -0 either way).
__device__ __forceinline__ double lanes_sums(const SiteLane& g, double f) {
    const int s1[6] = {1, 2, 5, 6, 7, 8}, s2[6] = {3, 4, 5, 6, 7, 8};
    const int c1[6] = {1, -1, 1, -1, 1, -1}, c2[6] = {1, -1, 1, -1, -1, 1};
    double acc = 0.0;
#pragma unroll
    for (int q = 0; q < 9; q++) {
        const int p = q < 6 ? q : 5;
        const int src = g.role == 0 ? q : (g.role == 1 ? s1[p] : s2[p]);
        double x = lane_get(f, g.base + src);
        if (g.role != 0) x = q < 6 ? sgn_c(g.role == 1 ? c1[p] : c2[p], x) : 0.0;
        acc = q == 0 ? x : acc + x;
    }
    return pos_zero(acc);
}

// The velocity of macroscopic() from this lane's sum m, given y = RN(1/rho).
__device__ __forceinline__ void lanes_velocity(const SiteLane& g, double m, double rho, double y, double Fx, double Fy,
                                               double& ux, double& uy) {
    const double q = div_rn_recip(m + 0.5 * (g.role == 2 ? Fy : Fx), rho, y);
    ux = lane_get(q, g.base + 1);
    uy = lane_get(q, g.base + 2);
}

// macroscopic() / macroscopic_ibm(): F is the force in the half term.
__device__ __forceinline__ void lanes_macroscopic(const SiteLane& g, double f, double Fx, double Fy, double& rho,
                                                  double& ux, double& uy) {
    const double m = lanes_sums(g, f);
    rho = lane_get(m, g.base);
    lanes_velocity(g, m, rho, __drcp_rn(rho), Fx, Fy, ux, uy);
}

// equilibrium<CM>() of this lane's direction
template <bool CM>
__device__ __forceinline__ double lanes_equilibrium(const SiteLane& g, double rho, double ux, double uy) {
    const double w = wgt(g.v);
    if (CM) {
        // per axis ((9 u^2 +- 6 u) - 3 u^2) + 2; for c = 0 the first two are absent
        const double X2 = LSQ(ux), Y2 = LSQ(uy);
        const double px = 9.0 * X2 + sgn_c(g.cx, 6.0 * ux), py = 9.0 * Y2 + sgn_c(g.cy, 6.0 * uy);
        const double ax = (sel(g.cx == 0, 0.0, px) - 3.0 * X2) + 2.0;
        const double ay = (sel(g.cy == 0, 0.0, py) - 3.0 * Y2) + 2.0;
        return 0.25 * rho * w * ax * ay;
    }
    const double cu = sel(g.cx == 0, 0.0, sgn_c(g.cx, ux)) + sel(g.cy == 0, 0.0, sgn_c(g.cy, uy));
    double s = 1.0 + 3.0 * cu;
    s = s + 4.5 * (LSQ(ux) * (g.cx == 0 ? 0.0 - 1.0 / 3.0 : 1.0 - 1.0 / 3.0) +
                   LSQ(uy) * (g.cy == 0 ? 0.0 - 1.0 / 3.0 : 1.0 - 1.0 / 3.0));
    const int cc = g.cx * g.cy;
    s = s + sel(cc == 0, 0.0, sgn_c(cc, 9.0 * ux * uy));
    return rho * w * s;
}

// regularised() on lanes; `on`: whether this lane's site takes the condition
// (f is returned unchanged otherwise).
template <bool CM>
__device__ __forceinline__ double lanes_regularised(const SiteLane& g, double f, bool on, int type, int nx, int ny,
                                                    int nd, double rn, double u0, double u1, const LatDev& L,
                                                    double rho_x1, double rho_x2) {
    const bool corner = nx != 0 && ny != 0;
    const bool density = type == LIFE_VELOCITY || type == LIFE_WALL || type == LIFE_FREESLIP;
    const int nn = nd == 0 ? nx : ny;
    // the ordered sums over the directions with c.n = -1 (even lanes) and
    // c.n = 0 (odd lanes): nd 0: {2,6,8} or {1,5,7} and {0,3,4}; nd 1: {4,6,7}
    // or {3,5,8} and {0,1,2}
    const bool plus = (g.v & 1) == 0;
    int a, b, c;
    if (nd == 0) { a = plus ? (nn > 0 ? 2 : 1) : 0; b = plus ? (nn > 0 ? 6 : 5) : 3; c = plus ? (nn > 0 ? 8 : 7) : 4; }
    else { a = plus ? (nn > 0 ? 4 : 3) : 0; b = plus ? (nn > 0 ? 6 : 5) : 1; c = plus ? (nn > 0 ? 7 : 8) : 2; }
    const double fa = lane_get(f, g.base + a), fb = lane_get(f, g.base + b), fc = lane_get(f, g.base + c);
    const double part = pos_zero((fa + fb) + fc);
    const double num = 2.0 * lane_get(part, g.base) + lane_get(part, g.base + 1);
    const double un = nd == 0 ? u0 : u1;
    // (2 f+ + f0) / (1 - n u) or / rho_n; a site at rest divides by 1 exactly
    double den = type == LIFE_PRESSURE ? rn : 1.0 - sgn_c(nn, un);
    if (!on || corner) den = 1.0;
    double quo = num;
    if (__any_sync(kAllLanes, div_bits(den) != 0x3ff0000000000000ull)) quo = div_rn_recip(num, den, __drcp_rn(den));
    if (corner) {
        if (density) rn = 2.0 * rho_x1 - rho_x2;
    } else if (density) {
        rn = quo;
    } else if (type == LIFE_PRESSURE) {
        const double un_new = sgn_c(nn, 1.0 - quo);
        if (nd == 0) u0 = un_new;
        else u1 = un_new;
    }
    const double feq = lanes_equilibrium<CM>(g, rn, u0, u1);
    const double other = lane_get(f, g.opp) - lane_get(feq, g.opp);
    double h = f;
    if (corner) {
        if (g.cx == nx || g.cy == ny) h = nx * g.cx + ny * g.cy == 0 ? feq : feq + other;
    } else if ((nd == 0 ? g.cx : g.cy) == nn) {
        h = feq + other;
    }
    const double fneq = h - feq;
    // the stress sums: role 0 xx (1 2 5 6 7 8), role 1 yy (3 4 5 6 7 8),
    // role 2 xy (5 6 -7 -8), from +0 in the order of the directions
    double acc = 0.0;
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const int src = q < 2 ? (g.role == 1 ? 3 + q : 1 + q) : 3 + q;
        double x = lane_get(fneq, g.base + src);
        if (g.role == 2) x = q < 2 ? 0.0 : (q < 4 ? x : -x);
        acc = acc + x;
    }
    const double Sxx = lane_get(acc, g.base), Syy = lane_get(acc, g.base + 1), Sxy = lane_get(acc, g.base + 2);
    const double cs2 = LSQ(L.cs);
    const int cc = g.cx * g.cy;
    const double sxy = sel(cc == 0, 0.0, sgn_c(cc, scale2(Sxy, 1)));
    const double wq = g.v == 0 ? L.wreg[0] : (g.v < 5 ? L.wreg[1] : L.wreg[2]);
    const double reg = feq + wq * ((((g.cx == 0 ? 0.0 : 1.0) - cs2) * Sxx + ((g.cy == 0 ? 0.0 : 1.0) - cs2) * Syy) + sxy);
    return on ? reg : f;
}

// The first half of site_state() for the warp's three sites: this lane's
// population after the boundary condition, and the step's force at the site.
// STEP: called for a step (the outlet's speed term may have to be formed here,
// LatDev::outlet_form), not for a state already reached.
//
// The outlet's mean used to be a kernel of its own that everything waited for:
// 6 us of the 23 us step of a 1501 x 703 FP32 channel, 13-21 us with FP64
// storage and 400 rows (a sum in order).
template <bool CM, class S, bool STEP = false>
__device__ __forceinline__ double lanes_populations(const typename S::T* __restrict__ P, const LatDev& L, int t,
                                                    const SiteLane& g, int i, int j, double& Fx, double& Fy) {
    double f = lanes_gather<S>(P, L, g, i, j);
    force_xy_of(L, t, i, j, Fx, Fy);
    const int type = site_type(L, i, j);
    if (__any_sync(kAllLanes, type == LIFE_CONVECTIVE)) {
        double dU0 = 0.0, dU1 = 0.0;
        if (STEP && L.outlet_form == kOutletSites) {
            const double uOut = lanes_outlet_mean<S::prec == LIFE_PREC_F64>(L);
            if (type == LIFE_CONVECTIVE) {
                outlet_term(L, uOut, j, dU0, dU1);
                if (g.store && g.v == 0) {
                    L.delU[j * 2 + 0] = dU0;
                    L.delU[j * 2 + 1] = dU1;
                }
            }
        } else if (type == LIFE_CONVECTIVE) {
            dU0 = L.delU[j * 2 + 0];
            dU1 = L.delU[j * 2 + 1];
        }
        if (type == LIFE_CONVECTIVE && g.cx < 0) {
            const int k = g.v == 2 ? 0 : (g.v == 6 ? 1 : 2);
            f = L.outlet_f_prev[(size_t)j * 3 + k] + 3.0 * wgt(g.v) * (dU0 * (double)g.cx + dU1 * (double)g.cy);
        }
    }
    const bool reg = type != LIFE_FLUID && type != LIFE_CONVECTIVE;
    if (__any_sync(kAllLanes, reg)) {
        int nx = 0, ny = 0, nd = 0;
        if (reg) site_normal(L, i, j, nx, ny, nd);
        const bool corner = nx != 0 && ny != 0;
        double rn = 0.0, u0 = 0.0, u1 = 0.0, r1 = 0.0, r2 = 0.0;
        if (type == LIFE_VELOCITY) {
            const double ramp = L.steps[t % L.steps_cap].ramp;
            u0 = L.u_in[j * 2 + 0] * ramp;
            u1 = L.u_in[j * 2 + 1] * ramp;
        }
        const bool grad = type == LIFE_FREESLIP || type == LIFE_PRESSURE;
        const bool inner = reg && (grad || corner);
        if (__any_sync(kAllLanes, inner)) {
            // moments of the next two sites along the normal (own site: unused)
            double ax[2], ay[2], q[2];
#pragma unroll 1
            for (int k = 0; k < 2; k++) {
                const int ii = inner ? i + (k + 1) * nx : i, jj = inner ? j + (k + 1) * ny : j;
                const double fn = lanes_gather<S>(P, L, g, ii, jj);
                double Gx = Fx, Gy = Fy;
                if (L.site_force) force_xy_site(L, t, L.rho_prev[(size_t)jj * L.pitch + ii], Gx, Gy);
                double r, x, y;
                lanes_macroscopic(g, fn, Gx, Gy, r, x, y);
                q[k] = r;
                ax[k] = x;
                ay[k] = y;
            }
            if (grad) {
                if (type == LIFE_PRESSURE) rn = L.rho_in[j];
                const int d = 1 - nd;
                const double ud = (4.0 / 3.0) * (d == 0 ? ax[0] : ay[0]) - (1.0 / 3.0) * (d == 0 ? ax[1] : ay[1]);
                const int k = pressure_corner(type, nx, ny, i, j);
                const double un = k >= 0 ? L.corner_prev[k * 2 + nd] : 0.0;
                u0 = d == 0 ? ud : un;
                u1 = d == 0 ? un : ud;
            }
            if (inner && type != LIFE_PRESSURE) {
                r1 = q[0];
                r2 = q[1];
            }
        }
        f = lanes_regularised<CM>(g, f, reg, type, nx, ny, nd, rn, u0, u1, L, r1, r2);
    }
    return f;
}

// site_state() of the warp's three sites: this lane's population after the
// boundary condition and the site's moments (equal on the site's lanes).
template <bool CM, class S, bool STEP = false>
__device__ __forceinline__ void lanes_state(const typename S::T* __restrict__ P, const LatDev& L, int t,
                                            const SiteLane& g, int i, int j, double& f, double& rho, double& ux,
                                            double& uy) {
    double Fx, Fy;
    f = lanes_populations<CM, S, STEP>(P, L, t, g, i, j, Fx, Fy);
    lanes_macroscopic(g, f, Fx, Fy, rho, ux, uy);
}

// The written-out collision for values outside the factored form's range.
static __device__ __noinline__ double lanes_collide_cm_general(const SiteLane& g, double f, double rho, double ux,
                                                               double uy, double Fx, double Fy, double omega,
                                                               double cs) {
    double a[9], fs[9], r = 0.0;
#pragma unroll
    for (int v = 0; v < 9; v++) a[v] = lane_get(f, g.base + v);
    collide_cm<false>(a, rho, ux, uy, Fx, Fy, omega, cs, fs);
#pragma unroll
    for (int v = 0; v < 9; v++) r = v == g.v ? fs[v] : r;
    return r;
}

// collide<CM>() of this lane's population
template <bool CM>
__device__ __forceinline__ double lanes_collide(const SiteLane& g, double f, double rho, double ux, double uy,
                                                double Fx, double Fy, double omega, double cs) {
    const bool forced = (div_bits(Fx) << 1) != 0ull || (div_bits(Fy) << 1) != 0ull;
    if (!CM) {
        const double feq = lanes_equilibrium<false>(g, rho, ux, uy);
        double a = f + omega * (feq - f);
        if (__any_sync(kAllLanes, forced)) {
            const double cu = sel(g.cx == 0, 0.0, sgn_c(g.cx, ux)) + sel(g.cy == 0, 0.0, sgn_c(g.cy, uy));
            const double c3x = sgn_c(g.cx, 3.0), c3y = sgn_c(g.cy, 3.0);
            const double tx = g.cx == 0 ? -ux : ((double)g.cx - ux) + c3x * cu;
            const double ty = g.cy == 0 ? -uy : ((double)g.cy - uy) + c3y * cu;
            const double G = 3.0 * wgt(g.v) * (Fx * tx + Fy * ty);
            if (forced) a = a + (1.0 - 0.5 * omega) * G;
        }
        return a;
    }
    // k4Pre and k5Pre: the terms on their lanes, the two ordered sums on the
    // even and the odd lanes
    const double cx = (double)g.cx - ux, cy = (double)g.cy - uy;
    const double t4 = f * (LSQ(cx) - LSQ(cy)), t5 = f * cx * cy;
    double acc = 0.0;
#pragma unroll
    for (int q = 0; q < 9; q++) {
        const double x4 = lane_get(t4, g.base + q), x5 = lane_get(t5, g.base + q);
        const double x = (g.v & 1) ? x5 : x4;
        acc = q == 0 ? x : acc + x;
    }
    acc = pos_zero(acc);
    CmSite c;
    cm_site<false>(c, rho, ux, uy, Fx, Fy, lane_get(acc, g.base), lane_get(acc, g.base + 1), omega, cs);
    if (!__all_sync(kAllLanes, cm_factored_ok(c)))
        return lanes_collide_cm_general(g, f, rho, ux, uy, Fx, Fy, omega, cs);
    // (with any site forced the force terms are formed for all three; for an
    // unforced site they are exact zeros added to a non-zero sum)
    return cm_population(g.cx, g.cy, c, __any_sync(kAllLanes, forced));
}

// Site q of the perimeter: bottom row, top row, left column, right column.
__device__ __forceinline__ bool perimeter_ij(const LatDev& L, int q, int& i, int& j) {
    const int Nx = L.Nx, Ny = L.Ny;
    if (q < Nx) { i = q; j = 0; }
    else if (q < 2 * Nx) { i = q - Nx; j = Ny - 1; }
    else if (q < 2 * Nx + (Ny - 2)) { i = 0; j = q - 2 * Nx + 1; }
    else if (q < 2 * Nx + 2 * (Ny - 2)) { i = Nx - 1; j = q - 2 * Nx - (Ny - 2) + 1; }
    else return false;
    return true;
}

// boundary_site() for the warp's three sites (`site`: whether this lane's is one).
template <bool CM, class S>
__device__ __forceinline__ void lanes_boundary(const typename S::T* __restrict__ A, typename S::T* __restrict__ B,
                                               const LatDev& L, int t, bool site, int i, int j) {
    const SiteLane g = site_lane();
    const int type = site ? site_type(L, i, j) : LIFE_FLUID;
    if (!__any_sync(kAllLanes, type != LIFE_FLUID)) return;
    const bool store = g.store && type != LIFE_FLUID;
    double f, rho, ux, uy;
    lanes_state<CM, S, true>(A, L, t, g, i, j, f, rho, ux, uy);
    if (store && L.convective) {
        const int c = i - (L.Nx - 3);
        if (c >= 0 && g.v == 0) {
            L.outlet_u[((size_t)c * L.Ny + j) * 2 + 0] = ux;
            L.outlet_u[((size_t)c * L.Ny + j) * 2 + 1] = uy;
        }
        if (i == L.Nx - 1 && g.cx < 0) L.outlet_f_next[(size_t)j * 3 + (g.v == 2 ? 0 : (g.v == 6 ? 1 : 2))] = f;
    }
    if (store && g.v == 0) store_history(L, type, i, j, rho, ux, uy);
    double Fx, Fy;
    force_xy_next(L, t + 1, rho, Fx, Fy);
    const double fs = lanes_collide<CM>(g, f, rho, ux, uy, Fx + 0.0, Fy + 0.0, L.omega, L.cs);
    if (store) B[(size_t)g.v * L.S + (size_t)j * L.pitch + i] = S::save(fs, g.v);
}

}  // namespace life
