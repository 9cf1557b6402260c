// Immersed-boundary kernels (FP64), rigid and flexible markers.
//
//   k_ibm_interp    one warp per marker: rho and rho*u at the marker's
//                   support sites (reconstructed from P_t exactly as the step
//                   kernel computed them), then the direct force
//                   (IBMNodeClass::interpolate + forceCalc,
//                   reference src/IBMNode.cpp:26-58)
//   k_ibm_mark      list every site that some marker's support touches, once,
//                   and zero last step's IBM force at its support sites (for
//                   rigid markers the interpolation's warps do this)
//   k_ibm_spread    three listed sites per warp: each sums the contributions
//                   of the markers that reach it in marker order (the
//                   reference's ORDERED reduction, src/IBMNode.cpp:61-94)
//                   without atomics, applies the IBM velocity correction
//                   (updateMacroscopic, src/IBMNode.cpp:97-136) and collides
//                   the site again for the next step with the IBM force.
#include <cuda_runtime.h>

#include "collide_cm.cuh"
#include "ibm_kernels.h"
#include "lbm_device.cuh"
#include "lbm_lanes.cuh"

namespace life {

// Zero last step's IBM force at its support sites (thread q of `threads`).
__device__ __forceinline__ void clear_force(const IbmScratch& W, const LatDev& L, int q, int threads) {
    const int n = *W.nsites_prev;
    for (; q < n; q += threads) {
        const long long s = W.sites_prev[q];
        W.force_ibm[s] = 0.0;
        W.force_ibm[L.S + s] = 0.0;
    }
}

// List the support site (i, j), if no other entry has, and widen its range's
// support box by the marker's (once per marker: `first`).
__device__ __forceinline__ void mark_site(const IbmScratch& W, const LatDev& L, int k, int i, int j, bool first,
                                          const int4& bb) {
    const long long s = (long long)j * L.pitch + i;
    const unsigned bit = 1u << (s & 31);
    if (!(atomicOr(&W.site_flag[s >> 5], bit) & bit)) W.sites[atomicAdd(W.nsites, 1)] = s;
    if (first) {
        int4* box = W.range_box + W.range_of[k];
        atomicMin(&box->x, bb.x);
        atomicMax(&box->y, bb.y);
        atomicMin(&box->z, bb.z);
        atomicMax(&box->w, bb.w);
    }
}

// One warp per marker: lane s reconstructs support site s, and lanes 0, 1 and 2
// add the nsupp terms of rho, rho ux and rho uy in support order (the
// reference's loop), so the sums are formed exactly as in a sequential loop while
// the nine site states are computed side by side. (A lane past nsupp holds +0,
// which changes no sum that starts at +0.) MARK: also the work of k_ibm_mark (the
// markers do not move before the spread), by a second warp per marker: its
// atomics, each waiting for the one before, used to stand in front of the sums.
// A block per marker, so that a body's markers do not share an SM's FP64 unit: the
// kernel is bound by the chain of one warp (126 markers of the 1000 x 400 cylinder:
// 11.0 -> 8.8 us cold).
template <bool CM, class S, bool MARK>
__global__ void __launch_bounds__(MARK ? 64 : 32) k_ibm_interp(const typename S::T* __restrict__ P, LatDev L, int t,
                                                               MarkerDev M, IbmScratch W, double velScale,
                                                               const int* __restrict__ t_dev) {
    const int k = blockIdx.x;
    const int lane = threadIdx.x & 31;
    const int e = k * 9 + (lane < 9 ? lane : 0);
    const int ns = M.nsupp[k];
    const bool act = lane < ns;
    const int i = M.si[e], j = M.sj[e];
    const double d = M.sd[e], vel = lane == 1 || lane == 2 ? M.vel[k * 2 + lane - 1] : 0.0;
    const int imin = __reduce_min_sync(kAllLanes, act ? i : (1 << 30));
    const int imax = __reduce_max_sync(kAllLanes, act ? i : -(1 << 30));
    if (!MARK || threadIdx.x >= 32) {
        const int jmin = __reduce_min_sync(kAllLanes, act ? j : (1 << 30));
        const int jmax = __reduce_max_sync(kAllLanes, act ? j : -(1 << 30));
        const int4 bb = make_int4(imin, imax, jmin, jmax);
        if (lane == 0) M.bbox[k] = bb;
        if (MARK) {
            clear_force(W, L, k * 32 + lane, (int)gridDim.x * 32);
            if (act) mark_site(W, L, k, i, j, lane == 0, bb);
            return;
        }
    }
    t = t_dev ? *t_dev : step_t(L, t);  // inside a replayed graph the step comes from the device
    // support sites on a convective outlet: its speed term, formed here too
    // (nothing of this step has to be finished before the interpolation)
    double dU[2] = {0.0, 0.0};
    const bool form = L.convective && L.outlet_form == kOutletSites;
    if (form && imax == L.Nx - 1) {
        const double uOut = lanes_outlet_mean<S::prec == LIFE_PREC_F64>(L);
        if (act) outlet_term(L, uOut, j, dU[0], dU[1]);
    }
    double tr = 0.0, tx = 0.0, ty = 0.0;
    if (act) {
        double f[9], rho, ux, uy;
        site_state<CM, S>(P, L, t, i, j, f, rho, ux, uy, form ? dU : nullptr);
        tr = rho * d * 1.0 * 1.0;
        tx = rho * ux * d * 1.0 * 1.0;
        ty = rho * uy * d * 1.0 * 1.0;
    }
    double acc = 0.0;
#pragma unroll
    for (int q = 0; q < 9; q++) {
        const double r = lane_get(tr, q), x = lane_get(tx, q), y = lane_get(ty, q);
        acc += lane == 0 ? r : (lane == 1 ? x : y);
    }
    const double sc = velScale * lane_get(acc, 0);
    const double force = 2.0 * (sc * vel - acc);
    if (lane == 1 || lane == 2) M.force[k * 2 + lane - 1] = force;
}

// One thread per support entry: the first to set a site's bit lists the site.
__global__ void k_ibm_mark(MarkerDev M, IbmScratch W, LatDev L) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    clear_force(W, L, q, (int)(gridDim.x * blockDim.x));
    const int k = q / 9, e = q - 9 * k;
    if (k >= M.n || e >= M.nsupp[k]) return;
    mark_site(W, L, k, M.si[q], M.sj[q], e == 0, M.bbox[k]);
}

// One warp takes three listed sites, nine lanes each (lbm_lanes.cuh). The
// lanes scan the ranges of markers whose support box reaches one of the sites (in
// order) 32 markers at a time for all three sites; a marker that reaches a
// site leaves its contribution in shared memory, and one lane per site and
// component adds the chunk's contributions in marker order. The few hundred
// sites of a body are one warp's work on each SM, not a few warps' on the SMs
// that own their tiles: with one CTA per touched 16 x 16 tile and one thread
// per site (a chain of 700-900 FP64 instructions of 64 cycles) the kernel took
// 44 us for the 126 markers of the 1000 x 400 cylinder (central moments, FP32
// storage), 14.5 us now; 41 us for a circle and its tail of 132 markers (BGK,
// FP64), 12 us now. Bound by the latency of one chain: a second warp of the block
// forms the site's populations, their sums and the reciprocal of the density while
// the first scans the markers (15.9 us with one warp for both).
__device__ __forceinline__ bool box_has(const int4& b, int i, int j) {
    return i >= b.x && i <= b.y && j >= b.z && j <= b.w;
}

template <bool CM, class S>
__global__ void __launch_bounds__(64) k_ibm_spread(const typename S::T* __restrict__ A, typename S::T* __restrict__ B,
                                                   LatDev L, int t, MarkerDev M, IbmScratch W) {
    __shared__ double s_c[kLaneSites][2][32];
    __shared__ double s_a[kLaneSites][2];
    const int lane = threadIdx.x & 31;
    const bool scans = threadIdx.x < 32;
    const SiteLane g = site_lane();
    t = step_t(L, t);
    const int nsites = *W.nsites;
    // the next step's list starts empty
    if (blockIdx.x == 0 && scans) {
        if (lane == 0) *W.nsites_prev = 0;
        for (int b = lane; b < W.nranges; b += 32)
            W.range_box_next[b] = make_int4(0x7fffffff, -0x7fffffff, 0x7fffffff, -0x7fffffff);
    }
    for (int q0 = kLaneSites * (int)blockIdx.x; q0 < nsites; q0 += kLaneSites * (int)gridDim.x) {
        // this lane's site; a missing one repeats the first and is not stored
        const bool on = q0 + g.slot < nsites;
        const long long s = W.sites[on ? q0 + g.slot : q0];
        const int j = (int)(s / L.pitch), i = (int)(s - (long long)j * L.pitch);
        const bool store = on && g.store;
        double Fx = 0.0, Fy = 0.0, f = 0.0, m = 0.0, rho = 0.0, y = 0.0;
        if (!scans) {
            f = lanes_populations<CM, S>(A, L, t, g, i, j, Fx, Fy);
            m = lanes_sums(g, f);
            rho = lane_get(m, g.base);
            y = __drcp_rn(rho);
        } else {
            int is[kLaneSites], js[kLaneSites];
#pragma unroll
            for (int c = 0; c < kLaneSites; c++) {
                is[c] = __shfl_sync(kAllLanes, i, 9 * c);
                js[c] = __shfl_sync(kAllLanes, j, 9 * c);
            }
            // lanes 0 and 1 of a site sum the x and the y force
            const int comp = g.v == 1 ? 1 : 0;
            double acc = 0.0;
            for (int b0 = 0; b0 < W.nranges; b0 += 32) {
                bool near = false;
                if (b0 + lane < W.nranges) {
                    const int4 box = W.range_box[b0 + lane];
                    near = box_has(box, is[0], js[0]) || box_has(box, is[1], js[1]) || box_has(box, is[2], js[2]);
                }
                unsigned ranges = __ballot_sync(kAllLanes, near);
                while (ranges) {
                    const int b = b0 + __ffs(ranges) - 1;
                    ranges &= ranges - 1;
                    const int kbeg = W.range_start[b], kend = W.range_start[b + 1];
                    // the support box of the next chunk's marker comes while this
                    // chunk's is looked at, and what a hit needs with its entries
                    int4 next = kbeg + lane < kend ? M.bbox[kbeg + lane] : make_int4(0, -1, 0, -1);
                    for (int k0 = kbeg; k0 < kend; k0 += 32) {
                        const int k = k0 + lane;
                        const int4 bb = next;
                        next = k + 32 < kend ? M.bbox[k + 32] : make_int4(0, -1, 0, -1);
                        int at[kLaneSites];  // this marker's support entry at each site
                        bool any = false;
                        double mx = 0.0, my = 0.0, me = 0.0, ds = 0.0;
#pragma unroll
                        for (int c = 0; c < kLaneSites; c++) at[c] = -1;
                        if (k < kend) {
                            if (box_has(bb, is[0], js[0]) || box_has(bb, is[1], js[1]) || box_has(bb, is[2], js[2])) {
                                const int ns = M.nsupp[k];
                                mx = M.force[k * 2];
                                my = M.force[k * 2 + 1];
                                me = M.eps[k];
                                ds = M.ds[k];
#pragma unroll
                                for (int e = 8; e >= 0; e--) {
                                    const int ei = M.si[k * 9 + e], ej = M.sj[k * 9 + e];
#pragma unroll
                                    for (int c = 0; c < kLaneSites; c++)
                                        if (e < ns && ei == is[c] && ej == js[c]) at[c] = e;
                                }
                                any = at[0] >= 0 || at[1] >= 0 || at[2] >= 0;
                            }
                        }
                        if (!__any_sync(kAllLanes, any)) continue;
                        double gx = 0.0, gy = 0.0;
                        if (any) {
                            gx = mx * me * ds * 1.0;
                            gy = my * me * ds * 1.0;
                        }
                        unsigned hits = 0;
#pragma unroll
                        for (int c = 0; c < kLaneSites; c++) {
                            const unsigned h = __ballot_sync(kAllLanes, at[c] >= 0);
                            if (c == g.slot) hits = h;
                            if (at[c] >= 0) {
                                const double d = M.sd[k * 9 + at[c]];
                                s_c[c][0][lane] = gx * d;
                                s_c[c][1][lane] = gy * d;
                            }
                        }
                        __syncwarp();
                        while (hits) {
                            acc = acc + s_c[g.slot][comp][__ffs(hits) - 1];
                            hits &= hits - 1;
                        }
                        __syncwarp();
                    }
                }
            }
            if (g.store && g.v < 2) s_a[g.slot][g.v] = acc;
        }
        __syncthreads();
        const double ax = s_a[g.slot][0], ay = s_a[g.slot][1];
        __syncthreads();  // (the next three sites' sums may come)
        if (scans) {
            if (store && g.v == 0) {
                W.force_ibm[s] = ax;
                W.force_ibm[L.S + s] = ay;
                atomicAnd(&W.site_flag[s >> 5], ~(1u << (s & 31)));
            }
            continue;
        }
        double ux, uy;
        lanes_velocity(g, m, rho, y, Fx + ax, Fy + ay, ux, uy);
        if (store && g.v == 0) {
            store_history(L, site_type(L, i, j), i, j, rho, ux, uy);
            if (L.convective && i >= L.Nx - 3) {
                const int c = i - (L.Nx - 3);
                L.outlet_u[((size_t)c * L.Ny + j) * 2 + 0] = ux;
                L.outlet_u[((size_t)c * L.Ny + j) * 2 + 1] = uy;
            }
        }
        double Gx, Gy;
        force_xy_next(L, t + 1, rho, Gx, Gy);
        const double fs = lanes_collide<CM>(g, f, rho, ux, uy, Gx + ax, Gy + ay, L.omega, L.cs);
        if (store) B[(size_t)g.v * L.S + s] = S::save(fs, g.v);
    }
}

// ObjectsClass::removeOverlapMarkers (src/Objects.cpp:873-884): every marker
// pair n1 < n2 whose distance is below half a lattice spacing, with the
// reference's arithmetic (sum of squares from +0, square root, division).
// Block n1 (grid-stride) tests n2 > n1 on its threads; hits are appended in
// any order (the host sorts them) while the count stays within cap, and the
// count is returned in full so the host can retry with a larger list.
__global__ void k_overlap_pairs(const double* __restrict__ pos, int nm, double Dx, int* __restrict__ count,
                                int2* __restrict__ out, int cap) {
    for (int n1 = blockIdx.x; n1 < nm; n1 += gridDim.x) {
        const double x1 = pos[2 * n1], y1 = pos[2 * n1 + 1];
        for (int n2 = n1 + 1 + (int)threadIdx.x; n2 < nm; n2 += blockDim.x) {
            const double d0 = x1 - pos[2 * n2], d1 = y1 - pos[2 * n2 + 1];
            double dd = 0.0;
            dd += d0 * d0;
            dd += d1 * d1;
            if (sqrt(dd) / Dx < 0.5) {
                const int k = atomicAdd(count, 1);
                if (k < cap) out[k] = make_int2(n1, n2);
            }
        }
    }
}

cudaError_t launch_overlap_pairs(const double* pos, int nm, double Dx, int* count, int2* out, int cap,
                                 cudaStream_t s) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int grid = nm < 8 * sms ? (nm > 0 ? nm : 1) : 8 * sms;
    k_overlap_pairs<<<grid, 256, 0, s>>>(pos, nm, Dx, count, out, cap);
    return cudaGetLastError();
}

// ------------------------------------------------------------ launchers
#define IBM_DISPATCH(KERNEL, GRID, BLOCK, ...)                                                             \
    do {                                                                                                   \
        if (L.prec == LIFE_PREC_F64) {                                                                     \
            if (L.cm) KERNEL<true, StoreF64><<<GRID, BLOCK, 0, s>>>(__VA_ARGS__);                          \
            else KERNEL<false, StoreF64><<<GRID, BLOCK, 0, s>>>(__VA_ARGS__);                              \
        } else if (L.prec == LIFE_PREC_F32) {                                                              \
            if (L.cm) KERNEL<true, StoreF32><<<GRID, BLOCK, 0, s>>>(__VA_ARGS__);                          \
            else KERNEL<false, StoreF32><<<GRID, BLOCK, 0, s>>>(__VA_ARGS__);                              \
        } else {                                                                                           \
            if (L.cm) KERNEL<true, StoreF16><<<GRID, BLOCK, 0, s>>>(__VA_ARGS__);                          \
            else KERNEL<false, StoreF16><<<GRID, BLOCK, 0, s>>>(__VA_ARGS__);                              \
        }                                                                                                  \
    } while (0)

template <class T>
struct TypedPtr {
    const void* p;
    template <class U>
    operator const U*() const { return (const U*)p; }
    template <class U>
    operator U*() const { return (U*)const_cast<void*>(p); }
};

cudaError_t launch_ibm_interp(const void* P, const LatDev& L, int t, const MarkerDev& M, const IbmScratch* mark,
                              double velScale, cudaStream_t s, const int* t_dev) {
    if (M.n == 0) return cudaSuccess;
    TypedPtr<void> Pp{P};
#define LIFE_INTERP(CM, S)                                                                              \
    do {                                                                                                \
        if (mark) k_ibm_interp<CM, S, true><<<M.n, 64, 0, s>>>(Pp, L, t, M, *mark, velScale, t_dev);     \
        else k_ibm_interp<CM, S, false><<<M.n, 32, 0, s>>>(Pp, L, t, M, IbmScratch{}, velScale, t_dev);  \
    } while (0)
    if (L.prec == LIFE_PREC_F64) {
        if (L.cm) LIFE_INTERP(true, StoreF64);
        else LIFE_INTERP(false, StoreF64);
    } else if (L.prec == LIFE_PREC_F32) {
        if (L.cm) LIFE_INTERP(true, StoreF32);
        else LIFE_INTERP(false, StoreF32);
    } else {
        if (L.cm) LIFE_INTERP(true, StoreF16);
        else LIFE_INTERP(false, StoreF16);
    }
#undef LIFE_INTERP
    return cudaGetLastError();
}

cudaError_t launch_ibm_mark(const LatDev& L, const MarkerDev& M, const IbmScratch& W, cudaStream_t s) {
    if (M.n == 0) return cudaSuccess;
    k_ibm_mark<<<(9 * M.n + 127) / 128, 128, 0, s>>>(M, W, L);
    return cudaGetLastError();
}

cudaError_t launch_ibm_spread(const void* A, void* B, const LatDev& L, int t, const MarkerDev& M,
                              const IbmScratch& W, cudaStream_t s) {
    if (M.n == 0) return cudaSuccess;
    // a warp per three sites, nine sites per marker at most; beyond 4096
    // blocks (about 27 per SM) a block takes further sites in turn
    const int grid = 3 * M.n < 4096 ? 3 * M.n : 4096;
    TypedPtr<void> Ap{A}, Bp{B};
    IBM_DISPATCH(k_ibm_spread, grid, 64, Ap, Bp, L, t, M, W);
    return cudaGetLastError();
}

}  // namespace life
