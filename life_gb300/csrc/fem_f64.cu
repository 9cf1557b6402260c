// Flexible-body kernels (FP64, --fmad=false, reference operation order).
//
// One CTA per flexible body runs the FEM work of that body:
//   k_fsi_predict   predictor (first subiteration) or Aitken relaxation,
//                   then updateFEMValues / finishNewmark / updateIBMValues
//                   (FEMBodyClass::predictor, src/FEMBody.cpp:259-289;
//                   ObjectsClass::recomputeObjectVals, src/Objects.cpp:152-232)
//   k_fem_dynamic   FEMBodyClass::dynamicFEM (src/FEMBody.cpp:26-68): load
//                   vector, Newton-Raphson with Newmark and the dense LU solve,
//                   marker update, subiteration residual
// and
//   k_fsi_support   findSupport + computeDs of flexible markers
//   k_fsi_epsilon   epsilon systems (per flexible body or all markers)
//   k_fsi_residual  femKernel's ordered residual sums, the loop condition and
//                   the next Aitken factor (src/Objects.cpp:63-99, 179-190)
//
// Element matrices are computed in parallel and assembled entry by entry in
// element order, the order of the reference's sequential assembly. Products
// with the element rotation T skip its structural zeros; a skipped term is an
// exact zero, so results are unchanged.
#include <cuda_runtime.h>

#include <atomic>

#include "band_lu.h"
#include "crtrig.h"
#include "div_rn.cuh"
#include "fem_kernels.h"

namespace life {

#define DSQ(x) ((x) * (x))
#define DTH(x) ((x) * (x) * (x))
__device__ constexpr double kPI = 3.14159265358979323846;

__device__ __forceinline__ double* vec(FemBodyDev& B, int name) { return B.pool + (size_t)B.slots[name] * B.n; }

__device__ __forceinline__ double shift_angle_d(double a) {
    a = fmod(a + kPI, 2.0 * kPI);
    if (a < 0.0) a += 2.0 * kPI;
    return a - kPI;
}

// diracDelta (inc/Utils.h:220-232): beyond 1/2 (5 - 3 a - sqrt(1 - 3 (1-a)^2)) / 6,
// else (1 + sqrt(1 - 3 a^2)) / 3. Lanes differ in the branch, so both take one
// root and one quotient (-3 x + 1 and 1 - 3 x round alike).
__device__ __forceinline__ double dirac_d(double dist) {
    const double a = fabs(dist);
    if (a > 1.5) return 0.0;
    const bool outer = a > 0.5;
    const double t = outer ? 1.0 - a : a;
    const double root = sqrt(1.0 - 3.0 * DSQ(t));
    const double num = (outer ? 5.0 - 3.0 * a : 1.0) + (outer ? -root : root);
    return num / (outer ? 6.0 : 3.0);
}

// Element rotation T = diag(R, R), R = [[c, s, 0], [-s, c, 0], [0, 0, 1]]
// (FEMElementClass::setElementTransform, src/FEMElement.cpp:255-262).
__host__ __device__ constexpr bool tnz(int i, int j) {
    return (i < 2 && j < 2) || (i == 2 && j == 2) || (i >= 3 && i < 5 && j >= 3 && j < 5) || (i == 5 && j == 5);
}
__device__ __forceinline__ double tval(int i, int j, double c, double s) {
    const int a = i % 3, b = j % 3;
    if (a == 2) return 1.0;
    if (a == 0) return b == 0 ? c : s;
    return b == 0 ? -s : c;
}

// Structurally non-zero entries of the local element matrices, bit 6 i + j: the
// mass and linear stiffness matrices couple the axial displacements {0, 3} and
// the bending ones {1, 2, 4, 5} separately; the geometric stiffness couples the
// displacements {0, 1, 3, 4} without the axial pairs.
__host__ __device__ constexpr unsigned long long pattern(bool geometric) {
    unsigned long long m = 0;
    for (int i = 0; i < 6; i++)
        for (int j = 0; j < 6; j++) {
            const bool nz = geometric ? i % 3 != 2 && j % 3 != 2 && (i % 3 == 1 || j % 3 == 1) : (i % 3 == 0) == (j % 3 == 0);
            if (nz) m |= 1ull << (6 * i + j);
        }
    return m;
}
// +0 + x (which is x but for the sign of a zero), without the FP64 unit
__device__ __forceinline__ double from_zero(double x) {
    return (unsigned long long)__double_as_longlong(x) == 0x8000000000000000ull ? 0.0 : x;
}

// out = T^T A T with the reference's summation order over non-zero terms of T
// and of A (pattern MASK); the other terms are exact zeros.
template <unsigned long long MASK>
__device__ __forceinline__ void tt_a_t(const double* A, double c, double s, double* out) {
    double R1[36];
    bool full[36];
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
        for (int j = 0; j < 6; j++) {
            double acc = 0.0;
            bool any = false;
#pragma unroll
            for (int k = 0; k < 6; k++)
                if (tnz(k, i) && ((MASK >> (6 * k + j)) & 1)) {
                    const double x = tval(k, i, c, s) * A[k * 6 + j];
                    acc = any ? acc + x : from_zero(x);
                    any = true;
                }
            R1[i * 6 + j] = acc;
            full[i * 6 + j] = any;
        }
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
        for (int j = 0; j < 6; j++) {
            double acc = 0.0;
            bool any = false;
#pragma unroll
            for (int k = 0; k < 6; k++)
                if (tnz(k, j) && full[i * 6 + k]) {
                    const double x = R1[i * 6 + k] * tval(k, j, c, s);
                    acc = any ? acc + x : from_zero(x);
                    any = true;
                }
            out[i * 6 + j] = acc;
        }
}

// FEMBodyClass::updateFEMValues (src/FEMBody.cpp:198-223). The CTA's last warp
// runs `side` while the others evaluate the elements.
struct NoSideTask {
    __device__ void operator()() const {}
};
template <class Side = NoSideTask>
__device__ __forceinline__ void update_fem_values(FemBodyDev& B, Side side = Side{}) {
    const double* U = vec(B, V_U);
    for (int n = threadIdx.x; n < B.nNodes; n += blockDim.x) {
        double* nd = B.node + n * 6;
        nd[2] = nd[0] + U[n * 3 + 0];
        nd[3] = nd[1] + U[n * 3 + 1];
        nd[5] = nd[4] + U[n * 3 + 2];
    }
    __syncthreads();
    const int workers = (int)blockDim.x - 32;
    if ((int)threadIdx.x >= workers) side();
    for (int e = threadIdx.x; e < B.nEl && (int)threadIdx.x < workers; e += workers) {
        const double* n0 = B.node + e * 6;
        const double* n1 = B.node + (e + 1) * 6;
        const double ev0 = n1[2] - n0[2], ev1 = n1[3] - n0[3];
        double* el = B.el + (size_t)e * EL_STRIDE;
        // correctly rounded trigonometry (crtrig.h): the same bits on every
        // device and on a host checker
        const double ang = life_cr_atan2(ev1, ev0);
        double dd = 0.0;
        dd += ev0 * ev0;
        dd += ev1 * ev1;
        el[EL_ANG] = ang;
        el[EL_L] = sqrt(dd);
        double sa, ca;
        life_cr_sincos(ang, &sa, &ca);
        el[EL_COS] = ca;
        el[EL_SIN] = sa;
    }
    __syncthreads();
}

// FEMBodyClass::finishNewmark (src/FEMBody.cpp:129-144)
__device__ void finish_newmark(FemBodyDev& B, const FsiDev& F) {
    const double Dt = F.Dt, al = F.alpha, de = F.delta;
    const double a6 = 1.0 / (al * DSQ(Dt)), a7 = -1.0 / (al * Dt), a8 = -(1.0 / (2.0 * al) - 1.0);
    const double a9 = Dt * (1.0 - de), a10 = de * Dt;
    double* U = vec(B, V_U);
    double* Un = vec(B, V_Un);
    double* Ud = vec(B, V_Udot);
    double* Udd = vec(B, V_Udotdot);
    double* Udn = vec(B, V_Udotn);
    double* Uddn = vec(B, V_Udotdotn);
    for (int i = threadIdx.x; i < B.n; i += blockDim.x) {
        const double udd = a6 * (U[i] - Un[i]) + a7 * Udn[i] + a8 * Uddn[i];
        Udd[i] = udd;
        Ud[i] = Udn[i] + a9 * Uddn[i] + a10 * udd;
    }
    __syncthreads();
}

// FEMElementClass::shapeFuns (src/FEMElement.cpp:141-160)
__device__ __forceinline__ void shape_funs_d(double res[2], const double v[6], double zeta, double L) {
    const double N0 = 1.0 - (zeta + 1.0) / 2.0;
    const double N1 = 1.0 - 3.0 * DSQ((zeta + 1.0) / 2.0) + 2.0 * DTH((zeta + 1.0) / 2.0);
    const double N2 = ((zeta + 1.0) / 2.0 - 2.0 * DSQ((zeta + 1.0) / 2.0) + DTH((zeta + 1.0) / 2.0)) * L;
    const double N3 = (zeta + 1.0) / 2.0;
    const double N4 = 3.0 * DSQ((zeta + 1.0) / 2.0) - 2.0 * DTH((zeta + 1.0) / 2.0);
    const double N5 = (-DSQ((zeta + 1.0) / 2.0) + DTH((zeta + 1.0) / 2.0)) * L;
    res[0] = v[0] * N0 + v[3] * N3;
    res[1] = v[1] * N1 + v[2] * N2 + v[4] * N4 + v[5] * N5;
}

// T * v over non-zero entries of T.
__device__ __forceinline__ void t_vec(const double v[6], double c, double s, double out[6]) {
#pragma unroll
    for (int i = 0; i < 6; i++) {
        double acc = 0.0;
#pragma unroll
        for (int j = 0; j < 6; j++)
            if (tnz(i, j)) acc += tval(i, j, c, s) * v[j];
        out[i] = acc;
    }
}
// T^T * v over non-zero entries of T.
__device__ __forceinline__ void tt_vec(const double v[6], double c, double s, double out[6]) {
#pragma unroll
    for (int i = 0; i < 6; i++) {
        double acc = 0.0;
#pragma unroll
        for (int j = 0; j < 6; j++)
            if (tnz(j, i)) acc += tval(j, i, c, s) * v[j];
        out[i] = acc;
    }
}

// FEMBodyClass::updateIBMValues (src/FEMBody.cpp:147-195)
__device__ void update_ibm(FemBodyDev& B, const MarkerDev& M) {
    const double* U = vec(B, V_U);
    const double* Ud = vec(B, V_Udot);
    for (int i = threadIdx.x; i < B.nMark; i += blockDim.x) {
        const int e = B.mapEl[i];
        const double zeta = B.mapZeta[i];
        const double* el = B.el + (size_t)e * EL_STRIDE;
        const double c = el[EL_COS], s = el[EL_SIN], ang = el[EL_ANG], L = el[EL_L];
        double dU[6], dUd[6];
#pragma unroll
        for (int k = 0; k < 6; k++) {
            dU[k] = U[3 * e + k];
            dUd[k] = Ud[3 * e + k];
        }
        const double* nd0 = B.node + e * 6;
#pragma unroll
        for (int n = 0; n < 2; n++) {
            const double* nd = B.node + (e + n) * 6;
            dU[n * 3 + 0] += nd[0] - nd0[2];
            dU[n * 3 + 1] += nd[1] - nd0[3];
            dU[n * 3 + 2] += nd[4] - ang;
            dU[n * 3 + 2] = shift_angle_d(dU[n * 3 + 2]);
        }
        double lU[6], lUd[6], sU[2], sUd[2];
        t_vec(dU, c, s, lU);
        t_vec(dUd, c, s, lUd);
        shape_funs_d(sU, lU, zeta, L);
        shape_funs_d(sUd, lUd, zeta, L);
        const double gU0 = (0.0 + c * sU[0]) + (-s) * sU[1];
        const double gU1 = (0.0 + s * sU[0]) + c * sU[1];
        const double gV0 = (0.0 + c * sUd[0]) + (-s) * sUd[1];
        const double gV1 = (0.0 + s * sUd[0]) + c * sUd[1];
        const int k = B.mbase + i;
        M.pos[k * 2 + 0] = nd0[2] + gU0;
        M.pos[k * 2 + 1] = nd0[3] + gU1;
        M.vel[k * 2 + 0] = gV0;
        M.vel[k * 2 + 1] = gV1;
    }
    __syncthreads();
}

__device__ __forceinline__ void swap_slots(FemBodyDev& B, int a, int b) {
    const int t = B.slots[a];
    B.slots[a] = B.slots[b];
    B.slots[b] = t;
}

// Predictor (subiteration 0) or relaxation (later subiterations).
__global__ void __launch_bounds__(256) k_fsi_predict(FsiDev F, MarkerDev M) {
    FemBodyDev& B = F.bodies[blockIdx.x];
    const int subIt = F.s->subIt;
    const int t = F.s->t;
    if (subIt == 0) {
        if (threadIdx.x == 0) {
            // FEMBodyClass::resetValues (src/FEMBody.cpp:341-349)
            swap_slots(B, V_Unm2, V_Unm1);
            swap_slots(B, V_Unm1, V_Un);
            swap_slots(B, V_Un, V_U);
            swap_slots(B, V_Udotn, V_Udot);
            swap_slots(B, V_Udotdotn, V_Udotdot);
        }
        __syncthreads();
        double* U = vec(B, V_U);
        const double* Un = vec(B, V_Un);
        const double* Unm1 = vec(B, V_Unm1);
        const double* Unm2 = vec(B, V_Unm2);
        for (int i = threadIdx.x; i < B.n; i += blockDim.x) {
            if (t > 2) U[i] = 2.5 * Un[i] - 2.0 * Unm1[i] + 0.5 * Unm2[i];
            else if (t == 2) U[i] = 2.0 * Un[i] - Unm1[i];
            else if (t == 1) U[i] = Un[i];
        }
    } else {
        const double relax = F.s->relax;
        double* U = vec(B, V_U);
        const double* Uk = vec(B, V_Ukm1);
        for (int i = threadIdx.x; i < B.n; i += blockDim.x) U[i] = Uk[i] + relax * (U[i] - Uk[i]);
    }
    __syncthreads();
    update_fem_values(B);
    finish_newmark(B, F);
    update_ibm(B, M);
    if (threadIdx.x == 0) swap_slots(B, V_Ukm1, V_U);
}

// IBMNodeClass::findSupport + computeDs (src/IBMNode.cpp:139-204) for the
// markers of flexible bodies, one warp per marker. Lanes 0..24 test the 5 x 5
// lattice nodes around the nearest node, lane = 5*(i - inear + 2) + (j -
// jnear + 2), so the ballot packs the supporting nodes in the reference's
// loop order (i outer, j inner). The spacing ds is the minimum of sqrt(dd)/Dx
// over the body's other markers; correctly rounded sqrt and division are
// monotone, so it equals sqrt(min dd)/Dx, and the lanes only reduce dd.
__global__ void __launch_bounds__(128) k_fsi_support(FsiDev F, MarkerDev M) {
    const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (q >= F.nFlexMarkers) return;  // uniform per warp
    const int k = F.flexMarkers[q];
    const double Dx = F.Dx;
    const double px = M.pos[k * 2], py = M.pos[k * 2 + 1];
    const double sx = px / Dx, sy = py / Dx;
    const int inear = (int)round(sx), jnear = (int)round(sy);
    const int i = inear - 2 + lane / 5, j = jnear - 2 + lane % 5;
    double dX = 0.0, dY = 0.0;
    bool in = false;
    if (lane < 25) {
        dX = fabs(sx - i);
        dY = fabs(sy - j);
        in = dX < 1.5 && dY < 1.5 && i >= 0 && i <= F.Nx - 1 && j >= 0 && j <= F.Ny - 1;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, in);
    const int slot = __popc(bal & ((1u << lane) - 1u));
    const int total = __popc(bal);
    if (lane < 9) {
        M.si[k * 9 + lane] = 0;
        M.sj[k * 9 + lane] = 0;
        M.sd[k * 9 + lane] = 0.0;
    }
    __syncwarp();
    if (in && slot < 9) {
        M.si[k * 9 + slot] = i;
        M.sj[k * 9 + slot] = j;
        M.sd[k * 9 + slot] = dirac_d(dX) * dirac_d(dY);
    }
    if (lane == 0) {
        M.nsupp[k] = total < 9 ? total : 9;
        if (total > 9) atomicCAS(&F.status[0], 0, LIFE_ERR_SUPPORT);
    }
    const int b = F.markerBody[k];
    const int b0 = F.bodyStart[b], bn = F.bodyCount[b];
    // non-negative doubles order like their bit patterns; NaN never passes dd < best
    unsigned long long best = 0x7ff0000000000000ull;  // +inf
    for (int n = lane; n < bn; n += 32) {
        const int o = b0 + n;
        if (o != k) {
            const double d0 = px - M.pos[o * 2], d1 = py - M.pos[o * 2 + 1];
            double dd = 0.0;
            dd += d0 * d0;
            dd += d1 * d1;
            if (dd < __longlong_as_double((long long)best)) best = (unsigned long long)__double_as_longlong(dd);
        }
    }
    const unsigned bh = __reduce_min_sync(0xffffffffu, (unsigned)(best >> 32));
    const unsigned bl = __reduce_min_sync(0xffffffffu, (unsigned)(best >> 32) == bh ? (unsigned)best : 0xffffffffu);
    if (lane == 0) {
        const double mag = sqrt(__longlong_as_double((long long)(((unsigned long long)bh << 32) | bl))) / Dx;
        M.ds[k] = mag < 10.0 ? mag : 10.0;
    }
}

// Dense LU with band-limited loops (band_lu.h semantics) by one warp.
// M(i,j) = A[(bc+j)*dim + bc+i]. lmax[c] tracks the last row that can hold a
// multiplier of column c after row interchanges.
__device__ void warp_lu_factor(double* A, int dim, int bc, int kl, int ku, int* piv, int* lmax) {
    const int lane = threadIdx.x & 31;
    const int n = dim - bc;
    for (int c = lane; c < n; c += 32) lmax[c] = c;
    __syncwarp();
    for (int j = 0; j < n; j++) {
        const int imax = j + kl < n - 1 ? j + kl : n - 1;
        // first maximal |M(i,j)|, i in [j, imax] (LAPACK idamax semantics)
        int best = j;
        double bval = -1.0;
        for (int i0 = j; i0 <= imax; i0 += 32) {
            const int i = i0 + lane;
            double va = -1.0;
            int vi = i;
            if (i <= imax) va = fabs(lu_m(A, dim, bc, i, j));
            for (int o = 16; o > 0; o >>= 1) {
                const double oa = __shfl_down_sync(0xffffffffu, va, o);
                const int oi = __shfl_down_sync(0xffffffffu, vi, o);
                if (oa > va || (oa == va && oi < vi)) { va = oa; vi = oi; }
            }
            va = __shfl_sync(0xffffffffu, va, 0);
            vi = __shfl_sync(0xffffffffu, vi, 0);
            if (va > bval) { bval = va; best = vi; }
        }
        const int jp = best;
        if (lane == 0) piv[j] = jp;
        const double pv = lu_m(A, dim, bc, jp, j);
        if (pv != 0.0) {
            if (jp != j) {
                for (int k = lane; k < n; k += 32) {
                    const double tj = lu_m(A, dim, bc, j, k), tp = lu_m(A, dim, bc, jp, k);
                    if (k < j && tj != 0.0 && lmax[k] < jp) lmax[k] = jp;
                    lu_m(A, dim, bc, j, k) = tp;
                    lu_m(A, dim, bc, jp, k) = tj;
                }
                __syncwarp();
            }
            const double r = 1.0 / lu_m(A, dim, bc, j, j);
            for (int i = j + 1 + lane; i <= imax; i += 32) lu_m(A, dim, bc, i, j) *= r;
        }
        if (lane == 0 && lmax[j] < imax) lmax[j] = imax;
        __syncwarp();
        const int kmax = j + kl + ku < n - 1 ? j + kl + ku : n - 1;
        const int rows = imax - j, cols = kmax - j;
        for (int q = lane; q < rows * cols; q += 32) {
            const int i = j + 1 + q % rows, k = j + 1 + q / rows;
            const double t = -lu_m(A, dim, bc, j, k);
            lu_m(A, dim, bc, i, k) += lu_m(A, dim, bc, i, j) * t;
        }
        __syncwarp();
    }
}

// Transposed solve (lane 0); x has dim entries, the first bc zeroed.
__device__ void warp_lu_solve(const double* A_, int dim, int bc, int kl, int ku, const int* piv, const int* lmax,
                              const double* b, double* x) {
    const int lane = threadIdx.x & 31;
    double* A = const_cast<double*>(A_);
    const int n = dim - bc;
    for (int i = lane; i < bc; i += 32) x[i] = 0.0;
    for (int i = lane; i < n; i += 32) x[bc + i] = b[bc + i];
    __syncwarp();
    if (lane == 0) {
        double* y = x + bc;
        const int w = kl + ku;
        for (int i = 0; i < n; i++) {
            double t = y[i];
            for (int k = (i - w > 0 ? i - w : 0); k < i; k++) t -= lu_m(A, dim, bc, k, i) * y[k];
            y[i] = t / lu_m(A, dim, bc, i, i);
        }
        for (int i = n - 1; i >= 0; i--) {
            double t = y[i];
            const int kend = lmax[i];
            for (int k = i + 1; k <= kend; k++) t -= lu_m(A, dim, bc, k, i) * y[k];
            y[i] = t;
        }
        for (int i = n - 1; i >= 0; i--)
            if (piv[i] != i) {
                const double t = y[i];
                y[i] = y[piv[i]];
                y[piv[i]] = t;
            }
    }
    __syncwarp();
}


// ---------------------------------------------------------------------------
// Band LU in shared memory with the dense textbook arithmetic.
//
// M is nn x nn with kl sub- and ku super-diagonals; row i of Bd holds M(i, c)
// for c in [i-kl, i+kl+ku] at Bd[i*W + c - i + kl], W = 2*kl + ku + 1. The
// factorisation performs exactly the operations of the dense unblocked LU
// (first maximal pivot, reciprocal scaling, rank-1 update; band_lu.h), but
// like LAPACK's banded routine it does not move the multipliers of earlier
// columns when it swaps rows. The dense transposed solve reads each
// multiplier from the row where the later swaps would have carried it; the
// solve below follows each multiplier to that final row (Fp, updated swap by
// swap from the last step back), so it forms the same products and sums
// them in the same order as the dense solve. Results are bit-identical.
__device__ __forceinline__ double& bd(double* Bd, int W, int kl, int i, int c) { return Bd[i * W + c - i + kl]; }

// One warp; kl <= 31. Lane l holds the candidate M(j+l, j) of column j. The
// pivot is the first maximal magnitude (LAPACK idamax: a NaN in the first
// place wins, later NaNs never do); magnitudes are compared as bit patterns,
// which order like the values for non-negative doubles. Each candidate's
// reciprocal is formed while the pivot is being chosen and the pivot's is
// kept: the same correctly rounded 1/pivot as a division after the choice.
__device__ void band_factor_smem(double* Bd, int nn, int kl, int ku, int W, int* piv) {
    const int lane = threadIdx.x & 31;
    for (int j = 0; j < nn; j++) {
        const int imax = j + kl < nn - 1 ? j + kl : nn - 1;
        const int kmax = j + kl + ku < nn - 1 ? j + kl + ku : nn - 1;
        const bool valid = j + lane <= imax;
        const double v = valid ? bd(Bd, W, kl, j + lane, j) : 0.0;
        const double rc = 1.0 / v;
        unsigned long long key = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
        if (key > 0x7ff0000000000000ull) key = lane == 0 ? ~0ull : 0ull;
        const unsigned kh = (unsigned)(key >> 32), klo = (unsigned)key;
        const unsigned mh = __reduce_max_sync(0xffffffffu, valid ? kh : 0u);
        const bool c1 = valid && kh == mh;
        const unsigned ml = __reduce_max_sync(0xffffffffu, c1 ? klo : 0u);
        const int src = __ffs(__ballot_sync(0xffffffffu, c1 && klo == ml)) - 1;
        const int jp = j + src;
        const double pv = __shfl_sync(0xffffffffu, v, src);
        const double r = __shfl_sync(0xffffffffu, rc, src);
        if (lane == 0) piv[j] = jp;
        if (pv != 0.0) {
            if (jp != j) {
                for (int c = j + lane; c <= kmax; c += 32) {
                    const double t = bd(Bd, W, kl, j, c);
                    bd(Bd, W, kl, j, c) = bd(Bd, W, kl, jp, c);
                    bd(Bd, W, kl, jp, c) = t;
                }
                __syncwarp();
            }
            for (int i = j + 1 + lane; i <= imax; i += 32) bd(Bd, W, kl, i, j) *= r;
        }
        __syncwarp();
        const int rows = imax - j, cols = kmax - j;
        for (int q = lane; q < rows * cols; q += 32) {
            const int i = j + 1 + q % rows, k = j + 1 + q / rows;
            const double t = -bd(Bd, W, kl, j, k);
            bd(Bd, W, kl, i, k) += bd(Bd, W, kl, i, j) * t;
        }
        __syncwarp();
    }
}

__global__ void k_selftest_division(long long n, unsigned long long seed, unsigned long long* bad) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        // splitmix64 streams for the two operands; exponents over a wide range
        unsigned long long z = seed + 0x9e3779b97f4a7c15ull * (unsigned long long)(2 * q + 1);
        auto mix = [](unsigned long long x) {
            x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
            x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
            return x ^ (x >> 31);
        };
        const unsigned long long u = mix(z), v = mix(z + 0x9e3779b97f4a7c15ull);
        const unsigned long long w = mix(z ^ 0x5851f42d4c957f2dull);
        // exponent spread: mostly near 1, sometimes anywhere in the normal range
        const int span = (w & 7) == 0 ? 2000 : 80;
        const long long xa = (long long)(1023 + (long long)((w >> 8) % span) - span / 2);
        const long long xb = (long long)(1023 + (long long)((w >> 24) % span) - span / 2);
        // one pair in 16 has equal or almost equal significands (a quotient at 1)
        const unsigned long long ua = ((w >> 50) & 15) == 0 ? (u & 0x8000000000000000ull) | ((v + ((w >> 54) & 7) - 3) & 0xfffffffffffffull) : u;
        const unsigned long long ba = (ua & 0x800fffffffffffffull) | ((unsigned long long)(xa < 1 ? 1 : (xa > 2046 ? 2046 : xa)) << 52);
        const unsigned long long bb = (v & 0x800fffffffffffffull) | ((unsigned long long)(xb < 1 ? 1 : (xb > 2046 ? 2046 : xb)) << 52);
        // one numerator in 64 is a signed zero (the velocity of a site at rest)
        const double a = ((w >> 40) & 63) == 0 ? __longlong_as_double((long long)(u & 0x8000000000000000ull))
                                                : __longlong_as_double((long long)ba);
        const double b = __longlong_as_double((long long)bb);
        const double ref = a / b;
        const double got = div_rn_recip(a, b, __drcp_rn(b));
        if (__double_as_longlong(ref) != __double_as_longlong(got) && !(ref != ref && got != got)) atomicAdd(bad, 1ull);
        // the integer reciprocal and quotient, where they decide
        unsigned long long X;
        if (recip64(b, X)) {
            double r, i;
            if (recip_round(b, X, r) && __double_as_longlong(r) != __double_as_longlong(__drcp_rn(b))) atomicAdd(bad, 1ull);
            if (quotient_round(a, b, X, i) && __double_as_longlong(i) != __double_as_longlong(ref)) atomicAdd(bad, 1ull);
        }
    }
}

__device__ __forceinline__ void named_bar(int id, int nthreads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// First maximal |v| over the lanes with `valid` (LAPACK idamax: a NaN in
// lane 0 wins, later NaNs never do), as the lane index. Magnitudes are
// compared as bit patterns, which order like the values for non-negative
// doubles. Whole warp.
__device__ __forceinline__ int pick_pivot(double v, bool valid, int lane) {
    unsigned long long key = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    if (key > 0x7ff0000000000000ull) key = lane == 0 ? ~0ull : 0ull;
    const unsigned kh = (unsigned)(key >> 32), klo = (unsigned)key;
    const unsigned mh = __reduce_max_sync(0xffffffffu, valid ? kh : 0u);
    const bool c1 = valid && kh == mh;
    const unsigned ml = __reduce_max_sync(0xffffffffu, c1 ? klo : 0u);
    return __ffs(__ballot_sync(0xffffffffu, c1 && klo == ml)) - 1;
}

// Rows k0..k0+m-1 (m <= 32) of the forward substitution by one warp: y_k =
// t_k / U(k,k), and every row r in (k, k+w] subtracts U(k,r) y_k; lane r & 31
// holds t of row r. The reciprocals of the diagonal, a row per lane, come first;
// rcp[k] = RN(1 / U(k,k)). (The loads of a row stand before the chain of the
// row above it.)
__device__ __forceinline__ void forward_rows(double* Bd, int nn, int kl, int W, int w, int k0, int m, int lane,
                                             const double* rcp, double* y, double& t) {
    const double mine = lane < m ? bd(Bd, W, kl, k0 + lane, k0 + lane) : 0.0;
    unsigned long long mX;
    const bool mok = recip64(mine, mX);
    auto upper = [&](int k) {
        const int rr = k + 1 + ((lane - k - 1) & 31);
        return rr <= k + w && rr < nn ? bd(Bd, W, kl, k, rr) : 0.0;
    };
    double u = upper(k0);
    for (int q = 0; q < m; q++) {
        const int k = k0 + q, owner = k & 31, rr = k + 1 + ((lane - k - 1) & 31);
        const double ukk = __shfl_sync(0xffffffffu, mine, q), uk = u;
        const unsigned long long X = __shfl_sync(0xffffffffu, mX, q);
        const bool ok = __shfl_sync(0xffffffffu, mok, q);
        const double tn = k + 32 < nn ? y[k + 32] : 0.0;
        if (q + 1 < m) u = upper(k + 1);
        const double tk = __shfl_sync(0xffffffffu, t, owner);
        double yk;
        if (!(quotient_round(tk, ukk, X, yk) && ok)) yk = div_rn_recip(tk, ukk, rcp[k]);
        if (lane == owner) {
            y[k] = yk;
            t = tn;
        }
        if (rr <= k + w && rr < nn) t = t - uk * yk;
    }
}

// Band LU and forward substitution for kl, ku <= 5 (the beams' systems, and the
// epsilon system of markers about a lattice unit apart): warp 0 factors with
// the whole active window in registers, warp 1 runs the forward substitution
// eight rows behind. The window of column j is rows j..j+5 and columns j..j+5:
// v0 = M(j, j); lane (i, k), i and k in 1..5, holds a = M(j+i, j), A = M(j+i, j+k)
// and the pivot row's uA = M(j, j+k). A column is one chain: the reciprocal of
// the diagonal (integer steps) with the pivot test beside it, multiplier,
// product and difference, and the broadcast of the next diagonal; the rest of
// the window moves up by shuffles, and its last row and column, which no step
// has touched, come from shared memory, in the shadow of the next reciprocal.
// One warp issues an instruction every few cycles, so what counts beside the
// chain is the number of instructions: every address is a lane's constant plus
// a row stride, every bound a lane's last column.
//
// An interchange (another candidate is larger) exchanges two rows of the window
// and takes a second reciprocal. The pivot row then reaches columns j+6..j+10:
// these columns join the window (uB, Bx) until six columns after the last
// interchange, when no remaining row has a changed entry that far right.
// Entries beyond the band or the matrix are zeros, whose products change
// nothing. The pipeline over four warps and shared memory below took 1290
// cycles a column, this takes 630: the reciprocal about 200, multiplier,
// product and difference 195, the pivot test, the stores and the shuffles the
// rest. k_fem_dynamic of the 1200 x 400 filament: 1.19 -> 0.76 million cycles.
__device__ __forceinline__ double band_entry(const double* Bd, int nn, int kl, int ku, int W, int r, int c) {
    return r < nn && c < nn && c - r <= ku && r - c <= kl ? Bd[r * W + c - r + kl] : 0.0;
}
__device__ __forceinline__ unsigned long long magnitude_key(double v, unsigned long long nan) {
    const unsigned long long key = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    return key > 0x7ff0000000000000ull ? nan : key;
}
constexpr int kForwardRows = 8;  // rows warp 1 takes at a time

__device__ void band_lu_window(double* Bd, int nn, int kl, int ku, int W, int* piv, double* y, double* rcp) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        const bool on = lane < 25;
        const int i = on ? 1 + lane / 5 : 5, k = on ? 1 + lane % 5 : 5;
        double v0 = band_entry(Bd, nn, kl, ku, W, 0, 0), a = band_entry(Bd, nn, kl, ku, W, i, 0);
        double uA = band_entry(Bd, nn, kl, ku, W, 0, k), A = band_entry(Bd, nn, kl, ku, W, i, k);
        double uB = 0.0, Bx = 0.0;
        // what enters window j+1: M(j+1+i, j+1+k) on the lanes i = 5 or k = 5,
        // M(j+1, j+6) on k = 5, M(j+6, j+1) on i = 5, as offsets from row j of
        // the band; loaded while j < the lane's limit (0: never)
        const int oA = (1 + i) * W + k - i + kl, oU = W + 5 + kl, oL = 6 * W + kl - 5;
        const int far = i > k ? i : k;
        const int nA = (i == 5 || k == 5) && k - i <= ku && i - k <= kl ? nn - 1 - far : 0;
        const int nU = k == 5 && ku >= 5 ? nn - 6 : 0, nL = i == 5 && kl >= 5 ? nn - 6 : 0;
        // stores of column j: the multiplier (lanes k = 1), U's row (lanes i = 1)
        const int sL = i * W + kl - i, sU = kl + k;
        const int mL = on && k == 1 && i <= kl ? nn - i : 0, mU = on && i == 1 && k <= kl + ku ? nn - k : 0;
        double* row = Bd;  // row j
        int last = -100;   // column of the last interchange
        for (int j = 0; j < nn; j++, row += W) {
            unsigned long long X;
            double r;
            bool ok = recip64(v0, X);
            ok &= recip_round(v0, X, r);
            const double eA = j < nA ? row[oA] : 0.0, eU = j < nU ? row[oU] : 0.0, eL = j < nL ? row[oL] : 0.0;
            int src = 0;
            // magnitudes by their high words first (a NaN on the diagonal stays)
            const unsigned ha = (unsigned)__double2hiint(a) & 0x7fffffffu;
            if (__any_sync(0xffffffffu, ha >= ((unsigned)__double2hiint(v0) & 0x7fffffffu))) {
                // the first maximal magnitude: a NaN on the diagonal wins,
                // others never do
                const bool cand = on && k == 1;
                const unsigned long long ka = magnitude_key(a, 0ull);
                if (__any_sync(0xffffffffu, cand && ka > magnitude_key(v0, ~0ull))) {
                    const unsigned kh = cand ? (unsigned)(ka >> 32) : 0u;
                    const unsigned mh = __reduce_max_sync(0xffffffffu, kh);
                    const bool c1 = cand && kh == mh;
                    const unsigned ml = __reduce_max_sync(0xffffffffu, c1 ? (unsigned)ka : 0u);
                    // lane (src, 1)
                    const int from = __ffs(__ballot_sync(0xffffffffu, c1 && (unsigned)ka == ml)) - 1;
                    src = 1 + from / 5;
                    if (j - last >= 6) {  // the far columns join
                        uB = 0.0;
                        Bx = band_entry(Bd, nn, kl, ku, W, j + i, j + k + 5);
                    }
                    last = j;
                    const double pv = __shfl_sync(0xffffffffu, a, from);
                    const double rA = __shfl_sync(0xffffffffu, A, from + k - 1);
                    const double rB = __shfl_sync(0xffffffffu, Bx, from + k - 1);
                    if (i == src) {
                        A = uA;
                        Bx = uB;
                        a = v0;
                    }
                    uA = rA;
                    uB = rB;
                    v0 = pv;
                    ok = recip64(v0, X);
                    ok &= recip_round(v0, X, r);
                }
            }
            double scale = r;
            if (!ok) {
                r = __drcp_rn(v0);
                // a zero pivot does not scale the column
                scale = ((unsigned long long)__double_as_longlong(v0) << 1) != 0ull ? r : 1.0;
            }
            const double L = a * scale;
            // x + L * (-u), written as the identical x - L * u
            A = A - L * uA;
            if (j < mL) row[sL] = L;
            if (j < mU) row[sU] = uA;
            if (lane == 0) {
                row[kl] = v0;
                piv[j] = j + src;
                rcp[j] = r;  // RN(1 / U(j,j)) for the forward solve
            }
            const bool far_in = j - last < 6;
            if (far_in) {
                Bx = Bx - L * uB;
                if (on && i == 1 && k + 5 <= kl + ku && j + k + 5 < nn) row[sU + 5] = uB;
            }
            if (j % kForwardRows == kForwardRows - 1 || j == nn - 1) named_bar(1, 64);
            // the window of column j+1
            v0 = __shfl_sync(0xffffffffu, A, 0);
            const double fa = __shfl_sync(0xffffffffu, A, 5 * i), fA = __shfl_down_sync(0xffffffffu, A, 6);
            const double pA = __shfl_sync(0xffffffffu, A, k);
            a = i < 5 ? fa : eL;
            uA = k < 5 ? pA : eU;
            A = i < 5 && k < 5 ? fA : eA;
            if (far_in) {
                const double fB0 = __shfl_sync(0xffffffffu, Bx, 5 * i), fB = __shfl_down_sync(0xffffffffu, Bx, 6);
                const double pB0 = __shfl_sync(0xffffffffu, Bx, 0), pB = __shfl_sync(0xffffffffu, Bx, k);
                if (k == 5) {
                    uA = pB0;
                    if (i < 5) A = fB0;
                }
                uB = k < 5 ? pB : 0.0;
                Bx = i == 5 ? band_entry(Bd, nn, kl, ku, W, j + 6, j + 6 + k) : (k < 5 ? fB : 0.0);
            }
        }
    } else if (warp == 1) {
        double t = lane < nn ? y[lane] : 0.0;
        for (int k0 = 0; k0 < nn; k0 += kForwardRows) {
            named_bar(1, 64);
            const int m = nn - k0 < kForwardRows ? nn - k0 : kForwardRows;
            forward_rows(Bd, nn, kl, W, kl + ku, k0, m, lane, rcp, y, t);
        }
        __syncwarp();
    }
}

// Band LU of M and the forward half of the transposed solve (U^T y = b, y in
// place) by warps 0-3 of the CTA; kl <= 31 and kl + ku <= 31. Bands of up to
// five go to band_lu_window; wider ones are pipelined.
// The operations are those of band_factor_smem followed by the row-ordered
// forward substitution; only who does them, and when, differs. The critical
// path is warp 0's chain per column: reciprocal of the pivot, multipliers,
// update of the next column's candidates. Everything else runs beside it:
//   warp 0: the reciprocals of column j's candidates (each lane its own; the
//           pivot's is kept, the same correctly rounded 1/pivot as a division
//           after the choice) from integer steps, the choice of the pivot
//           between them, barrier 2, the row swap, the scaling and the step-j
//           update of column j+1, barrier 1. Column j+1's candidates are then
//           already in its registers (the rows it just updated, plus one row
//           no earlier step touched);
//   warps 1, 3: after barrier 1, the step-j update of columns j+2..kmax,
//           split between them, then barrier 2 (which warp 0 waits on before
//           the swap of step j+1, the first thing to touch those rows again);
//   warp 2: after barrier 1, forward row j (row j of U is final once the swap
//           of step j is done): y_j = t_j / U(j,j) and every row r in
//           (j, j+kl+ku] subtracts U(j,r) y_j. Each row still subtracts its
//           terms in ascending order, so every sum is formed as before.
// Barrier counts: warp 0 calls barrier 1 nn times and barrier 2 nn-1 times
// (before each swap after the first); warps 1 and 3 call barrier 1 nn times
// and barrier 2 after every step but the last; warp 2 calls barrier 1 nn
// times. The k-th calls pair up, so every barrier completes. Needs at least
// 128 threads; with fewer, warp 0 does everything.
// (With the reciprocal in FP64, and the pivot chosen by warp 3 and handed over
// through barrier 2, a column took 1271 cycles.)
__device__ void band_lu_forward(double* Bd, int nn, int kl, int ku, int W, int* piv, double* y, double* rcp) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (blockDim.x < 128) {
        if (warp == 0) {
            band_factor_smem(Bd, nn, kl, ku, W, piv);
            if (lane == 0)
                for (int i = 0; i < nn; i++) {
                    double t = y[i];
                    for (int k = (i - kl - ku > 0 ? i - kl - ku : 0); k < i; k++) t -= bd(Bd, W, kl, k, i) * y[k];
                    y[i] = t / bd(Bd, W, kl, i, i);
                }
            __syncwarp();
        }
        return;
    }
    if (kl <= 5 && ku <= 5) {
        band_lu_window(Bd, nn, kl, ku, W, piv, y, rcp);
        return;
    }
    if (warp == 0) {
        // lane l holds the pivot candidate M(j+l, j)
        double v = lane <= (kl < nn - 1 ? kl : nn - 1) ? bd(Bd, W, kl, lane, 0) : 0.0;
        for (int j = 0; j < nn; j++) {
            const int imax = j + kl < nn - 1 ? j + kl : nn - 1;
            const int kmax = j + kl + ku < nn - 1 ? j + kl + ku : nn - 1;
            const bool row = j + lane <= imax, early = j + 1 <= kmax;
            // the candidates' reciprocals, and the choice among them meanwhile
            unsigned long long X;
            double rc;
            bool ok = recip64(v, X);
            ok &= recip_round(v, X, rc);
            const int src = pick_pivot(v, row, lane);
            // the row that enters column j+1's candidates: no step has touched it
            const double entering =
                lane == kl && j + 1 + kl < nn ? bd(Bd, W, kl, j + 1 + kl, j + 1) : 0.0;
            if (j > 0) named_bar(2, 96);
            double x = row && early ? bd(Bd, W, kl, j + lane, j + 1) : 0.0;
            const int jp = j + src;
            const double pv = __shfl_sync(0xffffffffu, v, src), v0 = __shfl_sync(0xffffffffu, v, 0);
            const double u1 = __shfl_sync(0xffffffffu, x, src), x0 = __shfl_sync(0xffffffffu, x, 0);
            double r = __shfl_sync(0xffffffffu, rc, src);
            if (!__shfl_sync(0xffffffffu, ok, src)) r = __drcp_rn(pv);
            // pivot != 0 (NaN counts as non-zero), tested on the bits
            const bool nz = ((unsigned long long)__double_as_longlong(pv) << 1) != 0ull;
            const bool swapped = nz && src != 0;
            // values after the swap (which a zero pivot does not make)
            const double a = swapped && lane == src ? v0 : v;
            if (swapped && lane == src) x = x0;
            const double L = nz ? a * r : a;
            // x + L * (-u1), written as the identical x - L * u1
            const bool mrow = lane >= 1 && row;  // multiplier row i = j + lane
            const double nx = mrow && early ? x - L * (swapped ? u1 : x0) : 0.0;
            if (swapped) {
                const int c = j + lane;
                if (c <= kmax) {
                    const double rj = bd(Bd, W, kl, j, c), rp = bd(Bd, W, kl, jp, c);
                    bd(Bd, W, kl, j, c) = rp;
                    if (c >= j + 2) bd(Bd, W, kl, jp, c) = rj;
                }
                __syncwarp();
            }
            if (lane == 0) {
                piv[j] = jp;
                rcp[j] = r;  // RN(1 / U(j,j)) for the forward solve
            }
            if (mrow) {
                bd(Bd, W, kl, j + lane, j) = L;
                if (early) bd(Bd, W, kl, j + lane, j + 1) = nx;
            }
            named_bar(1, 128);
            // column j+1's candidates: lane l+1 holds the updated row j+1+l
            v = __shfl_down_sync(0xffffffffu, nx, 1);
            if (lane == kl) v = entering;
        }
    } else if (warp == 1 || warp == 3) {
        // entry q of the kl x (kl+ku-1) block of a full step, kept in registers
        const int q0 = lane + (warp == 3 ? 32 : 0);
        const int fr = kl > 0 ? kl : 1, fc = kl + ku - 1;
        const int qi0 = q0 % fr, qk0 = q0 / fr, qi1 = (q0 + 64) % fr, qk1 = (q0 + 64) / fr;
        for (int j = 0; j < nn; j++) {
            named_bar(1, 128);
            const int imax = j + kl < nn - 1 ? j + kl : nn - 1;
            const int kmax = j + kl + ku < nn - 1 ? j + kl + ku : nn - 1;
            const int rows = imax - j, cols = kmax - j - 1;
            if (rows == kl && cols == fc && rows * cols <= 128) {
                // bd(i,k) + bd(i,j) * (-bd(j,k)), written as the identical
                // bd(i,k) - bd(i,j) * bd(j,k)
                if (q0 < rows * cols) {
                    const int i = j + 1 + qi0, k = j + 2 + qk0;
                    bd(Bd, W, kl, i, k) = bd(Bd, W, kl, i, k) - bd(Bd, W, kl, i, j) * bd(Bd, W, kl, j, k);
                }
                if (q0 + 64 < rows * cols) {
                    const int i = j + 1 + qi1, k = j + 2 + qk1;
                    bd(Bd, W, kl, i, k) = bd(Bd, W, kl, i, k) - bd(Bd, W, kl, i, j) * bd(Bd, W, kl, j, k);
                }
            } else {
                for (int q = q0; q < rows * cols; q += 64) {
                    const int i = j + 1 + q % rows, k = j + 2 + q / rows;
                    bd(Bd, W, kl, i, k) = bd(Bd, W, kl, i, k) - bd(Bd, W, kl, i, j) * bd(Bd, W, kl, j, k);
                }
            }
            if (j < nn - 1) named_bar(2, 96);
        }
    } else if (warp == 2) {
        const int w = kl + ku;
        double t = lane < nn ? y[lane] : 0.0;
        for (int k = 0; k < nn; k++) {
            named_bar(1, 128);
            forward_rows(Bd, nn, kl, W, w, k, 1, lane, rcp, y, t);
        }
        __syncwarp();
    }
}

// The forward half of the transposed solve alone (U^T y = b, y in place) on
// factors band_lu_forward produced earlier: warp 2's part of that routine
// without the pipeline, the same operations in the same order. One warp.
__device__ void band_forward_only(const double* Bd_, int nn, int kl, int ku, int W, double* y, const double* rcp) {
    double* Bd = const_cast<double*>(Bd_);
    const int lane = threadIdx.x & 31, w = kl + ku;
    double t = lane < nn ? y[lane] : 0.0;
    for (int k0 = 0; k0 < nn; k0 += 32) forward_rows(Bd, nn, kl, W, w, k0, nn - k0 < 32 ? nn - k0 : 32, lane, rcp, y, t);
    __syncwarp();
}

// The products pr of lanes 0..m-1 subtracted from acc in lane order.
__device__ __forceinline__ double subtract_lanes(double acc, double pr, int m) {
    if (m == 5) {
#pragma unroll
        for (int q = 0; q < 5; q++) acc = acc - __shfl_sync(0xffffffffu, pr, q);
    } else {
        for (int q = 0; q < m; q++) acc = acc - __shfl_sync(0xffffffffu, pr, q);
    }
    return acc;
}

// Backward half of the transposed solve (L^T) after band_lu_forward, warps 0
// and 1 of the CTA: row i subtracts the products of the multipliers stored in
// band rows i+1..i+kl with y at their final rows, in ascending final row (the
// order of the dense solve); then the row interchanges. The chain of a row is
// one product and up to kl differences: its operands are loaded a row ahead,
// and the newest y stays in a register. With interchanges warp 1 follows the
// final rows (the swaps, from the last back) and leaves every row's terms in
// order in Fp, a chunk of rows ahead of warp 0. 590 -> 478 cycles a row (kl = 5)
// without interchanges; the chain alone is 415.
__device__ void band_solve_back(const double* Bd_, int nn, int kl, int W, const int* piv, int* Fp, double* y) {
    double* Bd = const_cast<double*>(Bd_);
    __shared__ double s_prod[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool any = false;
    for (int i0 = 0; i0 < nn; i0 += 32) {
        const int i = i0 + lane;
        any |= __any_sync(0xffffffffu, i < nn && piv[i] != i);
    }
    if (!any) {
        // every multiplier stays in its row: lane l's product is the l-th term
        if (warp != 0) return;
        double yw = 0.0, bv = 0.0, yi = y[nn - 1];  // lane l: y[i+1+l] and its multiplier
        int i = nn - 1;
        // the last kl rows have fewer terms
        for (; i >= 0 && i + kl > nn - 1; i--) {
            const double pr = bv * yw, yc = yi;
            if (i > 0) {
                yi = y[i - 1];
                bv = lane < kl && i + lane < nn ? bd(Bd, W, kl, i + lane, i - 1) : 0.0;
            }
            const double acc = subtract_lanes(yc, pr, nn - 1 - i);
            const double up = __shfl_up_sync(0xffffffffu, yw, 1);
            yw = lane == 0 ? acc : up;
            if (lane == 0) y[i] = acc;
        }
        // M(i+1+lane, i) is a lane's constant away from row i
        const double* at = Bd + (i + lane) * W + kl - 1 - lane;  // of row i-1
        const bool mine = lane < kl;
        if (kl == 5) {
            for (; i >= 0; i--, at -= W) {
                const double pr = bv * yw;
                double acc = yi;
                if (i > 0) {
                    yi = y[i - 1];
                    if (mine) bv = *at;
                }
                const double up = __shfl_up_sync(0xffffffffu, yw, 1);
#pragma unroll
                for (int q = 0; q < 5; q++) acc = acc - __shfl_sync(0xffffffffu, pr, q);
                yw = lane == 0 ? acc : up;
                if (lane == 0) y[i] = acc;
            }
        } else {
            for (; i >= 0; i--, at -= W) {
                const double pr = bv * yw;
                double acc = yi;
                if (i > 0) {
                    yi = y[i - 1];
                    if (mine) bv = *at;
                }
                const double up = __shfl_up_sync(0xffffffffu, yw, 1);
                for (int q = 0; q < kl; q++) acc = acc - __shfl_sync(0xffffffffu, pr, q);
                yw = lane == 0 ? acc : up;
                if (lane == 0) y[i] = acc;
            }
        }
        __syncwarp();
        return;
    }
    const int chunk = kl > 0 ? (nn / (2 * kl) < 32 ? nn / (2 * kl) : 32) : 0;
    if (kl > 8 || chunk < 1) {
        if (warp != 0) return;
        for (int r = lane; r < nn; r += 32) Fp[r] = r;
        __syncwarp();
        for (int i = nn - 1; i >= 0; i--) {
            const int rmax = i + kl < nn - 1 ? i + kl : nn - 1;
            const int m = rmax - i;
            const bool act = lane < m;
            const int fk = act ? Fp[i + 1 + lane] : 0x7fffffff;
            int rank = 0;
            for (int q = 0; q < m; q++) rank += __shfl_sync(0xffffffffu, fk, q) < fk ? 1 : 0;
            if (act) s_prod[rank] = bd(Bd, W, kl, i + 1 + lane, i) * y[fk];
            __syncwarp();
            if (lane == 0) {
                double ti = y[i];
                for (int q = 0; q < m; q++) ti = ti - s_prod[q];
                y[i] = ti;
                const int p = piv[i];
                const int tmp = Fp[i];
                Fp[i] = Fp[p];
                Fp[p] = tmp;
            }
            __syncwarp();
        }
    } else {
        // terms of row i: Fp[half][(rows into the chunk) * kl + rank], the band
        // row's offset from i+1 in the high half and the final row in the low
        const int nch = (nn + chunk - 1) / chunk;
        int F = 0;                            // warp 1: final row of band row i+1+lane
        double ti = 0.0, bv = 0.0, yv = 0.0;  // warp 0
        int fk = -1;
        for (int c = 0; c <= nch; c++) {
            if (warp == 1 && c < nch) {
                int* out = Fp + (c & 1) * chunk * kl;
                for (int q = 0; q < chunk; q++) {
                    const int i = nn - 1 - (c * chunk + q);
                    if (i < 0) break;
                    const int p = piv[i], m = (i + kl < nn - 1 ? i + kl : nn - 1) - i;
                    int rank = 0;
                    for (int e = 0; e < m; e++) rank += __shfl_sync(0xffffffffu, F, e) < F ? 1 : 0;
                    if (lane < m) out[q * kl + rank] = (lane << 16) | F;
                    // the swap of step i: rows i (still its own) and p
                    const int l = p - i - 1, fp = __shfl_sync(0xffffffffu, F, l >= 0 ? l : 0);
                    if (lane == l) F = i;
                    const int up = __shfl_up_sync(0xffffffffu, F, 1);
                    F = lane == 0 ? (l >= 0 ? fp : i) : up;
                }
            } else if (warp == 0 && c > 0) {
                const int* in = Fp + ((c - 1) & 1) * chunk * kl;
                const int i1 = nn - 1 - (c - 1) * chunk;  // the chunk's first row
                auto load = [&](int i) {
                    fk = -1;
                    bv = yv = 0.0;
                    if (lane < (i + kl < nn - 1 ? i + kl : nn - 1) - i) {
                        const int e = in[(i1 - i) * kl + lane];
                        fk = e & 0xffff;
                        bv = bd(Bd, W, kl, i + 1 + (e >> 16), i);
                        yv = y[fk];  // (the newest row is in ti)
                    }
                };
                load(i1);
                for (int i = i1; i >= 0 && i > i1 - chunk; i--) {
                    const int m = (i + kl < nn - 1 ? i + kl : nn - 1) - i;
                    const double pr = bv * (fk == i + 1 ? ti : yv), yc = y[i];
                    if (i > 0 && i - 1 > i1 - chunk) load(i - 1);
                    ti = subtract_lanes(yc, pr, m);
                    __syncwarp();
                    if (lane == 0) y[i] = ti;
                    __syncwarp();
                }
            }
            named_bar(3, 64);
        }
        if (warp != 0) return;
    }
    for (int i0 = ((nn - 1) / 32) * 32; i0 >= 0; i0 -= 32) {
        unsigned swaps = __ballot_sync(0xffffffffu, i0 + lane < nn && piv[i0 + lane] != i0 + lane);
        if (lane == 0)
            while (swaps) {
                const int i = i0 + 31 - __clz(swaps), p = piv[i];
                swaps &= ~(1u << (i - i0));
                const double tt = y[i];
                y[i] = y[p];
                y[p] = tt;
            }
        __syncwarp();
    }
}

// Transposed solve M^T x = y in place (one lane, any band); Fp is nn ints of
// scratch.
__device__ void band_solve_smem(double* Bd, int nn, int kl, int ku, int W, const int* piv, int* Fp, double* y) {
    const int w = kl + ku;
    for (int i = 0; i < nn; i++) {
        double t = y[i];
        for (int k = (i - w > 0 ? i - w : 0); k < i; k++) t -= bd(Bd, W, kl, k, i) * y[k];
        y[i] = t / bd(Bd, W, kl, i, i);
    }
    for (int r = 0; r < nn; r++) Fp[r] = r;
    int fk[32];
    double fv[32];
    for (int i = nn - 1; i >= 0; i--) {
        const int rmax = i + kl < nn - 1 ? i + kl : nn - 1;
        int m = 0;
        for (int r = i + 1; r <= rmax; r++) {
            const int k = Fp[r];
            const double v = bd(Bd, W, kl, r, i);
            int q = m++;
            while (q > 0 && fk[q - 1] > k) {
                fk[q] = fk[q - 1];
                fv[q] = fv[q - 1];
                q--;
            }
            fk[q] = k;
            fv[q] = v;
        }
        double t = y[i];
        for (int q = 0; q < m; q++) t -= fv[q] * y[fk[q]];
        y[i] = t;
        const int p = piv[i];
        const int tmp = Fp[i];
        Fp[i] = Fp[p];
        Fp[p] = tmp;
    }
    for (int i = nn - 1; i >= 0; i--)
        if (piv[i] != i) {
            const double t = y[i];
            y[i] = y[piv[i]];
            y[piv[i]] = t;
        }
}

// Dense LU and transposed solve (band_lu.h semantics) of a matrix whose
// nonzeros are few but not in a narrow band, by one CTA: the epsilon system of
// a closed line of markers (the first and the last are neighbours) or of
// several bodies that touch. M(i, k) is at D[k * n + i]; rmask holds, for each
// row, a bit per column that may be nonzero, cmask the same by column (nw
// words each). Elimination step j visits only the rows with a bit in column j
// and the columns with a bit in the pivot row, and spreads the bits as the
// update fills entries in. Every other entry is an exact zero, whose products
// leave the values they are added to unchanged, so each value is formed by the
// same operations in the same order as in the dense loops. A step:
//   phase 1  warp 0 takes the first maximal magnitude of column j's rows (the
//            diagonal's reciprocal is formed meanwhile) and the column's
//            multipliers; the last warp the forward substitution of step j-1
//            (y[k] -= U(j-1,k) y[j-1])
//   swap     only where the pivot is not on the diagonal: whole rows, their
//            masks, and row j's column list again
//   phase 2  one thread per updated entry, a 16 x 16 tile at a time; the masks;
//            the last warp divides y[j] by the pivot, the two before it list
//            the rows and columns of step j+1 (its masks with this step's bits,
//            which others may be adding at the same time: the same bits)
// b in y, the solution in y; rows and cols: 2n ints each, one after the other;
// mult: n doubles. Needs 256 threads. Returns false (uniformly) when a pivot is
// zero or not finite or the solution is not finite: then zeros do matter, and
// the caller runs the dense loops.
// One warp over all of the band (kl = ku = n) took 6.49 ms for the 132 markers
// of a circle and its tail; this takes 0.21 ms, bound by the latencies of a
// step (reciprocal, multiplier, product, difference, two barriers).
struct SparseLu {
    double* D;
    unsigned *rmask, *cmask;
    double *y, *rcp, *mult;
    int *piv, *rows, *cols;
};

// Set bits above `above` of lane-wise mask words (lane w holds word w; nw <= 32)
// as an ascending list (one warp); returns the count on every lane.
__device__ __forceinline__ int word_list(unsigned w, int above, int* out) {
    const int lane = threadIdx.x & 31;
    const int first = above + 1 - 32 * lane;  // first wanted bit of this word
    if (first >= 32) w = 0u;
    else if (first > 0) w &= ~0u << first;
    unsigned words = __ballot_sync(0xffffffffu, w != 0u);
    int base = 0;
    while (words) {
        const int q = __ffs(words) - 1;
        words &= words - 1;
        const unsigned word = __shfl_sync(0xffffffffu, w, q);
        if ((word >> lane) & 1u) out[base + __popc(word & ((1u << lane) - 1u))] = 32 * q + lane;
        base += __popc(word);
    }
    __syncwarp();
    return base;
}
__device__ __forceinline__ int mask_list(const unsigned* mask, int nw, int above, int* out) {
    const int lane = threadIdx.x & 31;
    return word_list(lane < nw ? mask[lane] : 0u, above, out);
}

__device__ __forceinline__ bool finite_bits(double x) {
    return ((unsigned)(__double_as_longlong(x) >> 32) & 0x7ff00000u) != 0x7ff00000u;
}

__device__ __forceinline__ bool sparse_lu_solve(const SparseLu& S, int n, int nw) {
    __shared__ int s_nr[2], s_nc[2], s_jp, s_bad, s_any, s_cnt[2][8];
    __shared__ unsigned long long s_X;  // recip64 of the pivot (0: it does not apply)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, last = (blockDim.x >> 5) - 1;
    double* D = S.D;
    if (tid == 0) { s_bad = 0; s_any = 0; }
    if (warp == last - 1) {
        const int c = mask_list(S.cmask, nw, 0, S.rows);
        if (lane == 0) s_nr[0] = c;
    } else if (warp == last) {
        const int c = mask_list(S.rmask, nw, 0, S.cols);
        if (lane == 0) s_nc[0] = c;
    }
    __syncthreads();
    for (int j = 0; j <= n; j++) {
        const int pb = j & 1;
        int *rows = S.rows + pb * n, *cols = S.cols + pb * n;  // below / right of the diagonal
        double* Dj = D + (size_t)j * n;
        // phase 1
        if (warp == 0 && j < n) {
            const int nr = s_nr[pb];
            // the first 32 candidates: the diagonal, then the listed rows
            const int row = lane == 0 || lane > nr ? j : rows[lane - 1];
            const double v = lane <= nr ? Dj[row] : 0.0;
            const double v0 = __shfl_sync(0xffffffffu, v, 0);
            int jp = j;
            double pv = v0, r;
            unsigned long long X;
            bool ok = recip64(v0, X);
            ok &= recip_round(v0, X, r);
            // magnitudes by their high words first
            const unsigned h0 = (unsigned)__double2hiint(v0) & 0x7fffffffu;
            if (nr > 31 || __any_sync(0xffffffffu, lane > 0 && ((unsigned)__double2hiint(v) & 0x7fffffffu) >= h0)) {
                // the first maximal magnitude: a NaN on the diagonal wins,
                // others never do
                unsigned long long best = magnitude_key(v0, ~0ull);
                for (int q0 = 0; q0 < nr; q0 += 32) {
                    const int i = q0 + lane < nr ? rows[q0 + lane] : -1;
                    const double x = i >= 0 ? Dj[i] : 0.0;
                    const unsigned long long key = i >= 0 ? magnitude_key(x, 0ull) : 0ull;
                    const unsigned kh = (unsigned)(key >> 32), klo = (unsigned)key;
                    const unsigned mh = __reduce_max_sync(0xffffffffu, kh);
                    const bool c1 = i >= 0 && kh == mh;
                    const unsigned ml = __reduce_max_sync(0xffffffffu, c1 ? klo : 0u);
                    const unsigned long long top = ((unsigned long long)mh << 32) | ml;
                    if (top > best) {
                        best = top;
                        const int src = __ffs(__ballot_sync(0xffffffffu, c1 && klo == ml)) - 1;
                        jp = __shfl_sync(0xffffffffu, i, src);
                        pv = __shfl_sync(0xffffffffu, x, src);
                    }
                }
                if (jp != j) {
                    ok = recip64(pv, X);
                    ok &= recip_round(pv, X, r);
                }
            }
            if (!ok) {
                r = __drcp_rn(pv);
                X = 0ull;
                if (lane == 0 && (pv == 0.0 || !finite_bits(pv))) s_bad = 1;
            }
            // the multipliers, as they stand after the interchange
            if (lane > 0 && lane <= nr) {
                const double m = (row == jp ? v0 : v) * r;
                S.mult[lane - 1] = m;
                Dj[row] = m;
            }
            for (int q = 31 + lane; q < nr; q += 32) {
                const int i = rows[q];
                const double m = (i == jp ? v0 : Dj[i]) * r;
                S.mult[q] = m;
                Dj[i] = m;
            }
            if (lane == 0) {
                Dj[j] = pv;
                s_jp = jp;
                S.piv[j] = jp;
                s_X = X;
                S.rcp[j] = r;
                if (jp != j) s_any = 1;
            }
        } else if (warp == last && j > 0) {
            const int k = j - 1, nc = s_nc[pb ^ 1];
            const int* pc = S.cols + (pb ^ 1) * n;
            const double yk = S.y[k];
            for (int q = lane; q < nc; q += 32) S.y[pc[q]] = S.y[pc[q]] - D[(size_t)pc[q] * n + k] * yk;
        }
        __syncthreads();
        if (j == n || s_bad) break;
        const int jp = s_jp;
        if (jp != j) {
            // (column j has its new values already)
            for (int k = tid; k < n; k += blockDim.x) {
                if (k != j) {
                    const double a = D[(size_t)k * n + j], b = D[(size_t)k * n + jp];
                    D[(size_t)k * n + j] = b;
                    D[(size_t)k * n + jp] = a;
                }
                unsigned* m = S.cmask + (size_t)k * nw;
                const unsigned bj = (m[j >> 5] >> (j & 31)) & 1u, bp = (m[jp >> 5] >> (jp & 31)) & 1u;
                // (in column j both stay: the pivot and what was the diagonal)
                if (bj != bp && k != j) {
                    m[j >> 5] ^= 1u << (j & 31);
                    m[jp >> 5] ^= 1u << (jp & 31);
                }
            }
            for (int w = tid; w < nw; w += blockDim.x) {
                const unsigned a = S.rmask[(size_t)j * nw + w];
                S.rmask[(size_t)j * nw + w] = S.rmask[(size_t)jp * nw + w];
                S.rmask[(size_t)jp * nw + w] = a;
            }
            __syncthreads();
            if (warp == 1) {
                const int nc = mask_list(S.rmask + (size_t)j * nw, nw, j, cols);
                if (lane == 0) s_nc[pb] = nc;
            }
            __syncthreads();
        }
        // phase 2
        const int nr = s_nr[pb], nc = s_nc[pb];
        if (warp == last) {
            // (y[j] has its last term: phase 1 took step j-1's)
            const double t = S.y[j], u = Dj[j];
            const unsigned long long X = s_X;
            double yk;
            if (!quotient_round(t, u, X, yk) || X == 0ull) yk = div_rn_recip(t, u, S.rcp[j]);
            if (lane == 0) S.y[j] = yk;
        } else if (warp >= last - 2 && j + 1 < n) {
            // column j+1 gains column j's rows if the pivot row reaches it, row
            // j+1 the pivot row's columns if column j reaches it
            const bool col = warp == last - 1;
            const unsigned* own = (col ? S.cmask : S.rmask) + (size_t)(j + 1) * nw;
            const unsigned* add = (col ? S.cmask : S.rmask) + (size_t)j * nw;
            const unsigned reach = (col ? S.rmask : S.cmask)[(size_t)j * nw + ((j + 1) >> 5)] >> ((j + 1) & 31) & 1u;
            unsigned w = 0u;
            if (lane < nw) w = own[lane] | (reach ? add[lane] : 0u);
            const int c = word_list(w, j + 1, (col ? S.rows : S.cols) + (pb ^ 1) * n);
            if (lane == 0) (col ? s_nr : s_nc)[pb ^ 1] = c;
        }
        const int a0 = tid & 15, b0 = tid >> 4;
        for (int b = b0; b < nc; b += 16) {
            double* Dk = D + (size_t)cols[b] * n;
            const double u = Dk[j];
            for (int a = a0; a < nr; a += 16) {
                const int i = rows[a];
                Dk[i] = Dk[i] - S.mult[a] * u;
            }
        }
        // the filled-in entries' bits; only columns above j and rows below the
        // diagonal
        // (by warps 1-4, which have no other task)
        for (int w = b0 - 2; w >= 0 && b0 < 10 && w < nw; w += 8) {
            const int first = j + 1 - 32 * w;
            const unsigned keep = first >= 32 ? 0u : (first > 0 ? ~0u << first : ~0u);
            const unsigned rj = S.rmask[(size_t)j * nw + w] & keep, cj = S.cmask[(size_t)j * nw + w] & keep;
            for (int a = a0; a < nr; a += 16) S.rmask[(size_t)rows[a] * nw + w] |= rj;
            for (int b = a0; b < nc; b += 16) S.cmask[(size_t)cols[b] * nw + w] |= cj;
        }
        __syncthreads();
    }
    if (s_bad) return false;  // (set before a barrier: the same on all threads)
    // L^T x = y from the last row up: the products of a column's multipliers on
    // lanes, subtracted in ascending row order by warp 0; the other warps list
    // the rows of the next `last` columns meanwhile (in rows and cols' place)
    const int cap = 4 * n / (2 * last) < 32 ? 4 * n / (2 * last) : 32, groups = (n + last - 1) / last;
    for (int g = 0; g <= groups; g++) {
        if (warp > 0 && g < groups) {
            const int i = n - 1 - (g * last + warp - 1);
            if (i >= 0) {
                const unsigned w = lane < nw ? S.cmask[(size_t)i * nw + lane] : 0u;
                const int first = i + 1 - 32 * lane;
                const int c = __reduce_add_sync(0xffffffffu, __popc(first >= 32 ? 0u : (first > 0 ? w & (~0u << first) : w)));
                if (c <= cap) word_list(w, i, S.rows + ((g & 1) * last + warp - 1) * cap);
                if (lane == 0) s_cnt[g & 1][warp] = c;
            }
        } else if (warp == 0 && g > 0) {
            const int i1 = n - 1 - (g - 1) * last;  // the group's first row
            const int* lists = S.rows + ((g - 1) & 1) * last * cap;
            const int rows_left = i1 + 1 < last ? i1 + 1 : last;
            // a row's count and list two rows ahead, its operands one ahead
            // (its newest term is in t)
            int c = 0, c1 = 0, k = -1, k1 = -1;
            double d = 0.0, yk = 0.0, yi = 0.0, t = 0.0;
            auto list_of = [&](int p) {
                c1 = p < rows_left ? s_cnt[(g - 1) & 1][p + 1] : 0;
                k1 = lane < c1 && c1 <= cap ? lists[p * cap + lane] : -1;
            };
            auto load = [&](int p) {
                c = c1;
                k = k1;
                d = yk = 0.0;
                yi = S.y[i1 - p];
                if (k >= 0) {
                    d = D[(size_t)(i1 - p) * n + k];
                    yk = S.y[k];
                }
                list_of(p + 1);
            };
            list_of(0);
            load(0);
            for (int p = 0; p < rows_left; p++) {
                const int i = i1 - p, m = c;
                const double pr = d * (p > 0 && k == i + 1 ? t : yk);
                t = yi;
                if (p + 1 < rows_left) load(p + 1);
                if (m <= cap) {
                    for (int q = 0; q < m; q++) t = t - __shfl_sync(0xffffffffu, pr, q);
                } else {  // more rows than a list holds: every row below
                    for (int q0 = i + 1; q0 < n; q0 += 32) {
                        const int kk = q0 + lane, mm = n - q0 < 32 ? n - q0 : 32;
                        const bool bit = kk < n && ((S.cmask[(size_t)i * nw + (kk >> 5)] >> (kk & 31)) & 1u);
                        const unsigned some = __ballot_sync(0xffffffffu, bit);
                        const double pq = bit ? D[(size_t)i * n + kk] * S.y[kk] : 0.0;
                        for (int q = 0; q < mm; q++)
                            if ((some >> q) & 1u) t = t - __shfl_sync(0xffffffffu, pq, q);
                    }
                }
                __syncwarp();
                if (lane == 0) S.y[i] = t;
                __syncwarp();
            }
        }
        __syncthreads();
    }
    if (tid == 0 && s_any)
        for (int i = n - 1; i >= 0; i--)
            if (S.piv[i] != i) {
                const double t = S.y[i];
                S.y[i] = S.y[S.piv[i]];
                S.y[S.piv[i]] = t;
            }
    __syncthreads();
    bool ok = true;
    for (int i = tid; i < n; i += blockDim.x) ok = ok && finite_bits(S.y[i]);
    return __syncthreads_and(ok) != 0;
}

// Epsilon system of a contiguous marker range [m0, m0+dim) (ObjectsClass::
// computeEpsilon, src/Objects.cpp:264-311). Markers interact only when both
// coordinates are within 3 lattice units (the support is +-1.5); those pairs
// set the band of the system.
__device__ __forceinline__ bool eps_near(const MarkerDev& M, int ki, int kj, double Dx) {
    return fabs(M.pos[ki * 2] - M.pos[kj * 2]) / Dx < 3.0 && fabs(M.pos[ki * 2 + 1] - M.pos[kj * 2 + 1]) / Dx < 3.0;
}

__device__ __forceinline__ double eps_entry(const MarkerDev& M, int ki, int kj, double Dx) {
    const double xj = M.pos[kj * 2], yj = M.pos[kj * 2 + 1];
    double acc = 0.0;
    const int ns = M.nsupp[ki];
    for (int s = 0; s < ns; s++) {
        const double dvi = M.sd[ki * 9 + s];
        const double dX = fabs(xj / Dx - M.si[ki * 9 + s]);
        const double dY = fabs(yj / Dx - M.sj[ki * 9 + s]);
        acc += dvi * (dirac_d(dX) * dirac_d(dY));
    }
    return acc * (1.0 * 1.0 * M.ds[kj]);
}

// Fast path of the epsilon system, all in shared memory (`sm`, `sm_doubles`):
//   xy[2*dim]    marker positions
//   ph[10*dim]   kernel tables: for marker k and axis a, s = pos/Dx and
//                ph[k*10 + 5a + o] = dirac(|s - c|) at lattice line
//                c = c0[2k+a] + o, c0 = floor(s) - 2, o = 0..4. The kernel is
//                zero beyond 1.5, so every line outside the table gives the
//                exact 0.0 the direct evaluation gives.
//   c0[2*dim]    (ints)
//   cand[cap]    pairs that pass a conservative prefilter (|dx| and |dy|
//                below about 3*Dx), then their matrix entries
//   band / y / pivots / final rows of the banded LU
// Entries use the same operations and operands as eps_entry, so they are
// identical. Returns false (uniformly) when the marker set does not fit; the
// caller then runs the direct path.
// (sd, si, sj: the marker's support; the nine loads of each go out together,
// the sum is in order)
__device__ __forceinline__ double eps_entry_tab(const double* sd, const int* si, const int* sj, int ns, int jl,
                                                const double* ph, const int* c0, double dsj) {
    int ei[9], ej[9];
    double dv[9];
#pragma unroll
    for (int s = 0; s < 9; s++) {
        ei[s] = si[s];
        ej[s] = sj[s];
        dv[s] = sd[s];
    }
    const int cx = c0[jl * 2], cy = c0[jl * 2 + 1];
    double acc = 0.0;
#pragma unroll
    for (int s = 0; s < 9; s++) {
        const int ox = ei[s] - cx, oy = ej[s] - cy;
        const double px = (ox >= 0 && ox < 5) ? ph[jl * 10 + ox] : 0.0;
        const double py = (oy >= 0 && oy < 5) ? ph[jl * 10 + 5 + oy] : 0.0;
        const double next = acc + dv[s] * (px * py);
        acc = s < ns ? next : acc;
    }
    return acc * (1.0 * 1.0 * dsj);
}

__device__ __forceinline__ bool epsilon_fast(const FsiDev& F, const MarkerDev& M, int m0, int dim, double* A, double* bx, int* piv,
                             int* lmax, double* sm, int sm_doubles) {
    __shared__ int s_kl, s_ku, s_nc;
    const long long fixed = 13LL * dim + 64;
    if (!sm || dim > 4096 || fixed >= sm_doubles) return false;
    const int cap = (int)((sm_doubles - fixed) / 3);
    double* xy = sm;
    double* ph = xy + 2 * dim;
    int* c0 = reinterpret_cast<int*>(ph + 10 * dim);
    double* cval = ph + 11 * dim + 1;
    int* ckey = reinterpret_cast<int*>(cval + cap);
    double* band = cval + cap + (cap + 1) / 2 + 1;
    const long long band_doubles = sm_doubles - (band - sm);
    const double Dx = F.Dx;
    if (threadIdx.x == 0) { s_kl = 0; s_ku = 0; s_nc = 0; }
    for (int q = threadIdx.x; q < 2 * dim; q += blockDim.x) xy[q] = M.pos[m0 * 2 + q];
    __syncthreads();
    // s = pos / Dx of every coordinate, and s in FP32 for the prefilter, at the
    // entries' place until those are formed
    const bool room = cap >= 3 * dim;
    double* sc = cval;
    float* sf = reinterpret_cast<float*>(cval + 2 * dim);
    if (room) {
        for (int q = threadIdx.x; q < 2 * dim; q += blockDim.x) {
            sc[q] = xy[q] / Dx;
            sf[q] = (float)sc[q];
        }
        __syncthreads();
    }
    for (int q = threadIdx.x; q < 10 * dim; q += blockDim.x) {
        const int k = q / 10, a = (q % 10) / 5, o = q % 5;
        const double sk = room ? sc[2 * k + a] : xy[2 * k + a] / Dx;
        const int base = (int)floor(sk) - 2;
        if (o == 0) c0[2 * k + a] = base;
        ph[q] = dirac_d(fabs(sk - (base + o)));
    }
    // prefilter + compaction, a row of pairs per warp (in FP32 with a margin well
    // above its rounding, so that no pair of the exact test is lost)
    const double lim = 3.0 * Dx * (1.0 + 0x1p-40), sure = 3.0 * Dx * (1.0 - 0x1p-40);
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x >> 5; i < dim; i += blockDim.x >> 5) {
        const float xi = room ? sf[2 * i] : 0.0f, yi = room ? sf[2 * i + 1] : 0.0f;
#pragma unroll 2
        for (int j0 = 0; j0 < dim; j0 += 32) {
            const int j = j0 + lane;
            bool c = false;
            if (j < dim) {
                if (room) {
                    const float xj = sf[2 * j], yj = sf[2 * j + 1];
                    c = fabsf(xi - xj) < fmaf(0x1p-21f, fabsf(xi) + fabsf(xj), 3.001f) &&
                        fabsf(yi - yj) < fmaf(0x1p-21f, fabsf(yi) + fabsf(yj), 3.001f);
                } else {
                    c = fabs(xy[2 * i] - xy[2 * j]) < lim && fabs(xy[2 * i + 1] - xy[2 * j + 1]) < lim;
                }
            }
            const unsigned bal = __ballot_sync(0xffffffffu, c);
            if (bal == 0u) continue;
            int base = 0;
            if (lane == 0) base = atomicAdd(&s_nc, __popc(bal));
            base = __shfl_sync(0xffffffffu, base, 0);
            const int slot = base + __popc(bal & ((1u << lane) - 1u));
            if (c && slot < cap) ckey[slot] = i * dim + j;
        }
    }
    __syncthreads();
    const int nc = s_nc;
    if (nc > cap) return false;
    // the markers' supports, where the system will stand (a pair's entry reads
    // all of one: from global memory 32 lanes touch 32 lines at a time)
    const bool staged = 18LL * dim <= band_doubles;
    const double* gd = M.sd + (size_t)m0 * 9;
    const int *gi = M.si + (size_t)m0 * 9, *gj = M.sj + (size_t)m0 * 9;
    if (staged) {
        double* td = band;
        int *ti = reinterpret_cast<int*>(band + 9 * dim), *tj = ti + 9 * dim;
        for (int q = threadIdx.x; q < 9 * dim; q += blockDim.x) {
            td[q] = gd[q];
            ti[q] = gi[q];
            tj[q] = gj[q];
        }
        gd = td;
        gi = ti;
        gj = tj;
        __syncthreads();
    }
    for (int c = threadIdx.x; c < nc; c += blockDim.x) {
        const int pp = ckey[c];
        const int i = pp / dim, j = pp % dim;
        // (well below 3 Dx the quotient is below 3; only at the edge is it formed)
        const double ax = fabs(xy[2 * i] - xy[2 * j]), ay = fabs(xy[2 * i + 1] - xy[2 * j + 1]);
        if ((ax < sure || ax / Dx < 3.0) && (ay < sure || ay / Dx < 3.0)) {
            cval[c] = eps_entry_tab(gd + i * 9, gi + i * 9, gj + i * 9, M.nsupp[m0 + i], j, ph, c0, M.ds[m0 + j]);
            if (j > i) atomicMax(&s_kl, j - i);
            else if (i > j) atomicMax(&s_ku, i - j);
        } else {
            ckey[c] = -1;
        }
    }
    __syncthreads();
    const int kl = s_kl, ku = s_ku, W = 2 * kl + ku + 1;
    if (kl < 32 && kl + ku < 32 && (long long)dim * W + 3 * dim + 1 <= band_doubles) {
        double* Bd = band;
        double* y = Bd + (size_t)dim * W;
        int* sp = reinterpret_cast<int*>(y + dim);
        int* fp = sp + dim;
        for (int q = threadIdx.x; q < dim * W; q += blockDim.x) Bd[q] = 0.0;
        for (int i = threadIdx.x; i < dim; i += blockDim.x) y[i] = 1.0;
        __syncthreads();
        for (int c = threadIdx.x; c < nc; c += blockDim.x) {
            const int pp = ckey[c];
            if (pp >= 0) bd(Bd, W, kl, pp % dim, pp / dim) = cval[c];
        }
        __syncthreads();
        if (threadIdx.x < 128) band_lu_forward(Bd, dim, kl, ku, W, sp, y, reinterpret_cast<double*>(fp + dim));
        __syncthreads();
        if (threadIdx.x < 64) band_solve_back(Bd, dim, kl, W, sp, fp, y);
        __syncthreads();
        for (int i = threadIdx.x; i < dim; i += blockDim.x) M.eps[m0 + i] = y[i];
        __syncthreads();
        return true;
    }
    // wide band with few nonzeros: sparse elimination on a dense matrix behind
    // the entries in shared memory, or in the global scratch if it is too large
    const int nw = (dim + 31) / 32;
    if (nw <= 32 && nc + (nc + 1) / 2 + 1 <= cap) {
        // the entries' keys to the end of their values
        int* ck = reinterpret_cast<int*>(cval + nc);
        for (int c = threadIdx.x; c < nc; c += blockDim.x) ck[c] = ckey[c];
        __syncthreads();
        ckey = ck;
        double* at = cval + nc + (nc + 1) / 2;
        SparseLu S;
        S.y = at;
        S.rcp = S.y + dim;
        S.mult = S.rcp + dim;
        S.piv = reinterpret_cast<int*>(S.mult + dim);
        S.rows = S.piv + dim;
        S.cols = S.rows + 2 * dim;
        S.rmask = reinterpret_cast<unsigned*>(S.cols + 2 * dim);
        S.cmask = S.rmask + (size_t)dim * nw;
        const long long ints = 5LL * dim + 2LL * dim * nw;
        const long long used = (at - sm) + 3LL * dim + (ints + 1) / 2;
        if (used <= sm_doubles) {
            S.D = used + (long long)dim * dim <= sm_doubles ? sm + used : A;
            for (int q = threadIdx.x; q < dim * dim; q += blockDim.x) S.D[q] = 0.0;
            for (int q = threadIdx.x; q < 2 * dim * nw; q += blockDim.x) S.rmask[q] = 0u;
            for (int i = threadIdx.x; i < dim; i += blockDim.x) S.y[i] = 1.0;
            __syncthreads();
            for (int c = threadIdx.x; c < nc; c += blockDim.x) {
                const int pp = ckey[c];
                if (pp < 0) continue;
                const int k = pp / dim, i = pp % dim;  // A[k][i] is M(i, k)
                S.D[pp] = cval[c];
                atomicOr(&S.rmask[(size_t)i * nw + (k >> 5)], 1u << (k & 31));
                atomicOr(&S.cmask[(size_t)k * nw + (i >> 5)], 1u << (i & 31));
            }
            __syncthreads();
            if (sparse_lu_solve(S, dim, nw)) {
                for (int i = threadIdx.x; i < dim; i += blockDim.x) M.eps[m0 + i] = S.y[i];
                __syncthreads();
                return true;
            }
        }
    }
    // dense system in global scratch, same entries
    for (long long q = threadIdx.x; q < (long long)dim * dim; q += blockDim.x) A[q] = 0.0;
    for (int i = threadIdx.x; i < dim; i += blockDim.x) bx[i] = 1.0;
    __syncthreads();
    for (int c = threadIdx.x; c < nc; c += blockDim.x) {
        const int pp = ckey[c];
        if (pp >= 0) A[pp] = cval[c];
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        warp_lu_factor(A, dim, 0, kl, ku, piv, lmax);
        warp_lu_solve(A, dim, 0, kl, ku, piv, lmax, bx, bx);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < dim; i += blockDim.x) M.eps[m0 + i] = bx[i];
    __syncthreads();
    return true;
}

// Direct path (marker sets beyond the shared-memory plan): entries evaluated
// pair by pair, band LU in `smem` when it fits, else the dense LU in A.
__device__ __forceinline__ void epsilon_range(const FsiDev& F, const MarkerDev& M, int m0, int dim, double* A, double* bx, int* piv,
                              int* lmax, double* smem = nullptr, int smem_doubles = 0) {
    if (epsilon_fast(F, M, m0, dim, A, bx, piv, lmax, smem, smem_doubles)) return;
    __shared__ int s_kl, s_ku;
    if (threadIdx.x == 0) { s_kl = 0; s_ku = 0; }
    __syncthreads();
    const double Dx = F.Dx;
    // bandwidths of the LU's view M = A^T: A[i][j] sits at M(j, i)
    for (long long p = threadIdx.x; p < (long long)dim * dim; p += blockDim.x) {
        const int i = (int)(p / dim), j = (int)(p % dim);
        if (i != j && eps_near(M, m0 + i, m0 + j, Dx)) {
            if (j > i) atomicMax(&s_kl, j - i);
            else atomicMax(&s_ku, i - j);
        }
    }
    __syncthreads();
    const int kl = s_kl, ku = s_ku, W = 2 * kl + ku + 1;
    const long long need = (long long)dim * W + 3 * dim + 1;  // band, y, two int arrays, reciprocals
    if (smem && kl < 32 && need <= smem_doubles) {
        double* Bd = smem;
        double* y = Bd + (size_t)dim * W;
        int* sp = reinterpret_cast<int*>(y + dim);
        int* fp = sp + dim;
        for (long long q = threadIdx.x; q < (long long)dim * W; q += blockDim.x) Bd[q] = 0.0;
        for (int i = threadIdx.x; i < dim; i += blockDim.x) y[i] = 1.0;
        __syncthreads();
        const int bw = kl > ku ? kl : ku;
        for (long long p = threadIdx.x; p < (long long)dim * dim; p += blockDim.x) {
            const int i = (int)(p / dim), j = (int)(p % dim);
            if (j - i > bw || i - j > bw) continue;
            if (eps_near(M, m0 + i, m0 + j, Dx)) bd(Bd, W, kl, j, i) = eps_entry(M, m0 + i, m0 + j, Dx);
        }
        __syncthreads();
        if (kl + ku < 32) {
            if (threadIdx.x < 128) band_lu_forward(Bd, dim, kl, ku, W, sp, y, reinterpret_cast<double*>(fp + dim));
            __syncthreads();
            if (threadIdx.x < 64) band_solve_back(Bd, dim, kl, W, sp, fp, y);
        } else if (threadIdx.x < 32) {
            band_factor_smem(Bd, dim, kl, ku, W, sp);
            if (threadIdx.x == 0) band_solve_smem(Bd, dim, kl, ku, W, sp, fp, y);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < dim; i += blockDim.x) M.eps[m0 + i] = y[i];
        __syncthreads();
        return;
    }
    for (long long p = threadIdx.x; p < (long long)dim * dim; p += blockDim.x) A[p] = 0.0;
    __syncthreads();
    for (long long p = threadIdx.x; p < (long long)dim * dim; p += blockDim.x) {
        const int i = (int)(p / dim), j = (int)(p % dim);
        if (eps_near(M, m0 + i, m0 + j, Dx)) A[p] = eps_entry(M, m0 + i, m0 + j, Dx);
    }
    for (int i = threadIdx.x; i < dim; i += blockDim.x) bx[i] = 1.0;
    __syncthreads();
    if (threadIdx.x < 32) {
        warp_lu_factor(A, dim, 0, kl, ku, piv, lmax);
        warp_lu_solve(A, dim, 0, kl, ku, piv, lmax, bx, bx);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < dim; i += blockDim.x) M.eps[m0 + i] = bx[i];
    __syncthreads();
}

constexpr int kEpsSmemDoubles = 25000;  // 200000 bytes of dynamic shared memory (opt-in)

__global__ void __launch_bounds__(256, 1) k_fsi_epsilon_body(FsiDev F, MarkerDev M) {
    extern __shared__ double eps_smem[];
    FemBodyDev& B = F.bodies[blockIdx.x];
    epsilon_range(F, M, B.mbase, B.nMark, B.epsA, B.epsB, B.piv, B.lmax, eps_smem, kEpsSmemDoubles);
}

__global__ void __launch_bounds__(256, 1) k_fsi_epsilon_uni(FsiDev F, MarkerDev M) {
    extern __shared__ double eps_smem[];
    epsilon_range(F, M, 0, M.n, F.uniA, F.uniB, F.uniPiv, F.uniLmax, eps_smem, kEpsSmemDoubles);
}

// FEMBodyClass::dynamicFEM (src/FEMBody.cpp:26-68) for one body per CTA.
__global__ void __launch_bounds__(256, 1) k_fem_dynamic(FsiDev F, MarkerDev M) {
    FemBodyDev& B = F.bodies[blockIdx.x];
    __shared__ double s_res;
    __shared__ int s_it;
    const int n = B.n;
    const int nn = n - B.bc;
    constexpr int KW = 2 * 5 + 5 + 1;  // band width of the LU (kl = ku = 5)
    extern __shared__ double fem_smem[];
    double* sBd = fem_smem;            // [nn][KW] LU band
    double* sMb = sBd + nn * KW;       // [n][11] mass band
    double* sKe = sMb + n * 11;        // [n][11] stiffness band
    double* sV = sKe + n * 11;         // [n] Newmark vector
    double* sY = sV + n;               // [nn] right-hand side / solution
    int* sPiv = reinterpret_cast<int*>(sY + nn);
    int* sFp = sPiv + nn;
    double* sRcp = reinterpret_cast<double*>(sFp + nn);  // [nn] pivot reciprocals
    // Every subiteration restarts from U_n (U = U_n, Udot = Udot_n, ...), so
    // the first Newton iteration of every subiteration of a step builds the
    // same element matrices, internal force F, K_eff = K + a0 M and M v with
    // v = a0 (U_n - U) + a2 Udot + a3 Udotdot; only the load R differs.
    // Subiteration 0 keeps that iteration's LU factors, F and M v; the later
    // subiterations form F_eff = (R - F) + M v from them and solve with the
    // kept factors (the same factorisation of the same matrix).
    const bool reuse = F.s->subIt > 0;
    double* cBd = B.lu_cache;
    double* cRcp = cBd + (size_t)nn * KW;
    double* cF = cRcp + nn;
    double* cMv = cF + n;
    int* cPiv = reinterpret_cast<int*>(cMv + n);
    {
        double* U = vec(B, V_U);
        double* Ud = vec(B, V_Udot);
        double* Udd = vec(B, V_Udotdot);
        const double* Un = vec(B, V_Un);
        const double* Udn = vec(B, V_Udotn);
        const double* Uddn = vec(B, V_Udotdotn);
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            U[i] = Un[i];
            Ud[i] = Udn[i];
            Udd[i] = Uddn[i];
        }
    }
    __syncthreads();
    // updateFEMValues at U = U_n: subiteration 0 evaluates it and keeps the
    // node positions and element values (length, angle, cos, sin); the later
    // subiterations restart from the same U_n and copy them back
    {
        double* cNode = reinterpret_cast<double*>(cMv + n) + (nn + 1) / 2;
        double* cEl = cNode + 3 * (size_t)B.nNodes;
        if (!reuse) {
            update_fem_values(B);
            for (int q = threadIdx.x; q < B.nNodes; q += blockDim.x) {
                const double* nd = B.node + q * 6;
                cNode[q * 3 + 0] = nd[2];
                cNode[q * 3 + 1] = nd[3];
                cNode[q * 3 + 2] = nd[5];
            }
            for (int e = threadIdx.x; e < B.nEl; e += blockDim.x) {
                const double* el = B.el + (size_t)e * EL_STRIDE;
                cEl[e * 4 + 0] = el[EL_ANG];
                cEl[e * 4 + 1] = el[EL_L];
                cEl[e * 4 + 2] = el[EL_COS];
                cEl[e * 4 + 3] = el[EL_SIN];
            }
        } else {
            for (int q = threadIdx.x; q < B.nNodes; q += blockDim.x) {
                double* nd = B.node + q * 6;
                nd[2] = cNode[q * 3 + 0];
                nd[3] = cNode[q * 3 + 1];
                nd[5] = cNode[q * 3 + 2];
            }
            for (int e = threadIdx.x; e < B.nEl; e += blockDim.x) {
                double* el = B.el + (size_t)e * EL_STRIDE;
                el[EL_ANG] = cEl[e * 4 + 0];
                el[EL_L] = cEl[e * 4 + 1];
                el[EL_COS] = cEl[e * 4 + 2];
                el[EL_SIN] = cEl[e * 4 + 3];
            }
            __syncthreads();
        }
    }
    // constructRVector (src/FEMBody.cpp:226-234; FEMElementClass::loadVector,
    // src/FEMElement.cpp:27-69): contributions per force-map entry, then an
    // ordered assembly.
    {
        const double forceScale = F.Dm / DSQ(F.Dt);
        for (int q = threadIdx.x; q < B.nfmap; q += blockDim.x) {
            const int e = B.fmapEl[q];
            const double* el = B.el + (size_t)e * EL_STRIDE;
            const double c = el[EL_COS], s = el[EL_SIN], L = el[EL_L];
            const double wgt0 = el[EL_RHO] * el[EL_A] * F.gravityX, wgt1 = el[EL_RHO] * el[EL_A] * F.gravityY;
            const int k = B.mbase + B.fmapNode[q];
            const double a = B.fmapZ[q * 2], b = B.fmapZ[q * 2 + 1];
            const double sc = -M.eps[k] * 1.0 * forceScale;
            const double g0 = sc * M.force[k * 2] + wgt0, g1 = sc * M.force[k * 2 + 1] + wgt1;
            const double F0 = (0.0 + c * g0) + s * g1;
            const double F1 = (0.0 + (-s) * g0) + c * g1;
            double R[6], RG[6];
            R[0] = F0 * 0.5 * L * (0.5 * b - 0.5 * a + 0.25 * DSQ(a) - 0.25 * DSQ(b));
            R[1] = F1 * 0.5 * L * (0.5 * b - 0.5 * a - DSQ(a) * DSQ(a) / 16.0 + DSQ(b) * DSQ(b) / 16.0 + 3.0 * DSQ(a) / 8.0 - 3.0 * DSQ(b) / 8.0);
            R[2] = F1 * 0.5 * L * (L * (-DSQ(a) * DSQ(a) + DSQ(b) * DSQ(b)) / 32.0 - L * (-DTH(a) + DTH(b)) / 24.0 - L * (-DSQ(a) + DSQ(b)) / 16.0 + L * (b - a) / 8.0);
            R[3] = F0 * 0.5 * L * (-0.25 * DSQ(a) + 0.25 * DSQ(b) + 0.5 * b - 0.5 * a);
            R[4] = F1 * 0.5 * L * (0.5 * b - 0.5 * a + DSQ(a) * DSQ(a) / 16.0 - DSQ(b) * DSQ(b) / 16.0 - 3.0 * DSQ(a) / 8.0 + 3.0 * DSQ(b) / 8.0);
            R[5] = F1 * 0.5 * L * (L * (-DSQ(a) * DSQ(a) + DSQ(b) * DSQ(b)) / 32.0 + L * (-DTH(a) + DTH(b)) / 24.0 - L * (-DSQ(a) + DSQ(b)) / 16.0 - L * (b - a) / 8.0);
            tt_vec(R, c, s, RG);
            for (int r = 0; r < 6; r++) B.rgscr[q * 6 + r] = RG[r];
        }
        __syncthreads();
        double* Rv = vec(B, V_R);
        for (int r = threadIdx.x; r < n; r += blockDim.x) {
            double acc = 0.0;
            const int e1 = r / 3 - 1, e2 = r / 3;
            for (int e = (e1 < 0 ? 0 : e1); e <= e2 && e < B.nEl; e++)
                for (int q = B.fmapStart[e]; q < B.fmapStart[e + 1]; q++) acc += B.rgscr[q * 6 + (r - 3 * e)];
            Rv[r] = acc;
        }
        __syncthreads();
    }
    const double Dt = F.Dt, al = F.alpha;
    const double a0 = 1.0 / (al * DSQ(Dt)), a2 = 1.0 / (al * Dt), a3 = 1.0 / (2.0 * al) - 1.0;
    if (threadIdx.x == 0) s_it = 0;
    __syncthreads();
    do {
        const bool first = s_it == 0;
        if (first && reuse) {
            // the kept factors and vectors of this step's first iteration
            double* Fv = vec(B, V_F);
            const double* Rv = vec(B, V_R);
            for (int q = threadIdx.x; q < nn * KW; q += blockDim.x) sBd[q] = cBd[q];
            for (int i = threadIdx.x; i < nn; i += blockDim.x) {
                sPiv[i] = cPiv[i];
                sRcp[i] = cRcp[i];
            }
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                const double fe = Rv[i] - cF[i] + cMv[i];
                Fv[i] = fe;
                if (i >= B.bc) sY[i - B.bc] = fe;
            }
            __syncthreads();
            if (threadIdx.x < 32) band_forward_only(sBd, nn, 5, 5, KW, sY, sRcp);
            __syncthreads();
            if (threadIdx.x < 64) band_solve_back(sBd, nn, 5, KW, sPiv, sFp, sY);
            __syncthreads();
        } else {
            // buildGlobalMatrices (src/FEMBody.cpp:90-109): the stiffness and
            // the internal force of an element on one half of the threads, its
            // mass matrix on the other
            for (int q = threadIdx.x & 127; q < B.nEl; q += 128) {
                const int e = q;
                const double* el = B.el + (size_t)e * EL_STRIDE;
                const double c = el[EL_COS], s = el[EL_SIN];
                double* sc = B.elscr + (size_t)e * ES_STRIDE;
                if (threadIdx.x >= 128) {
                    tt_a_t<pattern(false)>(el + EL_M, c, s, sc + ES_M);
                    continue;
                }
                const double L = el[EL_L], L0 = el[EL_L0], E = el[EL_E], A = el[EL_A], I = el[EL_I], ang = el[EL_ANG];
                const double u = (DSQ(L) - DSQ(L0)) / (L + L0);
                const double th1 = shift_angle_d(B.node[e * 6 + 5] - ang);
                const double th2 = shift_angle_d(B.node[(e + 1) * 6 + 5] - ang);
                const double F0 = (E * A / L0) * u;
                const double bend = 2 * E * I / L0;
                const double M1 = bend * (2.0 * th1 + th2);
                const double M2 = bend * (th1 + 2.0 * th2);
                const double shear = (1.0 / L0) * (M1 + M2);
                double Fl[6];
                Fl[0] = -F0;
                Fl[1] = shear;
                Fl[2] = M1;
                Fl[3] = F0;
                Fl[4] = -shear;
                Fl[5] = M2;
                tt_vec(Fl, c, s, sc + ES_F);
                double G[36], G2[36], KNL[36];
                tt_a_t<pattern(false)>(el + EL_KL, c, s, G);
                const double v = Fl[4] / L0, f = -Fl[0] / L0;
#pragma unroll
                for (int q6 = 0; q6 < 36; q6++) KNL[q6] = 0.0;
                KNL[0 * 6 + 1] = -v;
                KNL[0 * 6 + 4] = v;
                KNL[1 * 6 + 0] = -v;
                KNL[1 * 6 + 1] = f;
                KNL[1 * 6 + 3] = v;
                KNL[1 * 6 + 4] = -f;
                KNL[3 * 6 + 1] = v;
                KNL[3 * 6 + 4] = -v;
                KNL[4 * 6 + 0] = v;
                KNL[4 * 6 + 1] = -f;
                KNL[4 * 6 + 3] = -v;
                KNL[4 * 6 + 4] = f;
                tt_a_t<pattern(true)>(KNL, c, s, G2);
                // (the geometric part has no rotations: rows and columns 2, 5)
#pragma unroll
                for (int q6 = 0; q6 < 36; q6++)
                    sc[ES_K + q6] = (q6 / 6) % 3 == 2 || q6 % 3 == 2 ? from_zero(G[q6]) : G[q6] + G2[q6];
            }
            __syncthreads();
            // Ordered assembly of M, K (band |r-c| <= 5) and F, then setNewmark
            // (src/FEMBody.cpp:112-126): K_eff = K + a0*M goes straight into the
            // shared-memory band of the LU's view M(i,j) = K_eff[bc+j][bc+i].
            {
                double* Fv = vec(B, V_F);
                for (int q = threadIdx.x; q < nn * KW; q += blockDim.x) sBd[q] = 0.0;
                for (int p = threadIdx.x; p < n * 11; p += blockDim.x) {
                    const int r = p / 11, cc = r - 5 + p % 11;
                    if (cc < 0 || cc >= n) continue;
                    double am = 0.0, ak = 0.0;
                    const int lo = (r > cc ? r : cc), hi = (r < cc ? r : cc);
                    for (int e = (lo / 3 - 1 < 0 ? 0 : lo / 3 - 1); e <= hi / 3 && e < B.nEl; e++) {
                        const int li = r - 3 * e, lj = cc - 3 * e;
                        if (li < 0 || li > 5 || lj < 0 || lj > 5) continue;
                        const double* sc = B.elscr + (size_t)e * ES_STRIDE;
                        am += sc[ES_M + li * 6 + lj];
                        ak += sc[ES_K + li * 6 + lj];
                    }
                    sMb[p] = am;
                    sKe[p] = ak;
                }
                for (int r = threadIdx.x; r < n; r += blockDim.x) {
                    double af = 0.0;
                    for (int e = (r / 3 - 1 < 0 ? 0 : r / 3 - 1); e <= r / 3 && e < B.nEl; e++)
                        af += B.elscr[(size_t)e * ES_STRIDE + ES_F + (r - 3 * e)];
                    Fv[r] = af;
                }
                const double* U = vec(B, V_U);
                const double* Un = vec(B, V_Un);
                const double* Ud = vec(B, V_Udot);
                const double* Udd = vec(B, V_Udotdot);
                for (int i = threadIdx.x; i < n; i += blockDim.x) sV[i] = a0 * (Un[i] - U[i]) + a2 * Ud[i] + a3 * Udd[i];
                __syncthreads();
                const double* Rv = vec(B, V_R);
                for (int i = threadIdx.x; i < n; i += blockDim.x) {
                    double mv = 0.0;
                    for (int j = (i - 5 < 0 ? 0 : i - 5); j <= i + 5 && j < n; j++) mv += sMb[i * 11 + (j - i + 5)] * sV[j];
                    if (first) {
                        cF[i] = Fv[i];
                        cMv[i] = mv;
                    }
                    const double fe = Rv[i] - Fv[i] + mv;
                    Fv[i] = fe;
                    if (i >= B.bc) sY[i - B.bc] = fe;
                }
                for (int p = threadIdx.x; p < n * 11; p += blockDim.x) {
                    const int r = p / 11, cc = r - 5 + p % 11;
                    if (cc < B.bc || cc >= n || r < B.bc) continue;
                    const double keff = sKe[p] + a0 * sMb[p];
                    bd(sBd, KW, 5, cc - B.bc, r - B.bc) = keff;
                }
            }
            __syncthreads();
            // delU = solveLAPACK(K, F, bcDOFs) (src/Utils.cpp:288-311)
            if (threadIdx.x < 128) band_lu_forward(sBd, nn, 5, 5, KW, sPiv, sY, sRcp);
            __syncthreads();
            if (first) {
                for (int q = threadIdx.x; q < nn * KW; q += blockDim.x) cBd[q] = sBd[q];
                for (int i = threadIdx.x; i < nn; i += blockDim.x) {
                    cPiv[i] = sPiv[i];
                    cRcp[i] = sRcp[i];
                }
            }
            if (threadIdx.x < 64) band_solve_back(sBd, nn, 5, KW, sPiv, sFp, sY);
            __syncthreads();
        }
        {
            double* dU = vec(B, V_delU);
            for (int i = threadIdx.x; i < n; i += blockDim.x) dU[i] = i < B.bc ? 0.0 : sY[i - B.bc];
        }
        __syncthreads();
        {
            double* U = vec(B, V_U);
            const double* dU = vec(B, V_delU);
            for (int i = threadIdx.x; i < n; i += blockDim.x) U[i] = U[i] + dU[i];
        }
        __syncthreads();
        // squares in parallel, then the sum in index order (one thread)
        {
            const double* dU = vec(B, V_delU);
            for (int i = threadIdx.x; i < n; i += blockDim.x) sV[i] = dU[i] * dU[i];
        }
        // (update_fem_values' first barrier stands between the squares and the sum)
        update_fem_values(B, [&]() {
            if ((threadIdx.x & 31) == 0) {
                double dd = 0.0;
                for (int i = 0; i < n; i++) dd += sV[i];
                s_res = sqrt(dd) / (F.ref_L * sqrt((double)n));
                s_it++;
            }
        });
    } while (s_res > 1e-10 && s_it < 20);
    finish_newmark(B, F);
    update_ibm(B, M);
    if (threadIdx.x == 0) {
        B.itNR = s_it;
        B.resNR = s_res;
        swap_slots(B, V_Rkm1, V_Rk);
    }
    __syncthreads();
    // FEMBodyClass::subResidual (src/FEMBody.cpp:244-256): the terms in
    // parallel, each of the three sums in index order by one thread of its
    // own warp.
    {
        double* Rk = vec(B, V_Rk);
        const double* Rkm1 = vec(B, V_Rkm1);
        const double* U = vec(B, V_U);
        const double* Uk = vec(B, V_Ukm1);
        double* tr = sMb;
        double* tn = sMb + n;
        double* td = sMb + 2 * n;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const double r = U[i] - Uk[i];
            const double d = r - Rkm1[i];
            Rk[i] = r;
            tr[i] = r * r;
            tn[i] = Rkm1[i] * d;
            td[i] = d * d;
        }
        __syncthreads();
        if ((threadIdx.x & 31) == 0 && threadIdx.x < 96) {
            const double* t = sMb + (threadIdx.x >> 5) * n;
            double acc = 0.0;
            for (int i = 0; i < n; i++) acc += t[i];
            if (threadIdx.x == 0) B.subRes = acc;
            else if (threadIdx.x == 32) B.subNum = acc;
            else B.subDen = acc;
        }
    }
}

// Standalone epsilon solve over n markers with caller-provided scratch
// (A: n*n, b: n, piv, lmax: n).
__global__ void __launch_bounds__(256, 1) k_epsilon_markers(FsiDev F, MarkerDev M, int n, double* A, double* b, int* piv,
                                                         int* lmax) {
    extern __shared__ double eps_smem[];
    epsilon_range(F, M, 0, n, A, b, piv, lmax, eps_smem, kEpsSmemDoubles);
}

// Element transform after a restart load (FEMElementClass::setElementTransform,
// src/FEMElement.cpp:255-262, called from ObjectsClass::readRestart,
// src/Objects.cpp:1195-1200): cos and sin of the loaded angles, with the
// same functions update_fem_values uses during a step.
__global__ void k_fem_element_trig(double* el, int nEl) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nEl) return;
    const double ang = el[(size_t)e * EL_STRIDE + EL_ANG];
    double sa, ca;
    life_cr_sincos(ang, &sa, &ca);
    el[(size_t)e * EL_STRIDE + EL_COS] = ca;
    el[(size_t)e * EL_STRIDE + EL_SIN] = sa;
}

cudaError_t launch_fem_element_trig(double* el, int nEl, cudaStream_t s) {
    if (nEl <= 0) return cudaSuccess;
    k_fem_element_trig<<<(nEl + 127) / 128, 128, 0, s>>>(el, nEl);
    return cudaGetLastError();
}

// The epsilon kernels take 200000 bytes of dynamic shared memory (opt-in);
// the attribute is set once per device.
cudaError_t epsilon_configure() {
    static std::atomic<int> done[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64 && done[dev].load()) return cudaSuccess;
    const int bytes = kEpsSmemDoubles * (int)sizeof(double);
    e = cudaFuncSetAttribute(k_fsi_epsilon_body, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_fsi_epsilon_uni, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_epsilon_markers, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev].store(1);
    return e;
}

cudaError_t launch_epsilon_markers(const MarkerDev& M, int n, double Dx, double* A, double* b, int* piv, int* lmax,
                                   cudaStream_t s) {
    FsiDev F{};
    F.Dx = Dx;
    cudaError_t e = epsilon_configure();
    if (e != cudaSuccess) return e;
    k_epsilon_markers<<<1, 256, kEpsSmemDoubles * sizeof(double), s>>>(F, M, n, A, b, piv, lmax);
    return cudaGetLastError();
}

// ObjectsClass::femKernel sums + loop condition + next relaxation factor.
// Inside the captured loop graph the condition also drives the WHILE node.
__global__ void k_fsi_residual(FsiDev F, cudaGraphConditionalHandle cond, int use_cond) {
    if (threadIdx.x != 0) return;
    FsiScalars& S = *F.s;
    double res = 0.0, num = 0.0, den = 0.0;
    for (int b = 0; b < F.nFlex; b++) {
        res += F.bodies[b].subRes;
        num += F.bodies[b].subNum;
        den += F.bodies[b].subDen;
    }
    S.subRes = sqrt(res) / (F.ref_L * sqrt((double)F.simDOFs));
    S.subNum = num;
    S.subDen = den;
    S.subIt += 1;
    S.lastNR = F.nFlex > 0 ? F.bodies[0].itNR : 0;
    const int cont = (S.subIt < 20 && S.subRes > F.subTol) ? 1 : 0;
    if (cont) {
        if (S.subIt == 1) {
            const double a = fabs(S.relax);
            const int sg = (0.0 < S.relax) - (S.relax < 0.0);
            S.relax = (double)(sg * (a < F.relaxMax ? a : F.relaxMax));
        } else {
            S.relax = -S.relax * S.subNum / S.subDen;
        }
    } else if (S.subIt == 20) {
        if (atomicCAS(&F.status[0], 0, LIFE_ERR_SUBITER) == 0) F.status[1] = S.t;
    }
    *F.cont = cont;
    if (use_cond) cudaGraphSetConditional(cond, cont ? 1u : 0u);
}

__global__ void k_fsi_begin(FsiDev F, int t, const int* t_dev, int t_off) {
    F.s->t = t_dev ? *t_dev + t_off : t;
    F.s->subIt = 0;
    *F.cont = 1;
}

size_t fem_dynamic_smem(int n, int bc) {
    const int nn = n - bc;
    return sizeof(double) * ((size_t)nn * 17 + (size_t)n * 22 + n + nn) + sizeof(int) * 2 * (size_t)nn;
}

// The opt-in shared-memory size is an attribute of the kernel, shared by every
// case on the device, so it only ever grows: a case created later with
// smaller bodies must not lower it below what a live case launches with.
cudaError_t fem_dynamic_configure(size_t smem) {
    static std::atomic<size_t> set[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    size_t cur = set[dev].load();
    if (smem > cur) {
        e = cudaFuncSetAttribute(k_fem_dynamic, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        while (cur < smem && !set[dev].compare_exchange_weak(cur, smem)) {
        }
    }
    return epsilon_configure();
}

cudaError_t launch_fsi_begin(const FsiDev& F, int t, cudaStream_t s, const int* t_dev, int t_off) {
    k_fsi_begin<<<1, 1, 0, s>>>(F, t, t_dev, t_off);
    return cudaGetLastError();
}

cudaError_t launch_fsi_subiteration(const FsiDev& F, const MarkerDev& M, const void* P, const LatDev& L, int t,
                                    double velScale, cudaStream_t s, int* launches,
                                    const cudaGraphConditionalHandle* cond) {
    k_fsi_predict<<<F.nFlex, 256, 0, s>>>(F, M);
    k_fsi_support<<<(F.nFlexMarkers + 3) / 4, 128, 0, s>>>(F, M);
    if (F.uni) k_fsi_epsilon_uni<<<1, 256, kEpsSmemDoubles * sizeof(double), s>>>(F, M);
    else k_fsi_epsilon_body<<<F.nFlex, 256, kEpsSmemDoubles * sizeof(double), s>>>(F, M);
    cudaError_t e = launch_ibm_interp(P, L, t, M, nullptr, velScale, s, cond ? &F.s->t : nullptr);
    if (e != cudaSuccess) return e;
    k_fem_dynamic<<<F.nFlex, 256, F.fem_smem, s>>>(F, M);
    k_fsi_residual<<<1, 32, 0, s>>>(F, cond ? *cond : cudaGraphConditionalHandle{}, cond ? 1 : 0);
    if (launches) *launches += 6;
    return cudaGetLastError();
}

}  // namespace life

namespace {
__global__ void k_selftest_trig(int op, long long n, const double* x, const double* y, double* out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        double s, c;
        if (op == 2) {
            out[i] = life_cr_atan2(y[i], x[i]);
        } else {
            life_cr_sincos(x[i], &s, &c);
            out[i] = op == 0 ? s : c;
        }
    }
}
}  // namespace

extern "C" int life_selftest_trig(int32_t op, int64_t n, const double* x, const double* y, double* out) {
    if (op < 0 || op > 2 || n <= 0 || !x || !out || (op == 2 && !y))
        return life::set_error(LIFE_ERR_INVALID, "bad arguments");
    double *dx = nullptr, *dy = nullptr, *dout = nullptr;
    const size_t bytes = sizeof(double) * (size_t)n;
    cudaError_t e = cudaMalloc(&dx, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&dout, bytes);
    if (e == cudaSuccess && op == 2) e = cudaMalloc(&dy, bytes);
    if (e == cudaSuccess) e = cudaMemcpy(dx, x, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && op == 2) e = cudaMemcpy(dy, y, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_selftest_trig<<<152 * 4, 256>>>(op, (long long)n, dx, dy, dout);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, bytes, cudaMemcpyDeviceToHost);
    cudaFree(dx);
    cudaFree(dy);
    cudaFree(dout);
    if (e != cudaSuccess) return life::cuda_fail(e, "life_selftest_trig");
    return LIFE_OK;
}

extern "C" int life_selftest_division(int64_t n, uint64_t seed, int64_t* mismatches) {
    if (n <= 0 || !mismatches) return life::set_error(LIFE_ERR_INVALID, "bad arguments");
    unsigned long long* d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof(unsigned long long));
    if (e == cudaSuccess) {
        life::k_selftest_division<<<152 * 8, 256>>>((long long)n, (unsigned long long)seed, d);
        e = cudaGetLastError();
    }
    unsigned long long h = 0;
    if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost);
    if (d) cudaFree(d);
    if (e != cudaSuccess) return life::cuda_fail(e, "life_selftest_division");
    *mismatches = (int64_t)h;
    return LIFE_OK;
}
