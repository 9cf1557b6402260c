// Device marker state and the IBM kernel launchers.
#pragma once
#include <cuda_runtime.h>

#include "life_types.h"

namespace life {

// Markers in global order (the reference's iNode order after de-overlap).
struct MarkerDev {
    int n;
    double* pos;    // [n][2]
    double* vel;    // [n][2]
    double* force;  // [n][2]
    double* eps;    // [n]
    double* ds;     // [n]
    int* nsupp;     // [n]
    int* si;        // [n][9]
    int* sj;        // [n][9]
    double* sd;     // [n][9] delta weights
    int4* bbox;     // [n] support bounding box (imin, imax, jmin, jmax)
    int* body;      // [n] owning body
};

// Scratch of the spread.
struct IbmScratch {
    double* force_ibm;        // [2][S] dense IBM force of the current step
    long long* sites;         // support sites written this step
    long long* sites_prev;    // support sites of the previous step
    int* nsites;
    int* nsites_prev;
    unsigned* site_flag;      // [S / 32] a bit per site: listed this step (clear between steps)
    // The markers in ranges [range_start[b], range_start[b+1]), a body or a part
    // of a long one, and the bounding box of a range's support this step (imin,
    // imax, jmin, jmax): a site of the spread scans only the ranges whose box
    // reaches it.
    int nranges;
    const int* range_start;   // [nranges + 1]
    const int* range_of;      // [n] the range of each marker
    int4* range_box;          // [nranges]
    int4* range_box_next;     // [nranges] the other of two, reset by this step's spread
};
// Markers of a range at most. With one range a body every site of a body scanned
// all of its markers: a circle 800 sites across (2513 markers, FP32 storage) took
// 170.7 us a step, 131.8 in ranges of 128 (131.0 of 64, 133.5 of 256), one 200
// across 25.8 and 22.5 (21.9, 24.0).
constexpr int kRangeMarkers = 128;

// The two lists of support sites (and the boxes of each) change roles every
// step, as the two population buffers do: the step that reads P[0] fills one
// list, the step that reads P[1] the other, also in step graphs captured long
// before.
inline void swap_site_lists(IbmScratch& W) {
    long long* const s = W.sites;
    int* const n = W.nsites;
    int4* const b = W.range_box;
    W.sites = W.sites_prev;
    W.nsites = W.nsites_prev;
    W.range_box = W.range_box_next;
    W.sites_prev = s;
    W.nsites_prev = n;
    W.range_box_next = b;
}

// Close marker pairs of removeOverlapMarkers (appended unordered, see
// k_overlap_pairs).
cudaError_t launch_overlap_pairs(const double* pos, int nm, double Dx, int* count, int2* out, int cap,
                                 cudaStream_t s);
// Population buffers are untyped; their element type follows L.prec.
// With t_dev, the step is read from device memory when the kernel runs. With
// `mark`, the launch also does the work of launch_ibm_mark.
cudaError_t launch_ibm_interp(const void* P, const LatDev& L, int t, const MarkerDev& M, const IbmScratch* mark,
                              double velScale, cudaStream_t s, const int* t_dev = nullptr);
// The list of support sites (after the step's last interpolation; it touches
// no populations), and the spread (after the list and the lattice step).
cudaError_t launch_ibm_mark(const LatDev& L, const MarkerDev& M, const IbmScratch& W, cudaStream_t s);
cudaError_t launch_ibm_spread(const void* A, void* B, const LatDev& L, int t, const MarkerDev& M,
                              const IbmScratch& W, cudaStream_t s);

}  // namespace life
