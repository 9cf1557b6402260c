// Which form the boundary-condition sites of a step take (host code; the forms are
// in lbm_walls.cuh).
#pragma once
#include "life_types.h"

namespace life {

// The lane and thread forms share one launch: first the sites for nine lanes (the
// four corners, then the edges of `lanes`: bottom, top, left, right as bits 0..3),
// three a warp, then the edges of `straight`, 32 sites a warp. Edges do not hold
// the corners. general: one thread a site around the whole perimeter instead.
struct WallPlan {
    int lane_sites, lane_warps, lanes, straight;
    int warps;
    int general;
};

#ifdef __CUDACC__
#define LIFE_HD __host__ __device__
#else
#define LIFE_HD
#endif
LIFE_HD inline int edge_sites(const LatDev& L, int e) { return (e < 2 ? L.Nx : L.Ny) - 2; }
LIFE_HD inline int edge_type(const LatDev& L, int e) { return L.wall[(e + 2) & 3]; }  // (walls: left, right, bottom, top)
inline bool step_forced(const LatDev& L) { return L.womersley || L.Fx0 != 0.0 || L.Fy0 != 0.0 || L.site_force; }

// Whether the one-thread form with shared products (wall_site) can take an edge.
inline bool straight_edge(const LatDev& L, int e) {
    const int type = edge_type(L, e);
    const bool formed = type != LIFE_CONVECTIVE || L.outlet_form == kOutletSites;
    return !step_forced(L) && formed && (type == LIFE_WALL || type == LIFE_VELOCITY || type == LIFE_CONVECTIVE);
}
// Sites on the other edges: pressure and free-slip walls, and any wall under a force.
inline int slow_wall_sites(const LatDev& L) {
    int n = 0;
    for (int e = 0; e < 4; e++)
        if (edge_type(L, e) != LIFE_FLUID && !straight_edge(L, e)) n += edge_sites(L, e);
    return n;
}

// A case alone with few boundary sites takes nine lanes for all of them: 14.2 us a
// step against 15.6 (256 x 256, 1020 sites); at 2800 sites the two were even (35.6
// and 35.8, measured where a body's spread waited for the walls), at 4400 the
// threads are ahead (17.2 against 19.4 us, 1501 x 703 FP32), and 64 lattices in a
// batch step in 573 us against 976.
constexpr int kFewWallSites = 2048;

// Nine lanes shorten the chain of a site, but three sites keep the FP64 unit as
// long as 21 of 32 do with a thread each, so from some number of sites on the
// general form takes the slow edges, with their stretches in between.
// Reduced precision: where the lanes' throughput passes the chain of a thread
// (free-slip channels 64 high, us a step, lanes and threads: FP32 BGK 2000 wide
// 19.8 and 22.9, 3000 25.1 and 23.4, 8000 59.8 and 27.3; central moments 2000 26.9
// and 29.1, 3000 35.5 and 30.5, 8000 83.7 and 37.3). In a batch the cases' walls
// fill the chip together (free-slip FP32 channels: 6 of them, 2856 sites, 27.5 and
// 31.6 us, 12, 6864 sites, 42.8 and 33.9; pressure outlets 12, 1640 sites, 28.5 and
// 33.0, 24, 4330 sites, 69.8 and 63.1).
constexpr int kManySlowBgk = 6400, kManySlowCm = 4800, kManySlowBatch = 4000;
// FP64 storage: the interior needs the same unit. Under a force, whose interior is
// all FP64, the threads are ahead once the lattice takes longer than their chain
// (1000 x 64 under gravity 36.1 and 33.0 us, 500 x 64 20.4 and 21.6; central moments
// 500 x 64 40.3 and 35.1, 250 x 64 23.6 and 23.7; 8000 x 400 2728 and 2683), without
// one at 3000 to 4000 slow sites (free-slip 1500 x 64 24.0 and 27.7, 2000 x 64 34.5
// and 30.3; central moments 50.0 and 52.2, 61.0 and 55.7).
constexpr long long kForcedSitesBgk = 50000, kForcedSitesCm = 30000;
constexpr int kManySlowF64 = 3500;

inline bool many_slow_sites(const LatDev& L) {
    const int own = slow_wall_sites(L);
    if (own == 0) return false;
    const long long slow = (long long)own + L.others_slow;
    if (L.prec != LIFE_PREC_F64)
        return slow >= (L.others_sites > 0 ? kManySlowBatch : (L.cm ? kManySlowCm : kManySlowBgk));
    if (step_forced(L)) return (long long)L.Nx * L.Ny + L.others_sites >= (L.cm ? kForcedSitesCm : kForcedSitesBgk);
    return slow >= kManySlowF64;
}

inline WallPlan wall_plan(const LatDev& L) {
    WallPlan p{};
    if (many_slow_sites(L)) {
        p.general = 1;
        p.warps = (2 * L.Nx + 2 * (L.Ny - 2) + 31) / 32;
        return p;
    }
    const bool few = L.others_sites == 0 && 2 * (L.Nx + L.Ny) < kFewWallSites;
    p.lane_sites = 4;
    for (int e = 0; e < 4; e++) {
        if (edge_type(L, e) == LIFE_FLUID) continue;
        if (!few && straight_edge(L, e)) {
            p.straight |= 1 << e;
            p.warps += (edge_sites(L, e) + 31) / 32;
        } else {
            p.lanes |= 1 << e;
            p.lane_sites += edge_sites(L, e);
        }
    }
    p.lane_warps = (p.lane_sites + 2) / 3;
    p.warps += p.lane_warps;
    return p;
}

}  // namespace life
