// Geometry of the NW fill (nw_fill.cuh), shared by host and device: rows per
// lane, stripes, period and trace layout of one alignment.
#pragma once
#include <stddef.h>

#ifdef __CUDACC__
#define IA_GEOM_FN __host__ __device__ inline
#else
#define IA_GEOM_FN inline
#endif

namespace ia {

struct FillGeom {
    int R;   // rows per lane
    int S;   // stripes of 32 R rows
    int W;   // warps sharing the alignment (stripe k belongs to warp k % W)
    int P2;  // steps (column pairs) from one stripe of a warp to its next
    int G;   // 16-step trace groups per stripe
};

// Least period when a warp walks several stripes.  W = 1: lane 31 writes a
// boundary pair 31 steps after lane 0 computed the pair, and boundary pairs
// and the next stripe's moved points change hands on 16-step group boundaries.
// W > 1: before warp 0 may enter its second stripe, the first boundary pairs
// must have come round through the other warps, each of which needs its
// neighbour 32 steps (and a group of 16 once) ahead, while warp 0 itself does
// not move: 32 W + 31 steps, or the warps would wait for one another.
IA_GEOM_FN constexpr int fill_min_period(int W) { return W > 1 ? 32 * W + 32 : 50; }
constexpr int kFillWarpsMax = 4;  // largest W

// Steps from a stripe's start to the next stripe's in another warp: 32 lanes
// and the 16-step groups in which progress is published.
constexpr int kFillLag = 49;

// Rows per lane by the modelled issue slots: steps x (25 per step of
// bookkeeping + 34 per row of 2 cells).  More rows per lane share the
// bookkeeping; fewer leave fewer idle rows in the last stripe and, with
// several warps, give more stripes to share.
IA_GEOM_FN FillGeom fill_geom(int plen, int nlen, int W) {
    const int n32 = (plen + 31) >> 5, np = (nlen + 1) >> 1;
    FillGeom g = {1, n32, W, np, 0};
    long long best = -1;
    for (int R = 4; R >= 1; R--) {
        const int S = (n32 + R - 1) / R, rounds = (S + W - 1) / W;
        const int P2 = rounds > 1 && np < fill_min_period(W) ? fill_min_period(W) : np;
        const long long steps = (long long)rounds * P2 + ((S < W ? S : W) - 1) * kFillLag + 31;
        const long long cost = steps * (25 + 34 * R);
        if (best < 0 || cost < best) {
            best = cost;
            g.R = R;
            g.S = S;
            g.P2 = P2;
        }
    }
    // a stripe's steps are base .. base + P2 + 30 with any base % 16
    g.G = (g.P2 + 45) / 16 + 1;
    return g;
}

// Trace words of any alignment of at most np x nn under any choice of rows per
// lane: 2 bits per cell in 2 planes; R S <= ceil(np / 32) + 3.
constexpr size_t fill_trace_words(int np, int nn) {
    const int pairs = (nn + 1) / 2, least = fill_min_period(kFillWarpsMax), P2 = pairs < least ? least : pairs;
    return (size_t)((np + 31) / 32 + 3) * 64 * (size_t)((P2 + 45) / 16 + 1);
}

// Floats of a boundary row for nn columns (H and its gap form per column).
constexpr size_t fill_boundary_floats(int nn) { return (size_t)((nn + 1) / 2) * 4; }

}  // namespace ia
