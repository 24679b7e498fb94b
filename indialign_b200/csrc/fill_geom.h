// Geometry of the NW fill (nw_fill.cuh), shared by host and device: rows per
// lane, stripes and trace layout of one alignment.
#pragma once
#include <math.h>
#include <stddef.h>

#ifdef __CUDACC__
#define IA_GEOM_FN __host__ __device__ inline
#else
#define IA_GEOM_FN inline
#endif

namespace ia {

struct FillGeom {
    int R;  // rows per lane
    int S;  // stripes of 32 R rows
    int W;  // warps sharing the alignment (stripe k belongs to warp k % W)
    int G;  // 16-step trace groups per stripe
};

// Points beyond this, in any coordinate, are kept from the distance fill's
// squares, which would overflow FP32 (three of 4 kFar, the longest difference
// that the fill's stand-ins for such points make, do not).
constexpr float kFar = 1e18f;
IA_GEOM_FN bool is_far(float x, float y, float z) {
    return !(fabsf(x) <= kFar && fabsf(y) <= kFar && fabsf(z) <= kFar);
}
// ... with FP32 coordinates that are finite: two such points may coincide.
IA_GEOM_FN bool is_far_point(const double *q) {
    const float x = (float)q[0], y = (float)q[1], z = (float)q[2];
    return is_far(x, y, z) && fabsf(x) < INFINITY && fabsf(y) < INFINITY && fabsf(z) < INFINITY;
}

// Padding pairs on each side of the staged columns and of a boundary row: a
// lane is up to 31 pairs left of the matrix when its stripe starts and up to
// 31 right of it when the stripe's last lane is done, and the boundary row is
// read one pair ahead.
constexpr int kFillPad = 33;

// Steps by which a stripe of another warp trails the stripe above: 32 lanes
// and the 16-step groups in which progress is published.
constexpr int kFillLag = 49;

// Rows per lane by the modelled issue slots: steps x (20 per step of
// bookkeeping + 32 per row of 2 cells).  More rows per lane share the
// bookkeeping; fewer leave fewer idle rows in the last stripe and, with
// several warps, give more stripes to share.  Three rows are taken when they
// save an eighth or more: warps that run the other loop at the same time cost
// instruction fetches.  k_chain, ms, on 64 pairs of L 40-300 / 160 pairs of L
// 20-1100: four rows only 54.4 / 87.0, three or four 52.6 / 86.6, without the
// eighth 52.7 / 87.4, two as well 53.1 / 87.8.
IA_GEOM_FN FillGeom fill_geom(int plen, int nlen, int W) {
    const int n32 = (plen + 31) >> 5, np = (nlen + 1) >> 1;
    FillGeom g = {4, n32, W, 0};
    long long best = -1;
    for (int R = 4; R >= 3; R--) {
        const int S = (n32 + R - 1) / R, rounds = (S + W - 1) / W;
        const long long steps = (long long)rounds * (np + 31) + ((S < W ? S : W) - 1) * kFillLag;
        const long long cost = steps * (20 + 32 * R) * (R < 4 ? 9 : 8);
        if (best < 0 || cost < best) {
            best = cost;
            g.R = R;
            g.S = S;
        }
    }
    g.G = (np + 31 + 15) / 16;
    return g;
}

// Native residue staged as column `half` of pair k of nlen columns: the last one
// right of the matrix; -1 left of it and where there is none (nlen = 0: pairs
// without a valid native residue have chains too).
IA_GEOM_FN int fill_column(int k, int half, int nlen) {
    if (k < 0 || nlen < 1) return -1;
    return 2 * k + half < nlen ? 2 * k + half : nlen - 1;
}

// Trace words of any alignment of at most np x nn under any choice of rows per
// lane: 2 bits per cell in 2 planes; R S <= ceil(np / 32) + 3.
constexpr size_t fill_trace_words(int np, int nn) {
    return (size_t)((np + 31) / 32 + 3) * 64 * (size_t)(((nn + 1) / 2 + 31 + 15) / 16);
}

// Floats of a boundary row (per column pair H and its gap form, twice) and of
// the staged columns for nn columns, with their padding.
constexpr size_t fill_boundary_floats(int nn) { return (size_t)((nn + 1) / 2 + 2 * kFillPad) * 4; }
constexpr size_t fill_column_floats(int nn) { return (size_t)((nn + 1) / 2 + 2 * kFillPad) * 6; }

}  // namespace ia
