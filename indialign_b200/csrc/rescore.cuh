// Same-index rescoring of a transform over the full pair.
#pragma once
#include "dmath.cuh"
#include "kernels.h"
#include "pipeline.h"

namespace ia {

// ---- same-index rescoring: tm_score_no_d8 over the full pair
// (indialign_c/indialign.cpp:86-88) -------------------------------------------
IA_DEV double pair_tm(const DevBatch &b, const PairInfo &I, const double *rec, int lane) {
    const int N = I.N, off = I.off;
    const double *P = b.pred + 3 * (size_t)off, *Q = b.nat + 3 * (size_t)off;
    const uint8_t *v = b.v + off;
    const double *R = rec + 1, *t = rec + 10;
    const double inv = 1.0 / fmax(I.d0 * I.d0, 1e-12);
    double s = 0.0;
    for (int i = lane; i < N; i += 32)
        if (v[i]) s += tm_term(dist2(R, t, P[3 * i], P[3 * i + 1], P[3 * i + 2], Q[3 * i], Q[3 * i + 1], Q[3 * i + 2]), inv);
    return warp_sum(s) / fmax(I.lnorm, 1.0);
}

}  // namespace ia
