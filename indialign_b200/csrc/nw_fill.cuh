// The NW fill and traceback of the search's own score matrices (distance
// scores of a transform, SS labels): Needleman-Wunsch over a matrix that is
// computed on the fly from the transformed pred rows and the native columns
// (indialign_c/nw.h:10-68, align.h:86-98, ss.h:56-136).
//
// Shape.  A lane owns R consecutive rows (R <= 4) of a stripe of 32 R rows and
// computes a block of R rows x 2 columns per step; lane l trails lane l-1 by
// one step, so the two bottom values of a lane reach the next lane by a
// shuffle of the step before.  The fill is bound by instruction issue and the
// half-rate ALU pipe, so the block is shaped to spend as few instructions per
// cell as possible:
//   * the two columns of a row share paired FP32 instructions for the score
//     entry (difference, d2, 1 + d2/d0^2, and the reciprocal's Newton step):
//     half an instruction per cell each, with the native columns staged
//     negated in pairs so that a step loads them with two shared-memory reads;
//   * one step's bookkeeping (shuffles, loads, loop, boundary) is shared by
//     2 R cells;
//   * a direction is two bits in two planes, "not diagonal" and "left < up",
//     each taken from the sign of one subtraction (FMA pipe) and shifted into
//     its word by one funnel shift, instead of compares and selects (ALU pipe).
//     All values are finite and >= 0 there, so a difference is +0 or positive
//     exactly when the comparison holds.
// A warp walks stripes w, w + W, w + 2W, ... (W warps share one alignment, or
// W = 1); its lanes wrap into the next stripe without draining, with period
// P2 steps.  The stripe's last row goes to the next stripe through a boundary
// row in memory; with W > 1 the producer publishes its step count once per 16
// steps and the consumer waits (bounded) before it starts a group of 16.
#pragma once
#include "dmath.cuh"
#include "fill_geom.h"
#include "kernels.h"
#include "pipeline.h"

namespace ia {

constexpr uint32_t kFillWaitLimit = 1u << 24;  // polls of a neighbour's progress before giving up

struct FillArgs {
    int plen, nlen;
    const double *P;          // compact pred xyz
    const double *rt;         // transform {R[9], t[3]}
    const float4 *qa;         // native column pairs {-x0, -x1, -y0, -y1} ...
    const float2 *qb;         // ... {-z0, -z1} (shared memory), or null:
    const double *Q;          // compact native xyz, converted on load
    const uint8_t *Lp, *Ln;   // SS labels (SS modes)
    float gap, inv_d0sq, cut2;
    uint32_t *trace;          // the alignment's trace block
    float *bw;                // boundary row this warp writes
    const float *br;          // boundary row of the stripe above (W = 1: the same row)
    volatile int *prog;       // W > 1: per warp, steps whose boundary values are written
    int *err;
};

// 1/x for x in [1, 2^127), correctly rounded: the hardware approximation
// (within 1 ulp) and one Newton-Raphson step with a fused residual, which
// rounds correctly for every float of that range (compared with __frcp_rn
// over all of them by the test suite).
IA_DEV float rcp_f32(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return fmaf(y, fmaf(-x, y, 1.f), y);
}

// Score entries of one row (its point in every half of mx, my, mz) and two
// columns: 1/(1 + d2/d0^2), or 0 beyond the cutoff (distance mode); plus 0.5
// for equal labels (SS4); label identity (SS2).  Operation order of a term:
// d2 = fma(dz, dz, fma(dx, dx, dy dy)), fma(d2, 1/d0^2, 1).
template <int SMODE>
IA_DEV float2 score_pair(float2 mx, float2 my, float2 mz, float4 qa, float2 qb, float2 ninv, float2 none, float inv,
                         float cut2, uint8_t lp, uint8_t ln0, uint8_t ln1) {
    if (SMODE == SMAT_SS2) return make_float2(lp == ln0 ? 1.f : 0.f, lp == ln1 ? 1.f : 0.f);
    const float2 dx = __fadd2_rn(mx, make_float2(qa.x, qa.y)), dy = __fadd2_rn(my, make_float2(qa.z, qa.w)),
                 dz = __fadd2_rn(mz, qb);
    const float2 d2 = __ffma2_rn(dz, dz, __ffma2_rn(dx, dx, __fmul2_rn(dy, dy)));
    if (SMODE == SMAT_SS4) {  // no cutoff: infinite and NaN distances reach the reciprocal
        const float r0 = __frcp_rn(fmaf(d2.x, inv, 1.f)), r1 = __frcp_rn(fmaf(d2.y, inv, 1.f));
        return make_float2(lp == ln0 ? r0 + 0.5f : r0, lp == ln1 ? r1 + 0.5f : r1);
    }
    const float2 nden = __ffma2_rn(d2, ninv, none);  // -(1 + d2/d0^2)
    float2 y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(-nden.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(-nden.y));
    const float2 r = __ffma2_rn(y, __ffma2_rn(nden, y, make_float2(1.f, 1.f)), y);
    return make_float2(d2.x <= cut2 ? r.x : 0.f, d2.y <= cut2 ? r.y : 0.f);
}

// One cell (indialign_c/nw.h:20-35): diag wins ties, then left, then up; a gap
// move out of a cell that was reached diagonally pays `gap`, so a cell hands
// on its H and, for gap moves, hp = H (+ gap if diagonal).  `a` and `b` take
// the bits "not diagonal" and "left < up".
template <int SMODE, bool GAP>
IA_DEV void fill_cell(float diag_src, float sc, float up, float left, float gap, float &h, float &hp, uint32_t &a,
                      uint32_t &b) {
    const float diag = diag_src + sc;
    if (SMODE == SMAT_SS4) {  // NaN scores: plain comparisons, H kept non-negative as the sign-encoded form does
        const bool isd = diag >= up && diag >= left, lu = left >= up;
        const float v = isd ? diag : (lu ? left : up);
        const float enc = isd ? -v : v;
        h = fabsf(enc);
        hp = h + (signbit(enc) ? gap : 0.f);
        a = (a << 1) | (isd ? 0u : 1u);
        b = (b << 1) | (lu ? 0u : 1u);
        return;
    }
    const float m = fmaxf(left, up), x = diag - m, y = left - up;
    a = __funnelshift_l(__float_as_uint(x), a, 1);
    b = __funnelshift_l(__float_as_uint(y), b, 1);
    h = fmaxf(diag, m);
    if (GAP) hp = diag >= m ? diag + gap : m;
    else hp = h;
}

// A lane's 2R trace words of one 16-step group, shifted left by sh.
template <int R>
IA_DEV void store_words(uint32_t *p, const uint32_t (&a)[R], const uint32_t (&b)[R], int sh) {
    if (R % 2 == 0) {
#pragma unroll
        for (int r = 0; r + 1 < R; r += 2)
            reinterpret_cast<uint4 *>(p)[r / 2] = make_uint4(a[r] << sh, b[r] << sh, a[r + 1] << sh, b[r + 1] << sh);
    } else {
#pragma unroll
        for (int r = 0; r < R; r++) reinterpret_cast<uint2 *>(p)[r] = make_uint2(a[r] << sh, b[r] << sh);
    }
}

// Fill the trace of the stripes of warp w.  slot: 3 R x 32 floats of shared
// memory of this warp (the moved points of its next stripe).  Called by whole
// warps; with W > 1 by all W warps of the alignment, prog[] zeroed before.
template <int SMODE, bool GAP, int R>
__device__ __noinline__ void nw_fill(const FillArgs &A, const FillGeom G, int w, float *slot) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int plen = A.plen, nlen = A.nlen, W = G.W, P2 = G.P2, S = G.S;
    const int np = (nlen + 1) >> 1;
    const int nq = S > w ? (S - w + W - 1) / W : 0;  // stripes of this warp
    if (nq == 0) return;
    const int k_last = w + (nq - 1) * W;
    const int last_lane = k_last == S - 1 ? (plen - 1 - k_last * 32 * R) / R : 31;
    const int total = (nq - 1) * P2 + last_lane + np;
    const float gap = A.gap, inv = A.inv_d0sq, cut2 = A.cut2;
    const float2 ninv = make_float2(-inv, -inv), none = make_float2(-1.f, -1.f);
    const float4 *qa = A.qa;
    const float2 *qb = A.qb;
    float2 mx[R], my[R], mz[R];
    uint8_t lp[R];
    float h[R], hp[R];
    uint32_t ta[R], tb[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        mx[r] = my[r] = mz[r] = make_float2(0.f, 0.f);
        h[r] = hp[r] = 0.f;
        ta[r] = tb[r] = 0u;
        lp[r] = 0;
    }
    float upprev = 0.f, hb0 = 0.f, hb1 = 0.f, pb0 = 0.f, pb1 = 0.f;
    float4 bn = make_float4(0.f, 0.f, 0.f, 0.f);  // lane 0: the boundary values of its next pair
    int s = P2 - lane, q = -1;                    // column pair, stripe of this lane
    bool ok = false;                              // the lane has a row of the matrix
    int wlim = 0, rlim = 0;                       // pairs whose boundary this lane writes / reads
    uint32_t *wp = A.trace;
    int tq = 0, qn = 0;  // step at which lane 0 enters its next stripe, and that stripe
    for (int t0 = 0; t0 < total; t0 += 16) {
        if (tq < t0 + 16 && qn < nq) {
            // moved points of the stripe entered next (FP64 transform, rounded
            // once), for all lanes together; the last reader of the slot's old
            // content entered at tq - P2 + 31 < t0 (fill_min_period)
            double Rm[9], tm[3];
#pragma unroll
            for (int a = 0; a < 9; a++) Rm[a] = A.rt[a];
#pragma unroll
            for (int a = 0; a < 3; a++) tm[a] = A.rt[9 + a];
            const int row0 = ((w + qn * W) * 32 + lane) * R;
            if (SMODE != SMAT_SS2) {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const double *p = A.P + 3 * (size_t)min(row0 + r, plen - 1);
                    double ax, ay, az;
                    xform(Rm, tm, p[0], p[1], p[2], ax, ay, az);
                    slot[(3 * r) * 32 + lane] = (float)ax;
                    slot[(3 * r + 1) * 32 + lane] = (float)ay;
                    slot[(3 * r + 2) * 32 + lane] = (float)az;
                }
            }
            tq += P2;
            qn++;
        }
        if (W > 1) {
            // the boundary pairs that lane 0 reads in this group (one ahead)
            int ql = t0 / P2, sl = t0 - ql * P2 + 16;
            if (sl >= P2) {
                ql++;
                sl -= P2;
            }
            if (ql >= nq) {
                ql = nq - 1;
                sl = np;
            }
            const int qp = w > 0 ? ql : ql - 1, wprod = w > 0 ? w - 1 : W - 1;
            if (qp >= 0) {
                const int need = qp * P2 + 32 + min(sl, np - 1);
                uint32_t it = 0;
                while (A.prog[wprod] < need && ++it < kFillWaitLimit) {
                }
                if (it >= kFillWaitLimit && lane == 0) atomicOr(A.err, DERR_NW_TIMEOUT);
                __threadfence_block();
            }
        }
        __syncwarp();
        const int n16 = min(16, total - t0);
#pragma unroll 1
        for (int u = 0; u < n16; u++) {
            float up0 = __shfl_up_sync(kFull, hb0, 1), up1 = __shfl_up_sync(kFull, hb1, 1);
            float pu0 = up0, pu1 = up1;
            if (GAP) {
                pu0 = __shfl_up_sync(kFull, pb0, 1);
                pu1 = __shfl_up_sync(kFull, pb1, 1);
            }
            if (s == P2) {  // enter the next stripe (once per P2 steps)
                if (ok && u > 0) store_words<R>(wp, ta, tb, 2 * (16 - u));
                s = 0;
                q++;
                const int k = w + q * W, row0 = (k * 32 + lane) * R;
                ok = q < nq && row0 < plen;
                upprev = 0.f;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    h[r] = hp[r] = 0.f;
                    ta[r] = tb[r] = 0u;
                    const float a = slot[(3 * r) * 32 + lane], b = slot[(3 * r + 1) * 32 + lane],
                                c = slot[(3 * r + 2) * 32 + lane];
                    mx[r] = make_float2(a, a);
                    my[r] = make_float2(b, b);
                    mz[r] = make_float2(c, c);
                    if (SMODE == SMAT_SS2 || SMODE == SMAT_SS4) lp[r] = A.Lp[min(row0 + r, plen - 1)];
                }
                wp = A.trace + ((size_t)(k * G.G + ((t0 + u) >> 4) - ((q * P2) >> 4)) * 32 + lane) * (2 * R);
                wlim = lane == 31 && ok && k + 1 < S ? np : 0;
                rlim = lane == 0 && ok && k > 0 ? np : 0;
                bn = make_float4(0.f, 0.f, 0.f, 0.f);
                if (rlim > 0) {
                    if (GAP) bn = *reinterpret_cast<const float4 *>(A.br);
                    else {
                        const float2 v = *reinterpret_cast<const float2 *>(A.br);
                        bn.x = v.x;
                        bn.z = v.y;
                    }
                }
            }
            if (lane == 0) {
                up0 = bn.x;
                up1 = bn.z;
                pu0 = GAP ? bn.y : bn.x;
                pu1 = GAP ? bn.w : bn.z;
            }
            if ((unsigned)(s + 1) < (unsigned)rlim) {  // lane 0: prefetch
                if (GAP) bn = reinterpret_cast<const float4 *>(A.br)[s + 1];
                else {
                    const float2 v = reinterpret_cast<const float2 *>(A.br)[s + 1];
                    bn.x = v.x;
                    bn.z = v.y;
                }
            }
            // column pair; a pair outside the matrix is computed on the last
            // one and never read by a cell inside it
            const int sc = (int)min((unsigned)s, (unsigned)(np - 1));
            float4 va = make_float4(0.f, 0.f, 0.f, 0.f);
            float2 vb = make_float2(0.f, 0.f);
            uint8_t ln0 = 0, ln1 = 0;
            if (SMODE != SMAT_SS2) {
                if (qa) {
                    va = qa[sc];
                    vb = qb[sc];
                } else {
                    const double *q0 = A.Q + 6 * (size_t)sc, *q1 = 2 * sc + 1 < nlen ? q0 + 3 : q0;
                    va = make_float4(-(float)q0[0], -(float)q1[0], -(float)q0[1], -(float)q1[1]);
                    vb = make_float2(-(float)q0[2], -(float)q1[2]);
                }
            }
            if (SMODE == SMAT_SS2 || SMODE == SMAT_SS4) {
                ln0 = A.Ln[2 * sc];
                ln1 = A.Ln[min(2 * sc + 1, nlen - 1)];
            }
            float2 e[R];
#pragma unroll
            for (int r = 0; r < R; r++)
                e[r] = score_pair<SMODE>(mx[r], my[r], mz[r], va, vb, ninv, none, inv, cut2, lp[r], ln0, ln1);
            float n0[R], p0[R];
#pragma unroll
            for (int r = 0; r < R; r++)
                fill_cell<SMODE, GAP>(r == 0 ? upprev : h[r > 0 ? r - 1 : 0], e[r].x, r == 0 ? pu0 : p0[r > 0 ? r - 1 : 0],
                                      hp[r], gap, n0[r], p0[r], ta[r], tb[r]);
#pragma unroll
            for (int r = 0; r < R; r++)
                fill_cell<SMODE, GAP>(r == 0 ? up0 : n0[r > 0 ? r - 1 : 0], e[r].y, r == 0 ? pu1 : hp[r > 0 ? r - 1 : 0],
                                      p0[r], gap, h[r], hp[r], ta[r], tb[r]);
            upprev = up1;
            hb0 = n0[R - 1];
            hb1 = h[R - 1];
            pb0 = p0[R - 1];
            pb1 = hp[R - 1];
            if ((unsigned)s < (unsigned)wlim) {  // lane 31: the stripe's last row
                if (GAP) reinterpret_cast<float4 *>(A.bw)[s] = make_float4(hb0, pb0, hb1, pb1);
                else reinterpret_cast<float2 *>(A.bw)[s] = make_float2(hb0, hb1);
            }
            s++;
        }
        if (ok) store_words<R>(wp, ta, tb, 2 * (16 - n16));
        wp += 64 * R;
#pragma unroll
        for (int r = 0; r < R; r++) ta[r] = tb[r] = 0u;
        if (W > 1) {
            __threadfence_block();
            __syncwarp();
            if (lane == 0) A.prog[w] = t0 + n16;
        }
    }
    __syncwarp();
}

template <int SMODE, bool GAP>
IA_DEV void nw_fill_r(const FillArgs &A, const FillGeom &G, int w, float *slot) {
    if (G.R == 4) nw_fill<SMODE, GAP, 4>(A, G, w, slot);
    else if (G.R == 3) nw_fill<SMODE, GAP, 3>(A, G, w, slot);
    else if (G.R == 2) nw_fill<SMODE, GAP, 2>(A, G, w, slot);
    else nw_fill<SMODE, GAP, 1>(A, G, w, slot);
}

// The path from (plen, nlen) by the trace's bits (indialign_c/nw.h:42-68);
// the aligned pairs go to al, last first; returns their number.  Lane l holds
// the two plane words around the current column of row rb - l, and the path
// is followed by runs: a diagonal run is found with one ballot over the lanes'
// bits along the diagonal (and written by the lanes side by side), a run of
// left moves with one bit count in the row's word, a run of up moves with one
// ballot along the column.
__device__ __noinline__ inline int nw_traceback(const uint32_t *trace, const FillGeom G, int plen, int nlen, uint32_t *al) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31, R = G.R, W = G.W;
    int i = plen, j = nlen, cnt = 0;
    while (i > 0 && j > 0) {
        const int r = i - lane;  // this lane's row (1-based)
        unsigned long long pa = 0, pb = 0;
        int c = 0;  // position of column jj in the plane words: c - jj
        if (r >= 1) {
            const int k = (r - 1) / (32 * R), ri = (r - 1) - k * 32 * R, l = ri / R, rr = ri - l * R;
            const int base = (k / W) * G.P2, first = (base + l) >> 4, word = (base + l + ((j - 1) >> 1)) >> 4;
            const uint32_t *p = trace + ((size_t)(k * G.G + word - (base >> 4)) * 32 + l) * (2 * R) + 2 * rr;
            uint2 lo = *reinterpret_cast<const uint2 *>(p), hi = make_uint2(0u, 0u);
            if (word > first) hi = *reinterpret_cast<const uint2 *>(p - 64 * R);
            pa = ((unsigned long long)hi.x << 32) | lo.x;
            pb = ((unsigned long long)hi.y << 32) | lo.y;
            c = 32 * word + 32 - 2 * (base + l);
        }
        int q = 0;  // lane of row i
        for (;;) {
            const int off = lane - q, jj = j - off, pos = c - jj;
            const bool in = off >= 0 && r >= 1 && jj >= 1 && pos < 64;
            const bool nd = in && ((pa >> pos) & 1ull);
            const unsigned stop = __ballot_sync(kFull, !in || nd) >> q;
            const int run = stop ? __ffs(stop) - 1 : 32 - q;
            if (off >= 0 && off < run) al[cnt + off] = ((uint32_t)(r - 1) << 16) | (uint32_t)(jj - 1);
            cnt += run;
            i -= run;
            j -= run;
            q += run;
            if (q >= 32 || i <= 0 || j <= 0) break;
            // the owner of row i says: 0 cell not held, > 0 left moves, -1 up
            int code = 0;
            if (nd) {
                const unsigned long long left = ~((pa & ~pb) >> pos);  // zeros: consecutive left moves
                code = (pb >> pos) & 1ull ? -1 : (left ? __ffsll((long long)left) - 1 : 64);
            }
            code = __shfl_sync(kFull, code, q);
            if (code == 0) break;
            if (code > 0) {
                j -= code;
            } else {
                const int pu = c - j;
                const bool up = lane >= q && r >= 1 && pu < 64 && ((pa & pb) >> pu & 1ull);
                const unsigned no = __ballot_sync(kFull, !up) >> q;
                const int ur = no ? __ffs(no) - 1 : 32 - q;
                i -= ur;
                q += ur;
                if (q >= 32) break;
            }
            if (i <= 0 || j <= 0) break;
        }
    }
    __syncwarp();
    return cnt;
}

}  // namespace ia
