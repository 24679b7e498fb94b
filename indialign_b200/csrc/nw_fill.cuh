// The NW fill and traceback of the search's own score matrices (distance
// scores of a transform, SS labels): Needleman-Wunsch over a matrix that is
// computed on the fly from the transformed pred rows and the native columns
// (indialign_c/nw.h:10-68, align.h:86-98, ss.h:56-136).
//
// Shape.  A lane owns R consecutive rows of a stripe of 32 R rows and computes
// a block of R rows x 2 columns per step; lane l trails lane l-1 by one step,
// so the two bottom values of a lane reach the next lane by a shuffle of the
// step before.  The fill is bound by instruction issue and instruction fetch
// (the chip's warps run several loops at once and each loop's code competes
// for the instruction cache), so the step is shaped to be short, in issue
// slots per cell and in code:
//   * the two columns of a row share paired FP32 instructions for the score
//     entry (difference, d2, 1 + d2/d0^2, and the reciprocal's Newton step):
//     half an instruction per cell each, with the native columns staged
//     negated in pairs;
//   * a direction is two bits in two planes, "not diagonal" and "left < up",
//     each taken from the sign of one subtraction (FMA pipe) and shifted into
//     its word by one funnel shift, instead of compares and selects (ALU pipe).
//     All values are finite there, so a difference is +0 or positive exactly
//     when the comparison holds;
//   * one step's bookkeeping (shuffles, loads, loop) is shared by 2 R cells and
//     has no branch: a stripe's lanes start together, and a lane whose first
//     column has not come yet works on staged NaN columns, on which a cell
//     leaves H = 0, the boundary value; columns and the boundary row carry
//     padding on both sides, so no index is clamped;
//   * the cutoff and the gap are factors (0 or 1) of fused multiply-adds, not
//     compares and selects: the ALU pipe runs at half the FMA pipe's rate.
// Stripes run one after the other (31 idle lane steps each).  The stripe's last
// row goes to the next stripe through a boundary row in memory.  W warps may
// share one alignment: warp w takes stripes w, w + W, ..., publishes per 16
// steps how many boundary pairs it has written, and waits (bounded) for those
// of the stripe above before it starts a group of 16.
//
// Measured (B200) against two rows per lane and one column per step with
// scalar entries, compare / select directions and a cell-by-cell traceback:
// fill 14 -> 3.0 warp cycles per cell on 48 pairs of L 30-1500, 19.5 -> 3.6 on
// 64 pairs of L 40-300 (whose last stripes are emptier; with selects for the
// cutoff and the gap 3.3 and 4.3); traceback 0.8 -> 0.14
// and 2.9 -> 0.72.  Lanes that wrap into the next stripe without draining, with
// the entry code inside the step loop, took 4.4 and 8.7 (half of the warps'
// time without an instruction to issue); unrolling that loop twice, 6.3 and 15.
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
    const float *q;           // native column pairs (stage_columns), pair 0
    const uint8_t *Lp, *Ln;   // SS labels (SS modes)
    float gap, inv_d0sq, cut2;
    uint32_t *trace;          // the alignment's trace block
    float *bw;                // boundary row this warp writes, pair 0
    const float *br;          // boundary row of the stripe above (W = 1: the same row)
    volatile int *prog;       // W > 1: per warp, boundary pairs written
    int *err;
};

// Native column pair k as {-x0, -x1, -y0, -y1, -z0, -z1} at dst + 6 k, for
// k = -kFillPad .. pairs + kFillPad - 1: NaN left of the matrix (see
// fill_cell), the last pair's values right of it.  A point with a non-finite
// coordinate, or one beyond kFar, is put at 2 kFar (moved_row puts such rows at
// -2 kFar): beyond the cutoff of every other point, as the comparison with NaN,
// infinity or a far distance makes it, with a finite square.  The modes SS4 (no
// cutoff) and SMAT_DP_FAR (far points may coincide) take the values as they are
// (`raw`).
IA_DEV void stage_columns(float *dst, const double *Q, int nlen, bool raw, int tid, int nthreads) {
    const int pairs = (nlen + 1) >> 1;
    for (int e = tid; e < 2 * (pairs + 2 * kFillPad); e += nthreads) {
        const int k = (e >> 1) - kFillPad, half = e & 1;
        const int c = fill_column(k, half, nlen);
        float x = NAN, y = NAN, z = NAN;
        if (c >= 0) {
            const double *q = Q + 3 * (size_t)c;
            x = (float)q[0];
            y = (float)q[1];
            z = (float)q[2];
            if (!raw && is_far(x, y, z)) x = y = z = 2 * kFar;
        }
        float *o = dst + 6 * k + half;
        o[0] = -x;
        o[2] = -y;
        o[4] = -z;
    }
}

// The cutoff as a factor of the FMA pipe instead of a compare and a select:
// with c the next float above cut2, sat((c - d2) 2^40) is 1 for d2 <= cut2 (the
// difference is then at least one unit in the last place of cut2, 2^-20 for
// the search's smallest cutoff of 3.5^2, and 1 already from cut2 >= 2^-16 on)
// and 0 for d2 >= c.
constexpr float kCutScale = 1099511627776.f;  // 2^40
IA_DEV float cut_limit(float cut2) { return nextafterf(cut2, INFINITY) * kCutScale; }

// Score entries of one row (its point in every half of mx, my, mz) and two
// columns: 1/(1 + d2/d0^2), or 0 beyond the cutoff (distance mode; NaN left of
// the matrix); plus 0.5 for equal labels (SS4); label identity (SS2).  In the
// mode SMAT_DP_FAR the squares may overflow, and the cutoff (`limit` is cut2
// itself) is a comparison.
// Operation order of a term: d2 = fma(dz, dz, fma(dx, dx, dy dy)),
// fma(d2, 1/d0^2, 1).
template <int SMODE>
IA_DEV float2 score_pair(float2 mx, float2 my, float2 mz, float2 qx, float2 qy, float2 qz, float2 ninv, float inv,
                         float limit, uint8_t lp, uint8_t ln0, uint8_t ln1, bool left_of) {
    float2 r;
    if (SMODE == SMAT_SS2) {
        r = make_float2(lp == ln0 ? 1.f : 0.f, lp == ln1 ? 1.f : 0.f);
        return left_of ? make_float2(NAN, NAN) : r;
    }
    const float2 dx = __fadd2_rn(mx, qx), dy = __fadd2_rn(my, qy), dz = __fadd2_rn(mz, qz);
    const float2 d2 = __ffma2_rn(dz, dz, __ffma2_rn(dx, dx, __fmul2_rn(dy, dy)));
    if (SMODE == SMAT_SS4 || SMODE == SMAT_DP_FAR) {  // infinite and NaN distances reach the reciprocal
        const float r0 = __frcp_rn(fmaf(d2.x, inv, 1.f)), r1 = __frcp_rn(fmaf(d2.y, inv, 1.f));
        if (SMODE == SMAT_SS4) r = make_float2(lp == ln0 ? r0 + 0.5f : r0, lp == ln1 ? r1 + 0.5f : r1);
        else r = make_float2(d2.x <= limit ? r0 : 0.f, d2.y <= limit ? r1 : 0.f);
        return left_of ? make_float2(NAN, NAN) : r;
    }
    const float2 nden = __ffma2_rn(d2, ninv, make_float2(-1.f, -1.f));  // -(1 + d2/d0^2)
    float2 y, e2;
    rcp_pair(nden, y, e2);
    // 1 within the cutoff, 0 beyond (cut_limit)
    float2 k;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(k.x) : "f"(d2.x), "f"(-kCutScale), "f"(limit));
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(k.y) : "f"(d2.y), "f"(-kCutScale), "f"(limit));
    const float2 yk = __fmul2_rn(y, k);
    return __ffma2_rn(yk, e2, yk);
}

// One cell (indialign_c/nw.h:20-35): diag wins ties, then left, then up; a gap
// move out of a cell that was reached diagonally pays `gap`, so a cell hands
// on its H and, for gap moves, hp = H (+ gap if diagonal).  `a` and `b` take
// the bits "not diagonal" and "left < up".  A NaN score left of the matrix
// (left = up = 0) gives H = hp = 0.
template <int SMODE>
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
    float isd;  // 1 if diagonal: one compare to a factor instead of compare, add and select
    asm("set.ge.f32.f32 %0, %1, %2;" : "=f"(isd) : "f"(diag), "f"(m));
    hp = fmaf(isd, gap, h);
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

// Row i of the matrix: the moved pred point, FP64, rounded once.
IA_DEV float3 moved_row(const FillArgs &A, int i, bool raw) {
    const double *p = A.P + 3 * (size_t)i;
    double x, y, z;
    xform(A.rt, A.rt + 9, p[0], p[1], p[2], x, y, z);
    float3 m = make_float3((float)x, (float)y, (float)z);
    if (!raw && is_far(m.x, m.y, m.z)) m.x = m.y = m.z = -2 * kFar;
    return m;
}

// Fill the trace of the stripes of warp w.  Called by whole warps; with W > 1
// by all W warps of the alignment, prog[] zeroed before.  Inlined: as a call it
// gets the registers that the chain loop leaves over (k_chain of 48 pairs of L
// 30-1500 151 ms against 152 to 159, by what lives around it).
template <int SMODE, int R>
IA_DEV void nw_fill(const FillArgs &A, const FillGeom G, int w) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int plen = A.plen, nlen = A.nlen, W = G.W, S = G.S;
    const int np = (nlen + 1) >> 1;
    const float gap = A.gap, inv = A.inv_d0sq, limit = SMODE == SMAT_DP_FAR ? A.cut2 : cut_limit(A.cut2);
    const float2 ninv = make_float2(-inv, -inv);
    for (int k = w; k < S; k += W) {
        const int row0 = (k * 32 + lane) * R;
        const bool ok = row0 < plen;  // the lane has a row of the matrix
        float2 mx[R], my[R], mz[R];
        uint8_t lp[R];
        float h[R], hp[R];
        uint32_t ta[R], tb[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int i = min(row0 + r, plen - 1);
            if (SMODE != SMAT_SS2) {
                const float3 m = moved_row(A, i, SMODE != SMAT_DP);
                mx[r] = make_float2(m.x, m.x);
                my[r] = make_float2(m.y, m.y);
                mz[r] = make_float2(m.z, m.z);
            } else {
                mx[r] = my[r] = mz[r] = make_float2(0.f, 0.f);
            }
            lp[r] = SMODE == SMAT_SS2 || SMODE == SMAT_SS4 ? A.Lp[i] : (uint8_t)0;
            h[r] = hp[r] = 0.f;
            ta[r] = tb[r] = 0u;
        }
        float upprev = 0.f, hb0 = 0.f, hb1 = 0.f, pb0 = 0.f, pb1 = 0.f;
        // lane 0 reads the boundary row of the stripe above, one pair ahead;
        // lane 31 writes this stripe's
        const bool rd = lane == 0 && k > 0, wr = lane == 31 && k + 1 < S;
        const float *qp = A.q - 6 * lane, *rp = A.br;
        float *wp = A.bw - 4 * 31;
        uint32_t *tp = A.trace + ((size_t)k * G.G * 32 + lane) * (2 * R);
        const int steps = np + (k == S - 1 ? (plen - 1 - k * 32 * R) / R : 31);
        const int qw = k / W, span = np + 64;  // progress: stripes of a warp, pairs
        float4 bn = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int t0 = 0; t0 < steps; t0 += 16) {
            if (W > 1 && k > 0) {
                // pairs that lane 0 reads in this group (one ahead), written by
                // the warp of stripe k - 1
                const int need = (w > 0 ? qw : qw - 1) * span + min(t0 + 17, np);
                const int wprod = w > 0 ? w - 1 : W - 1;
                uint32_t it = 0;
                while (A.prog[wprod] < need && ++it < kFillWaitLimit) {
                }
                if (it >= kFillWaitLimit && lane == 0) atomicOr(A.err, DERR_NW_TIMEOUT);
                __threadfence_block();
            }
            __syncwarp();
            if (t0 == 0 && rd) bn = *reinterpret_cast<const float4 *>(rp);
            const int n16 = min(16, steps - t0);
#pragma unroll 1
            for (int u = n16; u > 0; u--) {
                float up0 = __shfl_up_sync(kFull, hb0, 1), up1 = __shfl_up_sync(kFull, hb1, 1);
                float pu0 = __shfl_up_sync(kFull, pb0, 1), pu1 = __shfl_up_sync(kFull, pb1, 1);
                if (lane == 0) {
                    up0 = bn.x;
                    up1 = bn.z;
                    pu0 = bn.y;
                    pu1 = bn.w;
                }
                rp += 4;
                if (rd) bn = *reinterpret_cast<const float4 *>(rp);
                float2 qx, qy, qz;
                uint8_t ln0 = 0, ln1 = 0;
                bool left_of = false;
                if (SMODE != SMAT_SS2) {
                    qx = reinterpret_cast<const float2 *>(qp)[0];
                    qy = reinterpret_cast<const float2 *>(qp)[1];
                    qz = reinterpret_cast<const float2 *>(qp)[2];
                }
                if (SMODE != SMAT_DP) {
                    const int s = t0 + n16 - u - lane;
                    left_of = s < 0;
                    ln0 = A.Ln[min(max(2 * s, 0), nlen - 1)];
                    ln1 = A.Ln[min(max(2 * s + 1, 0), nlen - 1)];
                }
                qp += 6;
                float2 e[R];
#pragma unroll
                for (int r = 0; r < R; r++)
                    e[r] = score_pair<SMODE>(mx[r], my[r], mz[r], qx, qy, qz, ninv, inv, limit, lp[r], ln0, ln1, left_of);
                float n0[R], p0[R];
#pragma unroll
                for (int r = 0; r < R; r++)
                    fill_cell<SMODE>(r == 0 ? upprev : h[r > 0 ? r - 1 : 0], e[r].x, r == 0 ? pu0 : p0[r > 0 ? r - 1 : 0],
                                     hp[r], gap, n0[r], p0[r], ta[r], tb[r]);
#pragma unroll
                for (int r = 0; r < R; r++)
                    fill_cell<SMODE>(r == 0 ? up0 : n0[r > 0 ? r - 1 : 0], e[r].y, r == 0 ? pu1 : hp[r > 0 ? r - 1 : 0],
                                     p0[r], gap, h[r], hp[r], ta[r], tb[r]);
                upprev = up1;
                hb0 = n0[R - 1];
                hb1 = h[R - 1];
                pb0 = p0[R - 1];
                pb1 = hp[R - 1];
                if (wr) *reinterpret_cast<float4 *>(wp) = make_float4(hb0, pb0, hb1, pb1);
                wp += 4;
            }
            if (ok) store_words<R>(tp, ta, tb, 2 * (16 - n16));
            tp += 64 * R;
#pragma unroll
            for (int r = 0; r < R; r++) ta[r] = tb[r] = 0u;
            if (W > 1) {
                __threadfence_block();
                __syncwarp();
                if (lane == 0) A.prog[w] = qw * span + max(t0 + n16 - 31, 0);
            }
        }
        __syncwarp();
    }
}

// One code for every gap penalty: without one, hp = H + 0.  A version without
// the hp values has fewer instructions, but half of a launch's chains run it
// beside the other half's, and the two loops together cost more in instruction
// fetch than they save (k_chain of 64 pairs of L 40-300: 74.0 ms against 60.3).
template <int SMODE>
IA_DEV void nw_fill_r(const FillArgs &A, const FillGeom &G, int w) {
    if (G.R == 4) nw_fill<SMODE, 4>(A, G, w);
    else nw_fill<SMODE, 3>(A, G, w);
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
    const int lane = threadIdx.x & 31, R = G.R;
    int i = plen, j = nlen, cnt = 0;
    while (i > 0 && j > 0) {
        const int r = i - lane;  // this lane's row (1-based)
        unsigned long long pa = 0, pb = 0;
        int c = 0;  // position of column jj in the plane words: c - jj
        if (r >= 1) {
            const int k = (r - 1) / (32 * R), ri = (r - 1) - k * 32 * R, l = ri / R, rr = ri - l * R;
            const int word = (l + ((j - 1) >> 1)) >> 4;
            const uint32_t *p = trace + ((size_t)(k * G.G + word) * 32 + l) * (2 * R) + 2 * rr;
            uint2 lo = *reinterpret_cast<const uint2 *>(p), hi = make_uint2(0u, 0u);
            if (word > 0) hi = *reinterpret_cast<const uint2 *>(p - 64 * R);
            pa = ((unsigned long long)hi.x << 32) | lo.x;
            pb = ((unsigned long long)hi.y << 32) | lo.y;
            c = 32 * word + 32 - 2 * l;
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
            if (code > 0) {  // (the bits left of the matrix are arbitrary)
                j = max(j - code, 0);
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
