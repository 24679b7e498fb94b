// NW chains: score matrix + Needleman-Wunsch + traceback + Kabsch + the
// detailed seed search on the alignment, one warp per chain, or one CTA per
// chain when a launch has fewer chains than CTAs.
//
// Restates nw_dp / nw_traceback (indialign_c/nw.h:10-68), dp_refine_chunk
// (indialign_c/align.h:54-145) and the score matrices of ss_nw_align /
// evaluate_ss_seeds (indialign_c/ss.h:56-164).  The fill and the traceback of
// the search's own matrices are in nw_fill.cuh; the NW on an explicit FP64
// matrix is here.
#include <vector>

#include "../../include/indialign_b200.h"
#include "dmath.cuh"
#include "stage.cuh"
#include "pipeline.h"
#include "kernels.h"
#include "sched.cuh"
#include "nw_fill.cuh"

namespace ia {

constexpr unsigned kFull = 0xffffffffu;

// build-time tuning knob: minimum resident CTAs per SM for k_chain (caps
// registers)
#ifndef IA_CHAIN_MINB
#define IA_CHAIN_MINB 4
#endif

// Aligned pair k (forward order) from the reversed traceback list.
IA_DEV void al_get(const uint32_t *al, int na, int k, int &pi, int &ni) {
    uint32_t e = al[na - 1 - k];
    pi = (int)(e >> 16);
    ni = (int)(e & 0xffffu);
}

// One NW cell (indialign_c/nw.h:20-35).  With a gap penalty the "reached
// diagonally" bit of a cell travels in the sign of its H (H >= 0; -0 is a
// diagonal zero) and a gap move out of a diagonal cell pays the penalty;
// without one the bit is irrelevant and H is kept plain.  Ties prefer diag,
// then left, then up.  Selects only, so a step is one basic block.
template <bool GAPZ>
IA_DEV double nw_cell(double diag_src, double sc, double up_enc, double left_enc, double gap, uint32_t &dir) {
    const double diag = diag_src + sc;
    double up, left;
    if (GAPZ) {
        up = up_enc;
        left = left_enc;
    } else {
        up = fabs(up_enc) + (signbit(up_enc) ? gap : 0.0);
        left = fabs(left_enc) + (signbit(left_enc) ? gap : 0.0);
    }
    const bool is_diag = diag >= up && diag >= left;
    const bool l_ge_u = left >= up;
    dir = is_diag ? 0u : (l_ge_u ? 2u : 1u);
    const double nh = is_diag ? diag : (l_ge_u ? left : up);
    return (GAPZ || !is_diag) ? nh : -nh;
}

// Plain value of an encoded H.
template <bool GAPZ>
IA_DEV double hval(double h) { return GAPZ ? h : fabs(h); }

// Trace layout: cell (i, j) of stripe k = (i-1)/64, row ri = (i-1)%64 of it
// (lane ri/2, row ri%2 of the lane) is computed at step t = base(i) + j - 1
// with base(i) = k*P + ri.  Its 2 direction bits sit at bit 2*(t%16) of the
// word at ((k*G + g) * 64 + ri), g = t/16 - (k*P)/16 the step word within
// the stripe, G = (P + 127) / 16 words per stripe (a lane stays in stripe k
// for steps below (k+1)*P + 64, so g < G).  Every lane fills and stores its
// two rows' words on the same steps, at adjacent addresses.
IA_DEV int trace_base(int i, int P) { return ((i - 1) >> 6) * P + ((i - 1) & 63); }
IA_DEV int trace_G(int P) { return (P + 127) / 16; }
// Word of row i (1-based) whose row-relative index is w (w = t/16 -
// base(i)/16), as an offset from the trace block.
IA_DEV size_t trace_word(int i, int w, int P, int G) {
    const int k = (i - 1) >> 6, ri = (i - 1) & 63;
    const int g = w + ((k * P + ri) >> 4) - ((k * P) >> 4);
    return ((size_t)k * G + g) * 64 + ri;
}

// Fill the trace of the NW DP of an explicit plen x nlen matrix (FP64,
// row-major) and return the aligned pair count; the pairs are written
// (reversed) to al.
//
// Each lane owns two consecutive rows of a 64-row stripe; row r of lane l
// computes column j at step k*P + 2l + r + j - 1 for stripe k, with period
// P = max(nlen+1, 64).  Row 1 trails row 0 by one step inside the lane, lane
// l trails lane l-1 by two steps, and a lane moves on to its rows of the
// next stripe as soon as it finishes the current one (the top row of stripe
// k+1 reads the boundary row that lane 31 wrote for stripe k at least one
// step earlier, since P >= 64).  Cells outside the matrix are computed on
// clamped indices and never read by a valid one (a row's state is reset when
// it enters a stripe, its neighbours only read its in-range cells, and row
// 1's column-0 cell, which column 1 reads as its left neighbour, is replaced
// by the boundary +0), so the step has no per-cell branches.
#define IA_NW_ATTR __device__ __noinline__
template <bool GAPZ>
IA_NW_ATTR int nw_align_t(const double *smat, int plen, int nlen, double gap, double *bH, uint32_t *trace,
                          uint32_t *al) {
    const int lane = threadIdx.x & 31;
    const int P = max(nlen + 1, 64);
    const int G = trace_G(P);
    const int S = (plen + 63) >> 6;  // stripes
    for (int j = lane; j <= nlen; j += 32) bH[j] = 0.0;
    __syncwarp();
    int k = 0, j0 = 1 - 2 * lane;  // stripe and row-0 column of this lane
    int i0 = 2 * lane + 1;         // 1-based row of row 0
    double h0 = 0, h1 = 0, h0prev = 0, up0prev = 0;
    // direction bits enter at the top and move down 2 bits a step, so after
    // the word's 16th step the bits of its step t sit at 2*(t%16); a word
    // stored after m < 16 of its steps is shifted down by 32 - 2m
    uint32_t acc0 = 0, acc1 = 0;
    bool r0ok = false, r1ok = false;
    bool st31 = false;  // lane 31 writes the stripe's boundary row
    bool ld0 = false;   // lane 0 reads the previous stripe's boundary row
    // this lane's two rows in the current stripe's block: word g of them at
    // blk[g * 64 + 2 * lane], blk[g * 64 + 2 * lane + 1]; g0 = (k*P)/16.
    // Only lanes with a row inside the matrix store (a short window leaves
    // most of its stripe's lanes without one)
    uint2 *blk = reinterpret_cast<uint2 *>(trace) + lane;
    int g0 = 0;
    const int last_lane = ((plen - 1) & 63) >> 1;
    const int total_steps = (S - 1) * P + 2 * last_lane + 1 + nlen + 1;
#pragma unroll 1
    for (int step = 0; step < total_steps; step++) {
        double up0 = __shfl_up_sync(kFull, h1, 1);
        if (j0 > P) {  // next stripe (rare): flush the finished rows' last words
            const int w = (step - 1) >> 4;
            if (((step - 1) & 15) != 15 && r0ok) {  // else stored (and cleared) last step
                const int sh = 30 - 2 * ((step - 1) & 15);
                blk[(size_t)(w - g0) * 32] = make_uint2(acc0 >> sh, acc1 >> sh);
            }
            j0 -= P;
            k++;
            i0 += 64;
            blk = reinterpret_cast<uint2 *>(trace + (size_t)k * G * 64) + lane;
            g0 = (k * P) >> 4;
        }
        if (j0 == 1) {  // entering a stripe (rare): set up its two rows
            h0 = h1 = h0prev = up0prev = 0.0;
            acc0 = acc1 = 0;
            r0ok = k < S && i0 <= plen;
            r1ok = k < S && i0 + 1 <= plen;
            st31 = lane == 31 && k + 1 < S && r1ok;
            ld0 = k > 0 && r0ok;
        }
        if (lane == 0) up0 = (ld0 && (unsigned)(j0 - 1) < (unsigned)nlen) ? bH[j0] : 0.0;
        // 0-based columns; a cell outside the matrix (column < 1 or > nlen) is
        // computed on column nlen-1 and never read by a valid one
        const int jc = (int)min((unsigned)(j0 - 1), (unsigned)(nlen - 1));
        const int jc1 = (int)min((unsigned)(j0 - 2), (unsigned)(nlen - 1));
        const int a0 = min(i0, plen) - 1, a1 = min(i0 + 1, plen) - 1;
        uint32_t d0, d1;
        const double sc0 = smat[(size_t)a0 * nlen + jc], sc1 = smat[(size_t)a1 * nlen + jc1];
        const double n1 = nw_cell<GAPZ>(h0prev, sc1, h0, h1, gap, d1);
        const double n0 = nw_cell<GAPZ>(up0prev, sc0, up0, h0, gap, d0);
        acc0 = __funnelshift_r(acc0, d0, 2);
        acc1 = __funnelshift_r(acc1, d1, 2);
        if (st31 && (unsigned)(j0 - 2) < (unsigned)nlen) bH[j0 - 1] = n1;
        if ((step & 15) == 15) {  // uniform: the warp stores one 256-byte line
            if (r0ok) blk[(size_t)((step >> 4) - g0) * 32] = make_uint2(acc0, acc1);
            acc0 = acc1 = 0;
        }
        h0prev = hval<GAPZ>(h0);
        up0prev = hval<GAPZ>(up0);
        // on a stripe's first step row 1 sits on column 0: keep the boundary
        // H(i, 0) = +0 as its left neighbour for column 1
        h1 = j0 == 1 ? 0.0 : n1;
        h0 = n0;
        j0++;
    }
    if (((total_steps - 1) & 15) != 15 && r0ok) {  // flush the last rows' pending words
        const int sh = 30 - 2 * ((total_steps - 1) & 15);
        blk[(size_t)(((total_steps - 1) >> 4) - g0) * 32] = make_uint2(acc0 >> sh, acc1 >> sh);
    }
    __syncwarp();
    // traceback from (plen, nlen): diag emits a pair, up steps i, else j.
    // The walk only moves up and left.  A tile is 32 rows; lane l holds the
    // 4 trace words of row rb-l that end at the word of column jl (the
    // column when the tile was loaded), so a path crosses few tiles.
    int i = plen, j = nlen, cnt = 0, rb = -1, jl = 0;
    uint32_t t0 = 0, t1 = 0, t2 = 0, t3 = 0;
    while (i > 0 && j > 0) {
        const int bi = trace_base(i, P);
        const int wi = ((bi + j - 1) >> 4) - (bi >> 4);  // word of (i, j) in row i
        const int wl = ((bi + jl - 1) >> 4) - (bi >> 4);  // last word held for row i
        if (i > rb || i <= rb - 32 || wi < wl - 3) {
            rb = i;
            jl = j;
            const int r = rb - lane;
            if (r >= 1) {
                const int br = trace_base(r, P);
                const int wr = ((br + j - 1) >> 4) - (br >> 4);
                t3 = trace[trace_word(r, wr, P, G)];
                t2 = wr >= 1 ? trace[trace_word(r, wr - 1, P, G)] : 0u;
                t1 = wr >= 2 ? trace[trace_word(r, wr - 2, P, G)] : 0u;
                t0 = wr >= 3 ? trace[trace_word(r, wr - 3, P, G)] : 0u;
            }
        }
        const int wk = wi - (((bi + jl - 1) >> 4) - (bi >> 4)) + 3;  // 0..3 within the tile
        const uint32_t mine = wk == 3 ? t3 : wk == 2 ? t2 : wk == 1 ? t1 : t0;
        const uint32_t rw = __shfl_sync(kFull, mine, rb - i);
        const uint32_t dir = (rw >> (2 * ((bi + j - 1) & 15))) & 3u;
        if (dir == 0) {
            if (lane == 0) al[cnt] = ((uint32_t)(i - 1) << 16) | (uint32_t)(j - 1);
            cnt++;
            i--;
            j--;
        } else if (dir == 1) {
            i--;
        } else {
            j--;
        }
    }
    __syncwarp();
    return cnt;
}

// Kabsch on the aligned pairs + their compact TM (no d8)
// (indialign_c/align.h:106-124).
IA_DEV double aligned_kabsch(const Pts &x, const uint32_t *al, int na, double d0, double lnorm,
                             double *R, double *t, unsigned long long *ctr) {
    const int lane = threadIdx.x & 31;
    if (lane == 0) atomicAdd(ctr + CTR_CHAIN_RES, 2ull * (unsigned long long)na);
    Moments m;
    m.clear();
    for (int k = lane; k < na; k += 32) {
        int pi, ni;
        al_get(al, na, k, pi, ni);
        const double *p = x.P + 3 * pi, *q = x.Q + 3 * ni;
        m.add(p[0], p[1], p[2], q[0], q[1], q[2]);
    }
    m.warp_total();
    kabsch_from_moments(m, 3.0, R, t);
    const double inv = 1.0 / fmax(d0 * d0, 1e-12);
    double s = 0.0;
    for (int k = lane; k < na; k += 32) {
        int pi, ni;
        al_get(al, na, k, pi, ni);
        const double *p = x.P + 3 * pi, *q = x.Q + 3 * ni;
        s += tm_term(dist2(R, t, p[0], p[1], p[2], q[0], q[1], q[2]), inv);
    }
    return warp_sum(s) / fmax(lnorm, 1.0);
}

// alignment_detailed_search without fragments (indialign_c/align.h:15-50,
// use_frag = false): one all-pairs seed x 6 cutoffs x <= 8 iterations,
// d8-filtered score.  The all-pairs seed's Kabsch is the (R0,t0) just
// computed by aligned_kabsch.  Lane groups of 4 run the 6 cutoffs side by
// side; the first maximum in cutoff order wins.
IA_NW_ATTR double lite_detailed(const Pts &x, const uint32_t *al, int na, const double *R0,
                            const double *t0, const double *dcut, double d0, double sd8,
                            double lnorm, double *Ro, double *to, unsigned long long *ctr) {
    const int lane = threadIdx.x & 31, g = lane >> 2, sub = lane & 3;
    const bool grp = g < kDetC;
    const double cut = dcut[grp ? g : 0];
    const double cut2 = cut * cut;
    double R[9], t[3];
#pragma unroll
    for (int a = 0; a < 9; a++) R[a] = R0[a];
#pragma unroll
    for (int a = 0; a < 3; a++) t[a] = t0[a];
    bool running = grp;
    int prev = -1, iter = 0;
    while (__any_sync(kFull, running)) {
        Moments m;
        m.clear();
        int cnt = 0;
        if (running) {
            for (int k = sub; k < na; k += 4) {
                int pi, ni;
                al_get(al, na, k, pi, ni);
                const double *p = x.P + 3 * pi, *q = x.Q + 3 * ni;
                if (dist2(R, t, p[0], p[1], p[2], q[0], q[1], q[2]) <= cut2) {
                    m.add(p[0], p[1], p[2], q[0], q[1], q[2]);
                    cnt++;
                }
            }
        }
        m.group_sum(4);
        cnt += __shfl_xor_sync(kFull, cnt, 1);
        cnt += __shfl_xor_sync(kFull, cnt, 2);
        if (running) {
            if (cnt >= 3) kabsch_from_moments(m, 3.0, R, t);
            ++iter;
            if (cnt == prev || iter >= 8) running = false;
            prev = cnt;
        }
    }
    // residue visits: each active group ran `iter` passes + 1 score pass
    if (sub == 0 && grp) atomicAdd(ctr + CTR_CHAIN_RES, (unsigned long long)(iter + 1) * na);
    const double inv = 1.0 / fmax(d0 * d0, 1e-12), sd8sq = sd8 * sd8;
    double s = 0.0;
    if (grp) {
        for (int k = sub; k < na; k += 4) {
            int pi, ni;
            al_get(al, na, k, pi, ni);
            const double *p = x.P + 3 * pi, *q = x.Q + 3 * ni;
            double d2 = dist2(R, t, p[0], p[1], p[2], q[0], q[1], q[2]);
            if (d2 <= sd8sq) s += tm_term(d2, inv);
        }
    }
    s += __shfl_xor_sync(kFull, s, 1);
    s += __shfl_xor_sync(kFull, s, 2);
    const double score = s / fmax(lnorm, 1.0);
    // first max over cutoffs 0..5 (strict >, initial -1e30)
    double bs = kScoreInit;
    int bg = 0;
    for (int c = 0; c < kDetC; c++) {
        double sc = __shfl_sync(kFull, score, 4 * c);
        if (sc > bs) { bs = sc; bg = c; }
    }
#pragma unroll
    for (int a = 0; a < 9; a++) Ro[a] = __shfl_sync(kFull, R[a], 4 * bg);
#pragma unroll
    for (int a = 0; a < 3; a++) to[a] = __shfl_sync(kFull, t[a], 4 * bg);
    return bs;
}

// ---- the chain kernel ----------------------------------------------------
constexpr int kManyChains = 16;  // chains per warp from which an SM's CTAs start together

struct ChainCtl {
    int task;   // the task in hand, -1: none left
    int slot;   // of next_task
    int chain;  // one chain per CTA: its index in the task
    int na;     // one chain per CTA: aligned pairs of the last alignment
};

// Element `lane` of a result record {score, R[9], t[3]} by unrolled selects
// (a dynamic index into R or t would move them to local memory).
IA_DEV double rec_elem(int lane, double score, const double *R, const double *t) {
    double v = score;
#pragma unroll
    for (int a = 0; a < 9; a++) v = lane == 1 + a ? R[a] : v;
#pragma unroll
    for (int a = 0; a < 3; a++) v = lane == 10 + a ? t[a] : v;
    return v;
}

// dst[0..11] = {R[9], t[3]} written by lanes 0..11 of the warp.
IA_DEV void put_rt(double *dst, const double *R, const double *t, int lane) {
    const double v = rec_elem(lane + 1, 0.0, R, t);
    if (lane < 12) dst[lane] = v;
}

// EMIT = false: LITE dp_refine chains only (the hot rescue kernel, DP score
// mode only); EMIT = true: single NW alignments for SS seeds / full dp_refine.
// Two instantiations keep the hot kernel's code small.
//
// A CTA stays with a task while it has chains, whose warps take them one at a
// time: it stages the pair's columns once and its warps wait for one another
// only when the task has run out and the CTA goes on to the next one with
// chains left.  (Eight chains per CTA and piece, with a barrier after each,
// kept the warps waiting for 13 % of their time: k_chain of a learned search
// of 1024 pairs of L 40-1000 80 -> 61 ms, of 64 pairs of L 30-1500 30 -> 22.6.)
// CTAs start spread over the tasks by their share of the cells (by chains, long
// pairs were left for the end: 48 pairs of L 30-1500 157.6 ms against 154.2
// with the same loop); in launches of many chains per warp the CTAs of an SM
// start together, so that their loops' code and their pair's points are shared
// (64 pairs of L 40-300: 52.7 ms against 58.1 spread singly), in smaller ones
// apart, so that the longest chains do not share an SM (64 pairs learned: 22.6
// against 26.7), and a launch of fewer chains than warps gives each CTA as many
// warps as chains fall to it.
//
// A launch of at most coop_max chains leaves most of the chip idle with a warp
// per chain, and its time is the longest chain's: then a CTA takes one chain
// at a time, its warps share the fill's stripes, and warp 0 does the rest.
// Measured, both with the fill of nw_fill.cuh against a warp per chain with
// the fill before it: one pair of L = 1203 261 -> 60 ms (its SS and dp_refine
// stages, one or two alignments at a time, 80 -> 18 ms), learned search of 64
// pairs of L 30-1500 285 -> 60 ms. The line lies at one chain per CTA slot of
// the chip: above it the slots are full either way.
//
// FAR: launches with a pair whose native points lie beyond kFar, whose fill
// compares with the cutoff (the same bits for all other pairs).  Kept out of the
// other launches' kernel, where a call for such pairs alone cost 1 to 2 %.
template <bool EMIT, bool FAR>
__global__ void __launch_bounds__(32 * kChainWarps, IA_CHAIN_MINB)
k_chain(DevBatch b, const ChainTask *__restrict__ tasks, const int *__restrict__ chain_begin,
        const float *__restrict__ work_begin, int ntasks, const ScanOut *__restrict__ scan, int *left, ChainScratch sc) {
    extern __shared__ __align__(16) char smem[];
    __shared__ ChainCtl ctl;
    __shared__ uint64_t bar;
    // per warp: the LITE chain's current (R, t) and its best (R, t), kept in
    // shared memory so that no transform stays live in registers across the
    // NW fill
    __shared__ double s_rt[kChainWarps][24];
    __shared__ int s_prog[kChainWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // shared layout: [native column pairs][pred labels][native labels]
    // (flag 1), then per warp the NW boundary row (flag 2), the alignment
    // (flag 4) and the NW trace block (flag 8, short pairs); the FP64 point
    // sets are read from global memory (L1)
    const int pmax = sc.pmax, nmax = sc.nmax, flags = sc.flags;
    const bool coord_smem = flags & 1, bh_smem = flags & 2, al_smem = flags & 4, tr_smem = flags & 8;
    const uint32_t qfloats = (uint32_t)fill_column_floats(nmax), qbytes = (qfloats * 4u + 15u) & ~15u;
    const uint32_t plb = ((uint32_t)pmax + 47u) & ~15u, nlb = ((uint32_t)nmax + 47u) & ~15u;
    char *sLp = smem + (coord_smem ? qbytes : 0), *sLn = sLp + (coord_smem ? plb : 0);
    char *wbase = sLn + (coord_smem ? nlb : 0);
    float *cols = (coord_smem ? reinterpret_cast<float *>(smem) : sc.gcol + (size_t)blockIdx.x * qfloats) + 6 * kFillPad;
    const uint32_t bh_floats = (uint32_t)fill_boundary_floats(nmax);
    const uint32_t al_bytes = ((uint32_t)min(pmax, nmax) * 4u + 15u) & ~15u;
    float *bh0 = (bh_smem ? reinterpret_cast<float *>(wbase) : sc.gbh + (size_t)blockIdx.x * kChainWarps * bh_floats) +
                 4 * kFillPad;  // the CTA's boundary rows
    char *albase = wbase + (bh_smem ? kChainWarps * bh_floats * 4 : 0);
    char *trbase = albase + (al_smem ? kChainWarps * al_bytes : 0);
    uint32_t phase = 0;
    const int total = scan->total_chunks;
    const bool coop = total <= sc.coop_max;
    const int pull = min(kChainWarps, (total + (int)gridDim.x - 1) / (int)gridDim.x);  // warps that take chains
    if (threadIdx.x == 0) {
        mbar_init(&bar);
        // the CTA's first task: the one that holds its share of the launch's
        // chains (one chain per CTA: the CTA's chain).  The share only says
        // where a CTA begins to look for chains
        ctl.task = -1;
        uint32_t place = blockIdx.x, places = gridDim.x;
        if (total >= kManyChains * kChainWarps * (int)gridDim.x) {
            asm("mov.u32 %0, %%smid;" : "=r"(place));
            asm("mov.u32 %0, %%nsmid;" : "=r"(places));
            place = min(place, places - 1);
        }
        if (!coop) {
            ctl.task = task_at(work_begin, ntasks, scan->work * (((float)place + 0.5f) / (float)places));
        } else if ((int)blockIdx.x < total) {
            ctl.task = task_at(chain_begin, ntasks, (int)blockIdx.x);
            ctl.chain = (int)blockIdx.x - chain_begin[ctl.task];
        }
    }
    __syncthreads();
    // this warp's buffers (one chain per CTA: the CTA's first)
    const int slot = coop ? 0 : warp, gw = blockIdx.x * kChainWarps + slot;
    uint32_t *al = al_smem ? reinterpret_cast<uint32_t *>(albase + slot * al_bytes)
                           : sc.gal + (size_t)gw * min(pmax, nmax);
    uint32_t *trace = tr_smem ? reinterpret_cast<uint32_t *>(trbase) + (size_t)slot * sc.trace_words
                              : sc.gtrace + (size_t)gw * sc.trace_words;
    double *rt = s_rt[slot];  // [current R, t][best R, t]
    const bool lead = !coop || warp == 0;  // does a chain's work beside the fill
    int staged = -1;
    FillArgs fa;
    fa.q = cols;
    fa.trace = trace;
    fa.bw = bh0 + (size_t)warp * bh_floats;
    fa.br = bh0 + (size_t)(coop ? (warp + kChainWarps - 1) % kChainWarps : warp) * bh_floats;
    fa.prog = s_prog;
    fa.err = b.err;
    for (;;) {
        const int ti = ctl.task;
        if (ti < 0) break;
        const ChainTask &T = tasks[ti];
        const PairInfo &I = b.info[T.pair];
        const int off = I.off, plen = I.plen, nlen = I.nlen;
        Pts x = {b.predc + 3 * (size_t)off, b.natc + 3 * (size_t)off};
        if (T.pair != staged) {
            const uint8_t *gLp = reinterpret_cast<const uint8_t *>(b.sspc + off);
            const uint8_t *gLn = reinterpret_cast<const uint8_t *>(b.ssnc + off);
            fa.plen = plen;
            fa.nlen = nlen;
            fa.P = x.P;
            fa.Lp = gLp;
            fa.Ln = gLn;
            if (coord_smem && EMIT) {
                Copy cp[2];
                char *dst[2] = {sLp, sLn};
                cp[0] = plan_copy(gLp, (uint32_t)plen);
                cp[1] = plan_copy(gLn, (uint32_t)nlen);
                stage_copies(cp, dst, 2, &bar, phase, b.err);
                fa.Lp = reinterpret_cast<const uint8_t *>(sLp + cp[0].lead);
                fa.Ln = reinterpret_cast<const uint8_t *>(sLn + cp[1].lead);
            }
            // (all tasks of a launch share their score mode)
            stage_columns(cols, x.Q, nlen, FAR || (EMIT && T.smode == SMAT_SS4), threadIdx.x, blockDim.x);
            __syncthreads();
            staged = T.pair;
        }
        // dp_refine_chunk / ss_nw_align need >= 3 valid residues on each side
        // (indialign_c/align.h:141, ss.h:58)
        const bool sized = plen >= 3 && nlen >= 3;
        const FillGeom geom = fill_geom(plen, nlen, coop ? kChainWarps : 1);
        if (T.smode == SMAT_SS4) {
            const double d01 = fmax(I.d0 + 1.5, I.d0s);
            fa.inv_d0sq = (float)(1.0 / (d01 * d01));
            fa.cut2 = 0.f;
        } else {
            const double d0dp = fmax(I.d0, 1.0);
            fa.inv_d0sq = (float)(1.0 / fmax(d0dp * d0dp, 1e-12));
            fa.cut2 = (float)(T.sd8 * T.sd8);
        }
        // one alignment from the transform fa.rt: fill by this warp or, one
        // chain per CTA, by all of them; then the traceback
        auto align = [&](double gap) {
            if (coop) {
                if (threadIdx.x < kChainWarps) s_prog[threadIdx.x] = 0;
                __syncthreads();
            }
            const long long c0 = clock64();
            const int w = coop ? warp : 0;
            fa.gap = (float)gap;
            if (!EMIT || T.smode == SMAT_DP) {
                nw_fill_r<FAR ? SMAT_DP_FAR : SMAT_DP>(fa, geom, w);
            } else if (T.smode == SMAT_SS4) {
                nw_fill_r<SMAT_SS4>(fa, geom, w);
            } else {
                nw_fill_r<SMAT_SS2>(fa, geom, w);
            }
            if (coop) __syncthreads();
            int na = 0;
            const long long c1 = clock64();
            if (lead) {
                na = nw_traceback(trace, geom, plen, nlen, al);
                if (lane == 0) {
                    if (coop) ctl.na = na;
                    atomicAdd(b.ctr + CTR_NW_CELLS, (unsigned long long)plen * (unsigned long long)nlen);
                    atomicAdd(b.ctr + CTR_CYC_NW, (unsigned long long)(c1 - c0));
                    atomicAdd(b.ctr + CTR_CYC_TRACE, (unsigned long long)(clock64() - c1));
                }
            }
            return na;
        };
        // warps take the task's chains one at a time
        for (;;) {
            int chain = ctl.chain;
            if (!coop) {
                if (warp >= pull) break;
                int rest = 0;
                if (lane == 0) rest = atomicSub(left + ti, 1);
                rest = __shfl_sync(kFull, rest, 0);
                if (rest <= 0) break;
                chain = T.n_chains - rest;
            }
            if (lead && lane == 0) atomicAdd(b.ctr + CTR_CHAINS, 1ull);
            const int gaps = T.gaps;
            const int si = chain / gaps, g = chain % gaps;
            const double gap = (gaps == 2 ? g : si) == 0 ? T.gap0 : T.gap1;
            bool live = !(T.live && !T.live[si]);
            if (T.start == START_WINDOW) {
                if (lead) {
                    int flen, ps, ns;
                    double R[9], t[3];
                    window_at(plen, nlen, T.dense, T.wlist ? T.wlist[si] : si, flen, ps, ns);
                    warp_kabsch_window(x, ps, ns, flen, R, t);
                    put_rt(rt, R, t, lane);
                }
            } else {
                const double *r = T.rt + (size_t)si * kRec;
                live = live && r[0] > -1e299;  // start flag: kNegInf = no start
                if (lead && lane < 12) rt[lane] = r[1 + lane];
            }
            __syncwarp();
            fa.rt = rt;
            if (EMIT) {
                // EMIT: one alignment; aligned coordinates, count and (for
                // SMAT_DP) the Kabsch on it with its compact score.
                int na = 0;
                if (live && sized) na = align(gap);
                if (lead) {
                    if (lane == 0) T.na_out[si] = na;
                    double *aP = T.alP + (size_t)si * T.al_cap * 3;
                    double *aQ = T.alQ + (size_t)si * T.al_cap * 3;
                    for (int k = lane; k < na && k < T.al_cap; k += 32) {
                        int pi, ni;
                        al_get(al, na, k, pi, ni);
#pragma unroll
                        for (int d = 0; d < 3; d++) {
                            aP[3 * k + d] = x.P[3 * pi + d];
                            aQ[3 * k + d] = x.Q[3 * ni + d];
                        }
                    }
                    if (T.smode == SMAT_DP && na >= 3) {
                        double nR[9], nt[3];
                        double s = aligned_kabsch(x, al, na, I.d0, I.lnorm, nR, nt, b.ctr);
                        double *o = T.res + (size_t)si * kRec;
                        const double v = rec_elem(lane, s, nR, nt);
                        if (lane < kRec) o[lane] = v;
                    }
                }
            } else {
                // LITE dp_refine chain (indialign_c/align.h:54-145,
                // d0_search_lite): best starts at score 0 / identity.
                double bs = 0.0;
                if (lead) {
                    double iR[9], it_[3];
                    set_identity(iR, it_);
                    put_rt(rt + 12, iR, it_, lane);
                }
                __syncwarp();
                for (int it = 0; live && sized && it < T.max_iter; it++) {
                    int na = align(gap);
                    if (coop) {
                        __syncthreads();
                        na = ctl.na;
                    }
                    if (na < 3) break;  // same transform -> same alignment next time
                    if (!lead) continue;
                    double nR[9], nt[3], dR[9], dt[3];
                    const long long ck0 = clock64();
                    double s = aligned_kabsch(x, al, na, I.d0, I.lnorm, nR, nt, b.ctr);
                    const long long ck1 = clock64();
                    double ds = lite_detailed(x, al, na, nR, nt, I.dcut, I.d0, T.sd8, I.lnorm, dR, dt, b.ctr);
                    if (lane == 0) {
                        atomicAdd(b.ctr + CTR_CYC_KABSCH, (unsigned long long)(ck1 - ck0));
                        atomicAdd(b.ctr + CTR_CYC_DETAIL, (unsigned long long)(clock64() - ck1));
                    }
                    if (ds > s) {
                        s = ds;
#pragma unroll
                        for (int a = 0; a < 9; a++) nR[a] = dR[a];
#pragma unroll
                        for (int a = 0; a < 3; a++) nt[a] = dt[a];
                    }
                    __syncwarp();  // every lane's NW reads of the current (R, t) are done
                    put_rt(rt, nR, nt, lane);
                    if (s > bs) {
                        bs = s;
                        put_rt(rt + 12, nR, nt, lane);
                    }
                    __syncwarp();
                }
                double *o = T.res + (size_t)chain * kRec;
                if (lead && lane < kRec) o[lane] = lane == 0 ? (live ? bs : kNegInf) : rt[12 + lane - 1];
                __syncwarp();  // the slot is reused by this warp's next chain
            }
            if (coop) break;
        }
        if (coop) break;
        next_task(left, &ctl.task, ntasks, &ctl.slot);
    }
}

// ---- NW on an explicit score matrix (one warp per problem) ---------------
// nw_dp + nw_traceback (indialign_c/nw.h:10-68) on a caller-given FP64 score
// matrix, bit for bit the reference's alignment on identical inputs.
__global__ void k_nw_explicit(const double *__restrict__ smat, int np, int nn, double gap,
                              uint32_t *trace, double *bH, uint32_t *al, int *ap, int *an,
                              int *na_out) {
    int na = 0;
    if (np >= 1 && nn >= 1) {
        if (gap == 0.0) na = nw_align_t<true>(smat, np, nn, gap, bH, trace, al);
        else na = nw_align_t<false>(smat, np, nn, gap, bH, trace, al);
    }
    for (int k = threadIdx.x; k < na; k += 32) {
        const uint32_t e = al[na - 1 - k];
        ap[k] = (int)(e >> 16);
        an[k] = (int)(e & 0xffffu);
    }
    if (threadIdx.x == 0) *na_out = na;
}

size_t nw_trace_words(int np, int nn) { return nw_trace_words_for(np, nn); }

void launch_nw_explicit(const double *smat, int np, int nn, double gap, uint32_t *trace,
                        double *bH, uint32_t *al, int *ap, int *an, int *na, cudaStream_t st) {
    k_nw_explicit<<<1, 32, 0, st>>>(smat, np, nn, gap, trace, bH, al, ap, an, na);
}

size_t chain_smem_bytes(int pmax, int nmax, int flags) {
    size_t s = 0;
    if (flags & 1) {
        s += (fill_column_floats(nmax) * 4 + 15) & ~size_t(15);
        s += (((size_t)pmax + 47) & ~size_t(15)) + (((size_t)nmax + 47) & ~size_t(15));
    }
    if (flags & 2) s += kChainWarps * fill_boundary_floats(nmax) * 4;
    if (flags & 4) s += kChainWarps * (((size_t)min(pmax, nmax) * 4 + 15) & ~size_t(15));
    if (flags & 8) s += kChainWarps * fill_trace_words(pmax, nmax) * 4;
    return s;
}

void launch_chain(const DevBatch &b, const ChainTask *tasks, const int *chain_begin, const float *work_begin,
                  int ntasks, const ScanOut *scan, int *left, const ChainScratch &sc, int grid, bool emit, bool far,
                  cudaStream_t st) {
    const size_t sm = chain_smem_bytes(sc.pmax, sc.nmax, sc.flags);
    const auto kernel = emit ? (far ? k_chain<true, true> : k_chain<true, false>)
                             : (far ? k_chain<false, true> : k_chain<false, false>);
    kernel<<<grid, 32 * kChainWarps, sm, st>>>(b, tasks, chain_begin, work_begin, ntasks, scan, left, sc);
}

const void *chain_kernel_ptr() { return (const void *)k_chain<false, false>; }

cudaError_t chain_set_attributes() {
    for (const auto kernel : {k_chain<false, false>, k_chain<true, false>, k_chain<false, true>, k_chain<true, true>}) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChainSmemMax);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace ia

namespace ia {

// One alignment by the search's fill and traceback (warps: 1 or kChainWarps).
__global__ void __launch_bounds__(32 * kChainWarps, IA_CHAIN_MINB)
k_nw_selftest(FillArgs fa, const double *Q, float *cols, int smode, int warps, uint32_t *al, int *na_out) {
    __shared__ int s_prog[kChainWarps];
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x < kChainWarps) s_prog[threadIdx.x] = 0;
    fa.q = cols + 6 * kFillPad;
    stage_columns(cols + 6 * kFillPad, Q, fa.nlen, smode == SMAT_SS4 || smode == SMAT_DP_FAR, threadIdx.x, blockDim.x);
    __syncthreads();
    const FillGeom g = fill_geom(fa.plen, fa.nlen, warps);
    const size_t row = fill_boundary_floats(fa.nlen);
    float *bnd = fa.bw + 4 * kFillPad;
    fa.prog = s_prog;
    fa.bw = bnd + warp * row;
    fa.br = bnd + (warps > 1 ? (warp + warps - 1) % warps : 0) * row;
    if (smode == SMAT_SS2) nw_fill_r<SMAT_SS2>(fa, g, warp);
    else if (smode == SMAT_SS4) nw_fill_r<SMAT_SS4>(fa, g, warp);
    else if (smode == SMAT_DP_FAR) nw_fill_r<SMAT_DP_FAR>(fa, g, warp);
    else nw_fill_r<SMAT_DP>(fa, g, warp);
    __syncthreads();
    if (warp == 0) {
        const int na = nw_traceback(fa.trace, g, fa.plen, fa.nlen, al);
        if (threadIdx.x == 0) *na_out = na;
    }
}

// Floats of [1, 2^126) whose reciprocal by rcp_pair differs from the correctly
// rounded one: whole, as the seed bank's score pass has it, and times a cutoff
// factor of 1, as the fill has it.
__global__ void k_rcp_f32_check(unsigned long long *bad) {
    unsigned long long n = 0;
    for (uint32_t u = 2 * (blockIdx.x * blockDim.x + threadIdx.x); u < (126u << 23); u += 2 * gridDim.x * blockDim.x) {
        const float2 x = make_float2(__uint_as_float(0x3f800000u + u), __uint_as_float(0x3f800001u + u));
        float2 y, e;
        rcp_pair(make_float2(-x.x, -x.y), y, e);
        const float2 r = __ffma2_rn(y, e, y), yk = __fmul2_rn(y, make_float2(1.f, 1.f)), s = __ffma2_rn(yk, e, yk);
        const float a = __frcp_rn(x.x), b = __frcp_rn(x.y);
        n += (r.x != a || s.x != a) + (r.y != b || s.y != b);
    }
    if (n) atomicAdd(bad, n);
}

}  // namespace ia

// Diagnostics (include/indialign_b200.h): one alignment of host points by the
// chains' fill; the FP32 reciprocal over its whole range.
extern "C" int indialign_selftest_nw(int plen, int nlen, const double *pred, const double *native, const double *rt,
                                     const uint8_t *lp, const uint8_t *ln, int smode, float gap, float inv_d0sq,
                                     float cut2, int warps, int *ap, int *an, int *na) {
    using namespace ia;
    if (plen < 1 || nlen < 1 || plen > 65535 || nlen > 65535 || !pred || !native || !rt || !lp || !ln || !ap || !an ||
        !na || (warps != 1 && warps != kChainWarps) || smode < 0 || smode > SMAT_SS4)
        return INDIALIGN_E_INPUT;
    for (int k = 0; k < nlen && smode == SMAT_DP; k++)
        if (is_far_point(native + 3 * (size_t)k)) smode = SMAT_DP_FAR;
    const size_t words = fill_trace_words(plen, nlen), row = fill_boundary_floats(nlen);
    const size_t sizes[9] = {24 * (size_t)plen, 24 * (size_t)nlen, 96, (size_t)plen, (size_t)nlen, 4 * words,
                             16 * row, 4 * fill_column_floats(nlen), 4 * (size_t)(plen < nlen ? plen : nlen) + 16};
    size_t at[10] = {0};
    for (int k = 0; k < 9; k++) at[k + 1] = at[k] + (sizes[k] + 255) / 256 * 256;
    char *d = nullptr;
    if (cudaMalloc(&d, at[9]) != cudaSuccess) return INDIALIGN_E_CUDA;
    const void *src[5] = {pred, native, rt, lp, ln};
    cudaError_t e = cudaMemset(d, 0, at[9]);
    for (int k = 0; k < 5 && e == cudaSuccess; k++) e = cudaMemcpy(d + at[k], src[k], sizes[k], cudaMemcpyHostToDevice);
    std::vector<uint32_t> al(plen < nlen ? plen : nlen);
    int out[2] = {0, 0};
    if (e == cudaSuccess) {
        FillArgs fa = {};
        fa.plen = plen;
        fa.nlen = nlen;
        fa.P = reinterpret_cast<const double *>(d + at[0]);
        fa.rt = reinterpret_cast<const double *>(d + at[2]);
        fa.Lp = reinterpret_cast<const uint8_t *>(d + at[3]);
        fa.Ln = reinterpret_cast<const uint8_t *>(d + at[4]);
        fa.gap = gap;
        fa.inv_d0sq = inv_d0sq;
        fa.cut2 = cut2;
        fa.trace = reinterpret_cast<uint32_t *>(d + at[5]);
        fa.bw = reinterpret_cast<float *>(d + at[6]);
        uint32_t *dal = reinterpret_cast<uint32_t *>(d + at[8]);
        int *dna = reinterpret_cast<int *>(d + at[9] - 16);
        fa.err = dna + 1;
        k_nw_selftest<<<1, 32 * warps>>>(fa, reinterpret_cast<const double *>(d + at[1]),
                                         reinterpret_cast<float *>(d + at[7]), smode, warps, dal, dna);
        e = cudaMemcpy(out, dna, sizeof out, cudaMemcpyDeviceToHost);
        if (e == cudaSuccess) e = cudaMemcpy(al.data(), dal, al.size() * 4, cudaMemcpyDeviceToHost);
    }
    cudaFree(d);
    if (e != cudaSuccess) return INDIALIGN_E_CUDA;
    if (out[1]) return INDIALIGN_E_DEVICE;
    *na = out[0];
    for (int k = 0; k < out[0]; k++) {
        const uint32_t v = al[out[0] - 1 - k];
        ap[k] = (int)(v >> 16);
        an[k] = (int)(v & 0xffffu);
    }
    return INDIALIGN_OK;
}

extern "C" int indialign_selftest_rcp_f32(unsigned long long *mismatches) {
    unsigned long long *d = nullptr;
    if (!mismatches || cudaMalloc(&d, 8) != cudaSuccess) return INDIALIGN_E_CUDA;
    cudaMemset(d, 0, 8);
    ia::k_rcp_f32_check<<<1184, 256>>>(d);
    const cudaError_t e = cudaMemcpy(mismatches, d, 8, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? INDIALIGN_OK : INDIALIGN_E_CUDA;
}
