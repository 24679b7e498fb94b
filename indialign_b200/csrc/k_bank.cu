// Seed-bank kernel: iterative distance-cutoff Kabsch refinement of many
// (seed, cutoff) items over one point set, thread per item.
//
// Restates iterative_seed_refine / evaluate_seed_bank
// (indialign_c/search.h:28-138), refine_from_rt + gapless_threading_search
// (indialign_c/threading.h:15-80) and alignment_detailed_search
// (indialign_c/align.h:15-50).  All 32 lanes of a warp refine items of the
// same point set, so every residue load from shared memory is a broadcast;
// a lane's refinement is a sequential sum over residues in the reference's
// order.  Each item writes {score, R, t}; reduce_bank then applies the
// reference's serial first-max and early-termination rules.
//
// Precision: the residue visits -- transform, distance, inlier test, raw
// moment sums and the item's TM sum -- run in FP32 (the point set is staged
// as FP64, centred on its FP64 mean and converted to FP32 in shared memory;
// the TM sum is compensated; the operation order is fixed with explicit
// fused multiply-adds, as restated by the oracle's FP32 study build); each
// Kabsch eigen-solve runs in FP64 from the FP32 moments, and reduce_bank
// rescores the task's winning item in FP64, so every reported score is an
// FP64 TM-score of the returned (R, t).  The oracle rebuilt with this
// arithmetic in its seed banks stayed within 2e-8 of the reference build's
// final TM-scores on 560 pairs.
//
// k_bank is bound by the FMA pipe (62 % busy on the main bank of 61 pairs): a
// residue visit is 15 operations of distance, paired over two residues, and 15
// of sums.  The sums sit under one predicate per residue without a branch and
// the sweep takes four residue pairs at a time, so that distances of later
// residues fill the sums' latency: 167 -> 136 ms over the bank launches of a
// learned search of 1024 pairs of L 40-1000 (a branch around the sums 152,
// unrolled twice 150; eight times gained 1.5 % more in a third more code), and
// 129.6 with a vote that skips a pair no lane wants.
//
// A CTA stays with a task while it has items, whose warps take them as they
// become free.  (Chunks of 256 items with a barrier after each, for which every
// CTA staged the points again, kept the warps waiting for 13 % of their time:
// bank launches of 61 learned pairs 10.8 -> 9.5 ms, of one pair of 64 residues
// 0.65 -> 0.57, of the 1024 pairs 129.5 -> 126.)  CTAs start spread over the
// tasks by their work, items x residues, so that the tasks end together (spread
// by items alone, the banks of 64 learned pairs of L 30-1500 took 12.7 ms
// against 11.2), and a launch of few items gives each CTA as many warps as
// items fall to it.
#include "dmath.cuh"
#include "stage.cuh"
#include "pipeline.h"
#include "kernels.h"
#include "sched.cuh"

// build-time knob: minimum resident bank CTAs per SM (caps registers)
#ifndef IA_BANK_MINB
#define IA_BANK_MINB 4
#endif
// ... and the items per CTA up to which a launch is "few items"
#ifndef IA_BANK_WIDE
#define IA_BANK_WIDE 64
#endif


namespace ia {

// ---- the bank kernel -------------------------------------------------------
// A launch's units of work (kBankUnit items of a task).
struct BankWork {
    int *left;   // units left of the task in hand
    int *taken;  // units taken in the launch
    // Take up to `units` units; returns the first item, or -1.
    IA_DEV int take(const BankTask &T, int units) const {
        int rest = 0;
        if ((threadIdx.x & 31) == 0) {
            rest = atomicSub(left, units);
            if (rest > 0) atomicAdd(taken, min(units, rest));
        }
        rest = __shfl_sync(0xffffffffu, rest, 0);
        return rest <= 0 ? -1 : kBankUnit * ((T.n_items + kBankUnit - 1) / kBankUnit - rest);
    }
};

// Raw moments of the selected pairs in FP32 (counts exact).
struct MomentsF {
    float sp[3], sq[3], h[9];
    int w;
    IA_DEV void clear() {
#pragma unroll
        for (int i = 0; i < 3; i++) sp[i] = sq[i] = 0.f;
#pragma unroll
        for (int i = 0; i < 9; i++) h[i] = 0.f;
        w = 0;
    }
    IA_DEV void add(float px, float py, float pz, float qx, float qy, float qz) {
        sp[0] += px; sp[1] += py; sp[2] += pz;
        sq[0] += qx; sq[1] += qy; sq[2] += qz;
        h[0] = fmaf(px, qx, h[0]); h[1] = fmaf(px, qy, h[1]); h[2] = fmaf(px, qz, h[2]);
        h[3] = fmaf(py, qx, h[3]); h[4] = fmaf(py, qy, h[4]); h[5] = fmaf(py, qz, h[5]);
        h[6] = fmaf(pz, qx, h[6]); h[7] = fmaf(pz, qy, h[7]); h[8] = fmaf(pz, qz, h[8]);
        w++;
    }
    // add() if d2 <= lim, every instruction under the one predicate: no branch
    // around the sums, so the next residues' distances overlap them
    IA_DEV void add_if(float d2, float lim, float px, float py, float pz, float qx, float qy, float qz) {
        asm("{\n\t.reg .pred p;\n\t"
            "setp.le.f32 p, %16, %17;\n\t"
            "@p add.rn.f32 %0, %0, %18;\n\t@p add.rn.f32 %1, %1, %19;\n\t@p add.rn.f32 %2, %2, %20;\n\t"
            "@p add.rn.f32 %3, %3, %21;\n\t@p add.rn.f32 %4, %4, %22;\n\t@p add.rn.f32 %5, %5, %23;\n\t"
            "@p fma.rn.f32 %6, %18, %21, %6;\n\t@p fma.rn.f32 %7, %18, %22, %7;\n\t@p fma.rn.f32 %8, %18, %23, %8;\n\t"
            "@p fma.rn.f32 %9, %19, %21, %9;\n\t@p fma.rn.f32 %10, %19, %22, %10;\n\t"
            "@p fma.rn.f32 %11, %19, %23, %11;\n\t@p fma.rn.f32 %12, %20, %21, %12;\n\t"
            "@p fma.rn.f32 %13, %20, %22, %13;\n\t@p fma.rn.f32 %14, %20, %23, %14;\n\t"
            "@p add.s32 %15, %15, 1;\n\t}"
            : "+f"(sp[0]), "+f"(sp[1]), "+f"(sp[2]), "+f"(sq[0]), "+f"(sq[1]), "+f"(sq[2]), "+f"(h[0]), "+f"(h[1]),
              "+f"(h[2]), "+f"(h[3]), "+f"(h[4]), "+f"(h[5]), "+f"(h[6]), "+f"(h[7]), "+f"(h[8]), "+r"(w)
            : "f"(d2), "f"(lim), "f"(px), "f"(py), "f"(pz), "f"(qx), "f"(qy), "f"(qz));
    }
    // Kabsch in FP64 from these sums (identity below 3 pairs)
    IA_DEV void kabsch(double *R, double *t) const {
        Moments m;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            m.sp[i] = sp[i];
            m.sq[i] = sq[i];
        }
#pragma unroll
        for (int i = 0; i < 9; i++) m.h[i] = h[i];
        m.w = (double)w;
        kabsch_from_moments(m, 3.0, R, t);
    }
};

// The FP32 work runs on coordinates centred on their point set's FP64 mean
// (so the raw moments do not cancel against a large offset); the kernel's
// (R, t) live in that frame until an item is written out.  A point is a
// float4 (x, y, z, w) with w = 1 for a valid residue of the cutoff and score
// passes (V[i] != 0, or no mask) and 0 otherwise.
//
// The shared FP32 copy holds residues in pairs, so one paired FP32
// instruction (f32x2) serves two residues: pair k = residues 2k, 2k+1 is two
// float4 blocks {x_2k, x_2k+1, y_2k, y_2k+1} {z_2k, z_2k+1, w_2k, w_2k+1}; an
// odd set ends with a zero point of w = 0.
//
// Point i of a set in the centred FP32 frame: the converted shared copy, or
// converted on load from the FP64 global array (point sets too large for
// shared memory).  Both give the same floats, so a pair's results do not
// depend on which path its batch takes.
template <bool SMEM>
IA_DEV float4 point(const float4 *f, const double *d, const double *off, const uint8_t *V, int i) {
    if constexpr (SMEM) {
        const float *e = reinterpret_cast<const float *>(f) + (i >> 1) * 8 + (i & 1);
        return make_float4(e[0], e[2], e[4], e[6]);
    }
    else return make_float4((float)(d[3 * i] - off[0]), (float)(d[3 * i + 1] - off[1]),
                            (float)(d[3 * i + 2] - off[2]), (V == nullptr || V[i] != 0) ? 1.f : 0.f);
}

// Squared distance of p moved by (Rf, tf) from q, in a fixed FP32 operation
// order (the order the oracle's FP32 study build restates):
// d = ((t - q) + p_z R + p_y R) + p_x R per axis, d2 = (dx^2 + dy^2) + dz^2.
IA_DEV float dist2_f32(const float4 &p, const float4 &q, const float *Rf, const float *tf) {
    const float dx = fmaf(p.x, Rf[0], fmaf(p.y, Rf[3], fmaf(p.z, Rf[6], tf[0] - q.x)));
    const float dy = fmaf(p.x, Rf[1], fmaf(p.y, Rf[4], fmaf(p.z, Rf[7], tf[1] - q.y)));
    const float dz = fmaf(p.x, Rf[2], fmaf(p.y, Rf[5], fmaf(p.z, Rf[8], tf[2] - q.z)));
    return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

// A transform with every entry duplicated, the operand form of paired FP32
// instructions.
struct XformF2 {
    float2 r[9], t[3];
    IA_DEV void set(const double *R, const double *t_) {
#pragma unroll
        for (int a = 0; a < 9; a++) r[a] = make_float2((float)R[a], (float)R[a]);
#pragma unroll
        for (int a = 0; a < 3; a++) t[a] = make_float2((float)t_[a], (float)t_[a]);
    }
};

// dist2_f32 of the two residues of a staged pair (P blocks PA, PB; Q blocks
// QA, QB), element by element the same operations in the same order, two
// residues per paired instruction (t - q is the single rounding of
// q * (-1) + t).
IA_DEV float2 dist2_pair(const float4 &PA, const float4 &PB, const float4 &QA, const float4 &QB,
                         const XformF2 &X) {
    const float2 px = make_float2(PA.x, PA.y), py = make_float2(PA.z, PA.w), pz = make_float2(PB.x, PB.y);
    const float2 m1 = make_float2(-1.f, -1.f);
    float2 ax = __ffma2_rn(make_float2(QA.x, QA.y), m1, X.t[0]);
    float2 ay = __ffma2_rn(make_float2(QA.z, QA.w), m1, X.t[1]);
    float2 az = __ffma2_rn(make_float2(QB.x, QB.y), m1, X.t[2]);
    ax = __ffma2_rn(px, X.r[0], __ffma2_rn(py, X.r[3], __ffma2_rn(pz, X.r[6], ax)));
    ay = __ffma2_rn(px, X.r[1], __ffma2_rn(py, X.r[4], __ffma2_rn(pz, X.r[7], ay)));
    az = __ffma2_rn(px, X.r[2], __ffma2_rn(py, X.r[5], __ffma2_rn(pz, X.r[8], az)));
    return __ffma2_rn(az, az, __ffma2_rn(ay, ay, __fmul2_rn(ax, ax)));
}

// CTA-wide FP64 mean of the finite values of n points, per axis, into
// out[3] (shared); red holds 6 doubles per warp.  The summation order
// depends only on n, so both kernel paths get the same mean.  Non-finite
// coordinates are left out: the mean is only the frame the FP32 work runs
// in, and one Inf must not turn every centred point into NaN (the
// reference's FP64 seeds that avoid such a residue still score finitely).
// With all values finite this is the plain mean.
IA_DEV void points_mean(const double *src, int n, double *out, double *red) {
    double a[3] = {0.0, 0.0, 0.0}, c[3] = {0.0, 0.0, 0.0};
    for (int i = threadIdx.x; i < n; i += kBankChunk) {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const double x = src[3 * i + d];
            if (isfinite(x)) {
                a[d] += x;
                c[d] += 1.0;
            }
        }
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
        a[d] = warp_sum(a[d]);
        c[d] = warp_sum(c[d]);
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            red[6 * w + d] = a[d];
            red[6 * w + 3 + d] = c[d];
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double v = 0.0, m = 0.0;
        for (int k = 0; k < kBankChunk / 32; k++) {
            v += red[6 * k + threadIdx.x];
            m += red[6 * k + 3 + threadIdx.x];
        }
        out[threadIdx.x] = m > 0.0 ? v / m : 0.0;
    }
    __syncthreads();
}

// CTA-wide in-place conversion of n staged FP64 points (at src, inside the
// region that starts at dst) to centred FP32 residue pairs at dst (layout
// above), w from the validity bytes V (null: all valid).  Round r reads
// points [128r, 128r+128) before any thread writes them; its writes end at
// byte 16*128(r+1) + 16, below the first byte (24*128(r+1)) that a later
// round reads; the pairs of n points take 32*ceil(n/2) <= 16n + 16 bytes,
// inside the 24n + 32 bytes of the staged region.  `out` (native points): a
// residue outside the mask, and the point after an odd set, become NaN, so
// that their distance is never within a cutoff.
IA_DEV void points_to_f32(const double *src, float4 *dst4, int n, const double *off, const uint8_t *V, bool out) {
    float *dst = reinterpret_cast<float *>(dst4);
    for (int base = 0; base < n; base += kBankChunk) {
        const int i = base + (int)threadIdx.x;
        double x = out ? NAN : 0.0, y = 0.0, z = 0.0;
        float w = 0.f;
        if (i < n && !(out && V != nullptr && V[i] == 0)) {
            x = src[3 * i] - off[0];
            y = src[3 * i + 1] - off[1];
            z = src[3 * i + 2] - off[2];
            w = (V == nullptr || V[i] != 0) ? 1.f : 0.f;
        }
        __syncthreads();
        if (i < n || (i == n && (n & 1))) {  // residue i, or the zero point after an odd set
            float *e = dst + (i >> 1) * 8 + (i & 1);
            e[0] = (float)x;
            e[2] = (float)y;
            e[4] = (float)z;
            e[6] = w;
        }
    }
    __syncthreads();
}

// Each seed's own Kabsch, the start of its items at every cutoff: CTA (task,
// block of 128 seeds), thread per seed, {R[9], t[3]} in the tasks' centred
// frame to seed_rt[item_base / kDetC + seed] (a task has at least kDetC items
// per seed, so the tasks' ranges are disjoint).  Solved here over the seed's
// own residues, once for all its cutoffs, instead of per (seed, cutoff) item in
// k_bank with a sweep over the whole set.  The sums run in residue order, so a
// long window is a serial chain: points staged as FP32 with the mask as a
// number, {x, y, z, 0 if valid} and {x, y, z, 0 if valid & 1}, keep it free of
// branches (SMEM; point sets too large for it are read from global memory).
template <bool SMEM>
__global__ void __launch_bounds__(kBankChunk) k_bank_seeds(const BankTask *__restrict__ tasks, double *__restrict__ seed_rt) {
    extern __shared__ __align__(16) char smem[];
    __shared__ double oP[3], oQ[3], red[6 * (kBankChunk / 32)];
    const BankTask &T = tasks[blockIdx.x];
    const int C = T.C > 0 ? T.C : 1, K = T.n_items / C, sk = blockIdx.y * kBankChunk + threadIdx.x, n = T.n;
    if ((int)(blockIdx.y * kBankChunk) >= K) return;
    points_mean(T.P, n, oP, red);
    points_mean(T.Q, n, oQ, red);
    const uint8_t *V = T.V;
    float4 *sP = reinterpret_cast<float4 *>(smem), *sQ = sP + n;
    auto load = [&](int i, float4 &p, float4 &q) {
        if (SMEM) {
            p = sP[i];
            q = sQ[i];
            return;
        }
        p = point<false>(nullptr, T.P, oP, nullptr, i);
        q = point<false>(nullptr, T.Q, oQ, nullptr, i);
        const int v = V ? V[i] : 1;
        p.w = v != 0 ? 0.f : 1.f;
        q.w = v & 1 ? 0.f : 1.f;
    };
    if (SMEM) {
        for (int i = threadIdx.x; i < n; i += kBankChunk) {
            const float4 p = point<false>(nullptr, T.P, oP, nullptr, i), q = point<false>(nullptr, T.Q, oQ, nullptr, i);
            const int v = V ? V[i] : 1;
            sP[i] = make_float4(p.x, p.y, p.z, v != 0 ? 0.f : 1.f);
            sQ[i] = make_float4(q.x, q.y, q.z, v & 1 ? 0.f : 1.f);
        }
        __syncthreads();
    }
    if (sk >= K) return;
    const int k = T.slist ? T.slist[sk] : sk;
    MomentsF m;
    m.clear();
    int s = 0, len = 0;
    if (T.mode == SEED_TABLE) {
        const int2 e = T.table[k];
        s = e.x;
        len = e.y;
    } else {
        arith_seed(n, T.ms, k, s, len);
    }
    float4 p, q;
    if (s < 0) {  // bitmask seed: its bit and 1 & valid
        const uint32_t *row = T.bits + (size_t)(-1 - s) * T.words;
        for (int w = 0; w < T.words; w++)
            for (uint32_t x = row[w]; x; x &= x - 1) {
                const int i = w * 32 + __ffs(x) - 1;
                if (i >= n) break;
                load(i, p, q);
                m.add_if(q.w, 0.f, p.x, p.y, p.z, q.x, q.y, q.z);
            }
    } else {  // window of the valid residues
        const int end = min(s + len, n);
#pragma unroll 4
        for (int i = s; i < end; i++) {
            load(i, p, q);
            m.add_if(p.w, 0.f, p.x, p.y, p.z, q.x, q.y, q.z);
        }
    }
    double R[9], t[3];
    m.kabsch(R, t);
    double *o = seed_rt + 12 * ((size_t)(T.item_base / kDetC) + sk);
#pragma unroll
    for (int a = 0; a < 9; a++) o[a] = R[a];
#pragma unroll
    for (int a = 0; a < 3; a++) o[9 + a] = t[a];
}

// CTA-wide in-place conversion like points_to_f32, to one float4 per residue:
// P {x, y, z, 1 if valid}, Q {x, y, z, 1} or NaN outside the mask (`out`); the
// set is padded to a multiple of four with points that no cutoff selects.
IA_DEV void points_to_f4(const double *src, float4 *dst, int n, const double *off, const uint8_t *V, bool out) {
    for (int base = 0; base < n; base += kBankChunk) {
        const int i = base + (int)threadIdx.x;
        float4 v = make_float4(out ? NAN : 0.f, 0.f, 0.f, out ? 1.f : 0.f);
        if (i < n && (V == nullptr || V[i] != 0 || !out)) {
            v.x = (float)(src[3 * i] - off[0]);
            v.y = (float)(src[3 * i + 1] - off[1]);
            v.z = (float)(src[3 * i + 2] - off[2]);
            v.w = out || V == nullptr || V[i] != 0 ? 1.f : 0.f;
        }
        __syncthreads();
        if (i < ((n + 3) & ~3)) dst[i] = v;
    }
    __syncthreads();
}

// A task's items by four lanes each, for launches of few items:
// there a thread per item leaves the chip idle and the launch takes as long as
// one thread's sweeps, 15 operations of distance and 15 of sums per residue in
// turn.  The sums are the outer product (px, py, pz, 1) x (qx, qy, qz, 1): lane
// a of an item holds its row a and adds four products per selected residue;
// the distances of four residues go one to a lane.  Every sum still runs in
// residue order (sp + p is fma(p, 1, sp)), so an item's numbers are the same
// bits as in the thread-per-item loop.  It issues 1.6 times the instructions
// per residue and item and solves 8 systems per warp instead of 32, so the line
// lies at 64 items per resident CTA (IA_BANK_WIDE): k_bank's launches on one
// pair of 64 residues 0.70 -> 0.65 ms, of 1203 residues 6.8 -> 5.0 (0.57 and 4.3
// since the CTAs stay with a task); with the line at 128, a learned search of
// 61 pairs lost 0.9 of 10.9 ms.
IA_DEV void wide_items(const BankTask &T, const float4 *P4, const float4 *Q4, const double *oP, const double *oQ,
                       const double *__restrict__ seed_rt, double *__restrict__ item_res, const BankWork &work,
                       unsigned long long *ctr) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31, a = lane & 3, g0 = lane & 28, n = T.n, C = T.C > 0 ? T.C : 1;
    const float *Pa = reinterpret_cast<const float *>(P4) + a;
    for (;;) {
        const int gi = work.take(T, 1);
        if (gi < 0) break;
        const int pi = gi + (lane >> 2);
        const bool active = pi < T.n_items;
        int sk = 0, ci = 0;
        if (active) {
            const int K = T.n_items / C;
            sk = T.cutoff_major ? pi % K : pi / C;
            ci = T.cutoff_major ? pi / K : pi % C;
        }
        const double cut = T.cut[ci];
        const float cut2 = (float)(cut * cut);
        double R[9], t[3];
        const double *o = seed_rt + 12 * ((size_t)(T.item_base / kDetC) + sk);
#pragma unroll
        for (int k = 0; k < 9; k++) R[k] = o[k];
#pragma unroll
        for (int k = 0; k < 3; k++) t[k] = o[9 + k];
        float Rf[9], tf[3];
        auto round_rt = [&]() {
#pragma unroll
            for (int k = 0; k < 9; k++) Rf[k] = (float)R[k];
#pragma unroll
            for (int k = 0; k < 3; k++) tf[k] = (float)t[k];
        };
        bool running = active && T.max_iter > 0;
        int prev = -1, iter = 0;
        while (__any_sync(kFull, running)) {
            round_rt();
            const float lim = running ? cut2 : -1.f;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
            for (int base = 0; base < n; base += 4) {
                const unsigned in = __ballot_sync(kFull, dist2_f32(P4[base + a], Q4[base + a], Rf, tf) <= lim) >> g0;
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const float u = Pa[4 * (base + r)];
                    const float4 v = Q4[base + r];
                    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t@p fma.rn.f32 %0, %5, %6, %0;\n\t"
                        "@p fma.rn.f32 %1, %5, %7, %1;\n\t@p fma.rn.f32 %2, %5, %8, %2;\n\t"
                        "@p fma.rn.f32 %3, %5, %9, %3;\n\t}"
                        : "+f"(acc.x), "+f"(acc.y), "+f"(acc.z), "+f"(acc.w)
                        : "r"(in & (1u << r)), "f"(u), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w));
                }
            }
            MomentsF m;
#pragma unroll
            for (int r = 0; r < 3; r++) {
                m.h[3 * r] = __shfl_sync(kFull, acc.x, g0 + r);
                m.h[3 * r + 1] = __shfl_sync(kFull, acc.y, g0 + r);
                m.h[3 * r + 2] = __shfl_sync(kFull, acc.z, g0 + r);
                m.sp[r] = __shfl_sync(kFull, acc.w, g0 + r);
            }
            m.sq[0] = __shfl_sync(kFull, acc.x, g0 + 3);
            m.sq[1] = __shfl_sync(kFull, acc.y, g0 + 3);
            m.sq[2] = __shfl_sync(kFull, acc.z, g0 + 3);
            m.w = (int)__shfl_sync(kFull, acc.w, g0 + 3);
            if (running) {
                if (m.w >= 3) m.kabsch(R, t);
                ++iter;
                if (m.w == prev || iter >= T.max_iter) running = false;
                prev = m.w;
            }
        }
        // the compensated sum runs in residue order on every lane of the item,
        // over terms computed one to a lane
        round_rt();
        const float inv_d0sq = (float)(1.0 / fmax(T.d0 * T.d0, 1e-12)), sd8sq = (float)(T.sd8 * T.sd8);
        float sum = 0.f, comp = 0.f;
        for (int base = 0; base < n; base += 4) {
            const float4 p = P4[base + a];
            const float d2 = dist2_f32(p, Q4[base + a], Rf, tf);
            const unsigned in = __ballot_sync(kFull, p.w != 0.f && (!T.use_d8 || d2 <= sd8sq)) >> g0;
            const float term = __frcp_rn(fmaf(d2, inv_d0sq, 1.0f));
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float y = __shfl_sync(kFull, term, g0 + r) - comp, s2 = sum + y;
                if (in & (1u << r)) {
                    comp = (s2 - sum) - y;
                    sum = s2;
                }
            }
        }
        unsigned long long visits = active && a == 0 ? (unsigned long long)(iter + 1) * n : 0ull;
        unsigned long long items = active && a == 0 ? 1ull : 0ull;
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) {
            visits += __shfl_xor_sync(kFull, visits, k);
            items += __shfl_xor_sync(kFull, items, k);
        }
        if (lane == 0) {
            atomicAdd(ctr + CTR_BANK_RES, visits);
            atomicAdd(ctr + CTR_BANK_ITEMS, items);
        }
        if (active && a == 0) {
            double *rec = item_res + (size_t)(T.item_base + sk * C + ci) * kRec;
            rec[0] = (double)sum / fmax(T.lnorm, 1.0);
#pragma unroll
            for (int k = 0; k < 9; k++) rec[1 + k] = R[k];
#pragma unroll
            for (int k = 0; k < 3; k++)
                rec[10 + k] = t[k] + oQ[k] - (oP[0] * R[k] + oP[1] * R[3 + k] + oP[2] * R[6 + k]);
        }
    }
}

// CTAs go from task to task; their warps take a task's items 32 at a time (8 in
// a launch of at most wide_max items, see wide_items).
template <bool SMEM>
__global__ void __launch_bounds__(kBankChunk, IA_BANK_MINB)
k_bank(const BankTask *__restrict__ tasks, const float *__restrict__ work_begin,
       int ntasks, const ScanOut *__restrict__ scan, int *left, int *taken,
       const double *__restrict__ seed_rt, double *__restrict__ item_res, int *err, int nmax, int wide_max,
       unsigned long long *ctr) {
    extern __shared__ __align__(16) char smem[];
    __shared__ int s_task, s_slot;
    __shared__ uint64_t bar;
    __shared__ double oP[3], oQ[3], red[6 * (kBankChunk / 32)];  // point-set means
    // layout: P[nmax*3] Q[nmax*3] (each +16 B lead room), V, PV, NV bytes
    // room for a 15-byte lead and the rounded-up tail of a bulk copy
    const uint32_t coord_bytes = ((uint32_t)nmax * 24u + 47u) & ~15u;
    const uint32_t mask_bytes = ((uint32_t)nmax + 47u) & ~15u;
    char *sP = smem, *sQ = smem + coord_bytes, *sV = sQ + coord_bytes;
    char *sPV = sV + mask_bytes, *sNV = sPV + mask_bytes;
    uint32_t phase = 0;
    const int total = scan->total_chunks;
    if (total <= 0) return;
    const bool wide = SMEM && scan->items <= wide_max;
    const int units = wide ? 1 : 32 / kBankUnit;  // units a warp takes at a time
    // warps of a CTA that take items: in a launch of few, those that fall to it
    const int pull = min((int)blockDim.x / 32, (total / units + (int)gridDim.x) / (int)gridDim.x);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        mbar_init(&bar);
        s_task = first_task(work_begin, left, ntasks, scan->work, blockIdx.x, gridDim.x);
    }
    __syncthreads();
    const float4 *Pf = nullptr, *Qf = nullptr;  // shared FP32 copies (SMEM)
    const double *Pd = nullptr, *Qd = nullptr;  // global FP64 arrays (!SMEM)
    const uint8_t *V = nullptr, *PV = nullptr, *NV = nullptr;
    if (s_task < 0) next_task(left, &s_task, ntasks, &s_slot);
    for (;;) {
        const int ti = s_task;
        if (ti < 0) break;
        const BankTask &T = tasks[ti];
        const int n = T.n;
        {  // stage the task's points
            if (SMEM) {
                Copy cp[5];
                char *dst[5];
                int nc = 0;
                cp[nc] = plan_copy(T.P, (uint32_t)n * 24u); dst[nc++] = sP;
                cp[nc] = plan_copy(T.Q, (uint32_t)n * 24u); dst[nc++] = sQ;
                if (T.V) { cp[nc] = plan_copy(T.V, (uint32_t)n); dst[nc++] = sV; }
                if (T.PV) { cp[nc] = plan_copy(T.PV, (uint32_t)n); dst[nc++] = sPV; }
                if (T.NV) { cp[nc] = plan_copy(T.NV, (uint32_t)n); dst[nc++] = sNV; }
                stage_copies(cp, dst, nc, &bar, phase, err);
                const double *dP = reinterpret_cast<const double *>(sP + cp[0].lead);
                const double *dQ = reinterpret_cast<const double *>(sQ + cp[1].lead);
                points_mean(dP, n, oP, red);
                points_mean(dQ, n, oQ, red);
                int k = 2;
                V = T.V ? reinterpret_cast<const uint8_t *>(sV + cp[k++].lead) : nullptr;
                if (wide) {
                    points_to_f4(dP, reinterpret_cast<float4 *>(sP), n, oP, V, false);
                    points_to_f4(dQ, reinterpret_cast<float4 *>(sQ), n, oQ, V, true);
                } else {
                    points_to_f32(dP, reinterpret_cast<float4 *>(sP), n, oP, V, false);
                    points_to_f32(dQ, reinterpret_cast<float4 *>(sQ), n, oQ, V, true);
                }
                Pf = reinterpret_cast<const float4 *>(sP);
                Qf = reinterpret_cast<const float4 *>(sQ);
                PV = T.PV ? reinterpret_cast<const uint8_t *>(sPV + cp[k++].lead) : nullptr;
                NV = T.NV ? reinterpret_cast<const uint8_t *>(sNV + cp[k++].lead) : nullptr;
            } else {
                Pd = T.P; Qd = T.Q; V = T.V; PV = T.PV; NV = T.NV;
                points_mean(Pd, n, oP, red);
                points_mean(Qd, n, oQ, red);
            }
        }
        const BankWork work = {left + ti, taken};
        if (wide) {
            if constexpr (SMEM)
                if (warp < pull) wide_items(T, Pf, Qf, oP, oQ, seed_rt, item_res, work, ctr);
        }
        // the task's items go to the warps 32 at a time, so a warp whose items
        // converged early takes the next group
        while (!wide && warp < pull) {
        const int gi = work.take(T, units);
        if (gi < 0) break;
        const int pi = gi + lane;  // processing order within the task
        const bool active = pi < T.n_items;
        const int C = T.C > 0 ? T.C : 1;
        // item (seed sk, cutoff ci) and its record slot li = sk*C + ci: seed
        // major (the slot order), or cutoff major (a warp refines one cutoff
        // over 32 seeds; measured 1.38x faster than seed major on the
        // learned16384 step, because a warp iterates until its slowest item
        // converges and the iteration counts of one cutoff are far more alike
        // than those of one seed's cutoffs)
        int sk = 0, ci = 0;
        if (active) {
            if (T.cutoff_major) {
                const int K = T.n_items / C;
                sk = pi % K;
                ci = pi / K;
            } else {
                sk = pi / C;
                ci = pi % C;
            }
        }
        const int li = sk * C + ci;
        const double cut = T.cut[ci];
        const float cut2 = (float)(cut * cut);
        double R[9], t[3];
        MomentsF m;
        bool skip = false;
        if (T.mode == SEED_SHIFT) {
            const int o = offset_at(T.shift_lo, T.shift_stride, sk);
            m.clear();
            for (int i = max(0, o); i < min(n, n + o); i++) {
                const int j = i - o;
                if (active && PV[i] != 0 && NV[j] != 0) {
                    const float4 pp = point<SMEM>(Pf, Pd, oP, V, i), qq = point<false>(nullptr, T.Q, oQ, nullptr, j);
                    m.add(pp.x, pp.y, pp.z, qq.x, qq.y, qq.z);
                }
            }
            skip = m.w < T.shift_min;
            if (active && !skip) m.kabsch(R, t);
            else set_identity(R, t);
        } else {
            const double *o = seed_rt + 12 * ((size_t)(T.item_base / kDetC) + sk);
#pragma unroll
            for (int a = 0; a < 9; a++) R[a] = o[a];
#pragma unroll
            for (int a = 0; a < 3; a++) t[a] = o[9 + a];
        }
        // ---- cutoff iterations: select d2 <= cut^2, Kabsch, stop on a
        // repeated count ----
        bool running = active && !skip && T.max_iter > 0;
        int prev = -1, iter = 0;
        while (__any_sync(0xffffffffu, running)) {
            m.clear();
            const float lim = running ? cut2 : -1.f;
            if constexpr (SMEM) {
                // two residues per step: distances by paired instructions,
                // the accumulate per residue in residue order (a residue
                // outside the mask is staged with a NaN native point)
                XformF2 X;
                X.set(R, t);
                // distances of four pairs of residues side by side; the sums of
                // a pair are skipped when no lane's cutoff takes it (a learned
                // search of 1024 pairs: 134.9 -> 129.6 ms)
                constexpr int U = 4;
                const int pairs = (n + 1) >> 1;
                auto dist2 = [&](int k) { return dist2_pair(Pf[2 * k], Pf[2 * k + 1], Qf[2 * k], Qf[2 * k + 1], X); };
                auto add = [&](float2 d2, int k) {
                    const float4 PA = Pf[2 * k], PB = Pf[2 * k + 1], QA = Qf[2 * k], QB = Qf[2 * k + 1];
                    m.add_if(d2.x, lim, PA.x, PA.z, PB.x, QA.x, QA.z, QB.x);
                    m.add_if(d2.y, lim, PA.y, PA.w, PB.y, QA.y, QA.w, QB.y);
                };
                int k2 = 0;
#pragma unroll 1
                for (; k2 + U <= pairs; k2 += U) {
                    float2 d2[U];
#pragma unroll
                    for (int u = 0; u < U; u++) d2[u] = dist2(k2 + u);
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if (__any_sync(0xffffffffu, fminf(d2[u].x, d2[u].y) <= lim)) add(d2[u], k2 + u);
                }
#pragma unroll 1
                for (; k2 < pairs; k2++) add(dist2(k2), k2);
            } else {
                float Rf[9], tf[3];
#pragma unroll
                for (int a = 0; a < 9; a++) Rf[a] = (float)R[a];
#pragma unroll
                for (int a = 0; a < 3; a++) tf[a] = (float)t[a];
                for (int i = 0; i < n; i++) {
                    const float4 pp = point<SMEM>(Pf, Pd, oP, V, i), qq = point<SMEM>(Qf, Qd, oQ, nullptr, i);
                    if (pp.w != 0.f && dist2_f32(pp, qq, Rf, tf) <= lim) m.add(pp.x, pp.y, pp.z, qq.x, qq.y, qq.z);
                }
            }
            const int cnt = m.w;
            if (running) {
                if (cnt >= 3) m.kabsch(R, t);
                ++iter;
                if (cnt == prev || iter >= T.max_iter) running = false;
                prev = cnt;
            }
        }
        // ---- score: sum 1/(1+d2/d0^2) over the set (optionally d2 <= sd8^2)
        // divided by max(Lnorm, 1) (indialign_c/core.h:134-166), FP32 terms
        // with a compensated sum; reduce_bank rescores the winner in FP64 ----
        double score = kNegInf;
        if (active && !skip) {
            // term 1 / fma(d2, 1/d0^2, 1): a correctly rounded reciprocal of
            // one fused operation instead of two divisions
            const float inv_d0sq = (float)(1.0 / fmax(T.d0 * T.d0, 1e-12)), sd8sq = (float)(T.sd8 * T.sd8);
            float Rf[9], tf[3];
#pragma unroll
            for (int a = 0; a < 9; a++) Rf[a] = (float)R[a];
#pragma unroll
            for (int a = 0; a < 3; a++) tf[a] = (float)t[a];
            float sum = 0.f, comp = 0.f;
            const bool d8 = T.use_d8;
            auto add_term = [&](float d2, float term) {
                if (!d8 || d2 <= sd8sq) {
                    const float y = term - comp;
                    const float s2 = sum + y;
                    comp = (s2 - sum) - y;
                    sum = s2;
                }
            };
            if constexpr (SMEM) {
                XformF2 X;
                X.set(R, t);
                const float2 ninv = make_float2(-inv_d0sq, -inv_d0sq);
#pragma unroll 2
                for (int k2 = 0; k2 < (n + 1) >> 1; k2++) {
                    const float4 PA = Pf[2 * k2], PB = Pf[2 * k2 + 1], QA = Qf[2 * k2], QB = Qf[2 * k2 + 1];
                    const float2 d2 = dist2_pair(PA, PB, QA, QB, X);
                    // the correctly rounded reciprocals of a pair: approximation
                    // and one paired Newton step (rcp_pair), the division's own
                    // form only for huge and NaN distances (bank launches of
                    // 1024 learned pairs 125.7 -> 120.3 ms)
                    const float2 nden = __ffma2_rn(d2, ninv, make_float2(-1.f, -1.f));
                    float2 y, e2;
                    rcp_pair(nden, y, e2);
                    float2 r = __ffma2_rn(y, e2, y);
                    if (!(nden.x > -1e37f && nden.y > -1e37f)) r = make_float2(__frcp_rn(-nden.x), __frcp_rn(-nden.y));
                    if (PB.z != 0.f) add_term(d2.x, r.x);
                    if (PB.w != 0.f) add_term(d2.y, r.y);
                }
            } else {
                for (int i = 0; i < n; i++) {
                    const float4 pp = point<SMEM>(Pf, Pd, oP, V, i);
                    if (pp.w == 0.f) continue;
                    const float d2 = dist2_f32(pp, point<SMEM>(Qf, Qd, oQ, nullptr, i), Rf, tf);
                    add_term(d2, __frcp_rn(fmaf(d2, inv_d0sq, 1.0f)));
                }
            }
            score = (double)sum / fmax(T.lnorm, 1.0);
        }
        {
            // residue visits: `iter` cutoff passes + score pass (the seeds'
            // own windows, in k_bank_seeds or here, are not counted)
            unsigned long long visits = active && !skip ? (unsigned long long)(iter + 1) * n : 0ull;
            unsigned long long items = active ? 1ull : 0ull;
#pragma unroll
            for (int o2 = 16; o2 > 0; o2 >>= 1) {
                visits += __shfl_xor_sync(0xffffffffu, visits, o2);
                items += __shfl_xor_sync(0xffffffffu, items, o2);
            }
            if ((threadIdx.x & 31) == 0 && items) {
                atomicAdd(ctr + CTR_BANK_RES, visits);
                atomicAdd(ctr + CTR_BANK_ITEMS, items);
            }
        }
        if (active) {
            // back to the caller's frame: t = t_c + oQ - sum_k oP_k R[3k+d]
            double *o = item_res + (size_t)(T.item_base + li) * kRec;
            o[0] = score;
#pragma unroll
            for (int a = 0; a < 9; a++) o[1 + a] = R[a];
#pragma unroll
            for (int a = 0; a < 3; a++) o[10 + a] = t[a] + oQ[a] - (oP[0] * R[a] + oP[1] * R[3 + a] + oP[2] * R[6 + a]);
        }
        }  // next group of 32 items
        // all units taken: no task has any left
        if (__syncthreads_or(threadIdx.x == 0 && *(volatile int *)taken >= total)) break;
        next_task(left, &s_task, ntasks, &s_slot);
    }
}

// ---- first-max reduction of a task's items ---------------------------------
// Serial semantics of evaluate_seed_bank (indialign_c/search.h:62-98): seeds
// outer, cutoffs inner, a candidate replaces the best only if strictly
// greater, and before each seed the loop stops once best >= early_term.  The
// last seed processed is therefore k* = the first seed holding an item
// >= early_term; every earlier item is below early_term, so the result is the
// first maximum over the items of seeds 0..k*.
// `width` threads per task: a warp where tasks are many and short (threading
// offsets), else the CTA, whose loads over a long item list then overlap.
__global__ void __launch_bounds__(128) k_reduce_bank(const BankTask *__restrict__ tasks, int ntasks, int width,
                              const double *__restrict__ item_res,
                              PairState *__restrict__ state) {
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ double s_d[4];
    __shared__ int s_i[4], s_k[4];
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) / width;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, me = threadIdx.x % width;
    const bool cta = width > 32;  // w is then uniform over the CTA
    if (w >= ntasks) return;
    const BankTask &T = tasks[w];
    if (T.n_items <= 0) return;
    const int C = T.C > 0 ? T.C : 1;
    const double *base = item_res + (size_t)T.item_base * kRec;
    // first maximum of items [0, end) and the first seed holding an item >= early_term
    auto first_max = [&](int end, double &bs, int &bi, int &kst) {
        bs = kScoreInit;
        bi = -1;
        kst = 0x7fffffff;
#pragma unroll 4
        for (int i = me; i < end; i += width) {
            const double s = base[(size_t)i * kRec];
            if (s >= T.early_term) kst = min(kst, i / C);
            if (s > bs) { bs = s; bi = i; }  // thread-local: ascending i, strict >
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double s2 = __shfl_xor_sync(kFull, bs, o);
            const int i2 = __shfl_xor_sync(kFull, bi, o);
            kst = min(kst, __shfl_xor_sync(kFull, kst, o));
            if ((s2 > bs) || (s2 == bs && i2 >= 0 && (bi < 0 || i2 < bi))) { bs = s2; bi = i2; }
        }
        if (!cta) return;
        __syncthreads();
        if (lane == 0) {
            s_d[warp] = bs;
            s_i[warp] = bi;
            s_k[warp] = kst;
        }
        __syncthreads();
        for (int k = 0; k < 4; k++) {
            const double s2 = s_d[k];
            const int i2 = s_i[k];
            kst = min(kst, s_k[k]);
            if ((s2 > bs) || (s2 == bs && i2 >= 0 && (bi < 0 || i2 < bi))) { bs = s2; bi = i2; }
        }
    };
    double bs;
    int bi, kst;
    first_max(T.n_items, bs, bi, kst);
    if (T.early_term < 1e30 && kst != 0x7fffffff && (kst + 1) * C < T.n_items) first_max((kst + 1) * C, bs, bi, kst);
    // the winner's score in FP64 over the task's own point set (the items
    // were scored in FP32): the same formula as k_bank's score pass
    double score = kScoreInit;
    if (bi >= 0) {
        const double *rec = base + (size_t)bi * kRec;
        double R[9], t[3];
#pragma unroll
        for (int a = 0; a < 9; a++) R[a] = rec[1 + a];
#pragma unroll
        for (int a = 0; a < 3; a++) t[a] = rec[10 + a];
        const double inv = 1.0 / fmax(T.d0 * T.d0, 1e-12), sd8sq = T.sd8 * T.sd8;
        double sum = 0.0;
        for (int i = me; i < T.n; i += width) {
            if (T.V && T.V[i] == 0) continue;
            const double d2 = dist2(R, t, T.P[3 * i], T.P[3 * i + 1], T.P[3 * i + 2], T.Q[3 * i], T.Q[3 * i + 1],
                                    T.Q[3 * i + 2]);
            if (!T.use_d8 || d2 <= sd8sq) sum += tm_term(d2, inv);
        }
        sum = warp_sum(sum);
        if (cta) {
            __syncthreads();
            if (lane == 0) s_d[warp] = sum;
            __syncthreads();
            sum = (s_d[0] + s_d[1]) + (s_d[2] + s_d[3]);
        }
        score = sum / fmax(T.lnorm, 1.0);
    }
    double *out = T.out_rec >= 0 ? state[T.pair].rec[T.out_rec] : T.out;
    if (me < kRec) {
        double v;
        if (bi >= 0) v = me == 0 ? score : base[(size_t)bi * kRec + me];
        else v = me == 0 ? kScoreInit : ((me == 1 || me == 5 || me == 9) ? 1.0 : 0.0);
        out[me] = v;
    }
}

// ---- launch wrappers -------------------------------------------------------
size_t bank_smem_bytes(int nmax) {
    size_t coord = ((size_t)nmax * 24 + 47) & ~size_t(15);
    size_t mask = ((size_t)nmax + 47) & ~size_t(15);
    return 2 * coord + 3 * mask;
}

void launch_bank(const BankTask *tasks, const float *work_begin, int ntasks,
                 const ScanOut *scan, int *left, int *taken, double *seed_rt, int seed_blocks, double *item_res, int *err,
                 int nmax, int grid, unsigned long long *ctr, cudaStream_t st) {
    // offset items (no seeds) sum their starts in the thread-per-item form
    const int wide_max = seed_blocks > 0 ? IA_BANK_WIDE * grid : 0;
    if (seed_blocks > 0) {
        const size_t ss = (size_t)nmax * 2 * sizeof(float4);
        const dim3 g(ntasks, seed_blocks);
        if (ss <= kBankSmemMax) k_bank_seeds<true><<<g, kBankChunk, ss, st>>>(tasks, seed_rt);
        else k_bank_seeds<false><<<g, kBankChunk, 0, st>>>(tasks, seed_rt);
    }
    size_t sm = bank_smem_bytes(nmax);
    if (sm <= kBankSmemMax) {
        k_bank<true><<<grid, kBankChunk, sm, st>>>(tasks, work_begin, ntasks, scan, left, taken,
                                                   seed_rt, item_res, err, nmax, wide_max, ctr);
    } else {
        k_bank<false><<<grid, kBankChunk, 0, st>>>(tasks, work_begin, ntasks, scan, left, taken,
                                                   seed_rt, item_res, err, nmax, wide_max, ctr);
    }
}

void launch_reduce_bank(const BankTask *tasks, int ntasks, bool short_lists, const double *item_res,
                        PairState *state, cudaStream_t st) {
    if (ntasks <= 0) return;
    const int width = short_lists ? 32 : 128, per = 128 / width;
    k_reduce_bank<<<(ntasks + per - 1) / per, 128, 0, st>>>(tasks, ntasks, width, item_res, state);
}

const void *bank_kernel_ptr(bool smem) {
    return smem ? (const void *)k_bank<true> : (const void *)k_bank<false>;
}

cudaError_t bank_set_attributes() {
    cudaError_t e = cudaFuncSetAttribute(k_bank<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kBankSmemMax);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_bank_seeds<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBankSmemMax);
    return e;
}

}  // namespace ia
