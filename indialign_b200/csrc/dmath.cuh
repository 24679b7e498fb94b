// FP64 device math shared by every kernel of the search: the d0 schedule,
// the Horn-quaternion Kabsch solve, rigid transforms and TM terms.  The
// eigen-solve finds the dominant eigenvector from the characteristic
// polynomial (see qcp_rotation), which returns the reference Jacobi's
// rotation to rounding whenever the top eigenvalue is separated, and runs
// the reference's own Jacobi sequence (indialign_c/core.h:29-90) when it is
// not; covariances are formed from raw
// moments accumulated in one pass (sum p, sum q, sum p q^T, count) instead of
// the reference's centroid pass + centred pass (core.h:94-123), which is the
// same matrix up to FP64 rounding and lets a selection pass and its Kabsch
// fuse into a single sweep over the residues.
#pragma once
#include <stdint.h>

#define IA_DEV __device__ __forceinline__

namespace ia {

__constant__ static const double kD0Mults[6] = {2.0, 1.5, 1.0, 0.75, 0.5, 0.25};

// d0, d0_search and score_d8 from the normalisation length
// (indialign_c/core.h:12-25).
IA_DEV void d0_from_length(double L, double &d0, double &d0s, double &sd8) {
    double Lc = L > 1.0 ? L : 1.0;
    if (Lc <= 11.0) d0 = 0.3;
    else if (Lc <= 15.0) d0 = 0.4;
    else if (Lc <= 19.0) d0 = 0.5;
    else if (Lc <= 23.0) d0 = 0.6;
    else d0 = 0.7;
    if (Lc >= 30.0) d0 = 0.6 * sqrt(Lc - 0.5) - 2.5;
    if (d0 < 0.3) d0 = 0.3;
    double m = Lc - 15.0 > 0.0 ? Lc - 15.0 : 0.0;
    double v = 1.24 * cbrt(m) - 1.8;
    d0s = v < 4.5 ? 4.5 : (v > 8.0 ? 8.0 : v);
    sd8 = 1.5 * pow(Lc, 0.3) + 3.5;
}

// Cutoff list: d0s x {2,1.5,1,.75,.5,.25}, then d0+{1..5} unless within 0.01
// of an earlier entry (indialign_c/indialign.cpp:54-67).  Returns C <= 11.
IA_DEV int d0_candidates(double d0, double d0s, double *cand) {
    int C = 0;
    for (int c = 0; c < 6; c++) cand[C++] = d0s * kD0Mults[c];
    for (int c = 1; c <= 5; c++) {
        double v = d0 + (double)c;
        bool dup = false;
        for (int e = 0; e < C; e++) dup |= fabs(cand[e] - v) < 0.01;
        if (!dup) cand[C++] = v;
    }
    return C;
}

struct Rt {
    double R[9], t[3];
};

IA_DEV void set_identity(double *R, double *t) {
#pragma unroll
    for (int i = 0; i < 9; i++) R[i] = (i % 4 == 0) ? 1.0 : 0.0;
    t[0] = t[1] = t[2] = 0.0;
}

// aligned_d = sum_k p_k R[3k+d] + t_d (indialign_c/core.h:127-132)
IA_DEV void xform(const double *R, const double *t, double px, double py,
                  double pz, double &mx, double &my, double &mz) {
    mx = px * R[0] + py * R[3] + pz * R[6] + t[0];
    my = px * R[1] + py * R[4] + pz * R[7] + t[1];
    mz = px * R[2] + py * R[5] + pz * R[8] + t[2];
}

IA_DEV double dist2(const double *R, const double *t, double px, double py,
                    double pz, double qx, double qy, double qz) {
    double mx, my, mz;
    xform(R, t, px, py, pz, mx, my, mz);
    double dx = mx - qx, dy = my - qy, dz = mz - qz;
    return dx * dx + dy * dy + dz * dz;
}

// One Jacobi rotation of the pair (p,q), skipped when |A[p][q]| < 1e-15
// (indialign_c/core.h:39-58).  Indices are compile-time so A and V stay in
// registers.
template <int p, int q>
IA_DEV void jacobi_rot(double (&A)[4][4], double (&V)[4][4]) {
    double apq = A[p][q];
    if (fabs(apq) < 1e-15) return;
    double tau = (A[q][q] - A[p][p]) / (2.0 * apq);
    double t = (tau >= 0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
    double c = 1.0 / sqrt(1.0 + t * t), s = t * c;
    A[p][p] -= t * apq;
    A[q][q] += t * apq;
    A[p][q] = A[q][p] = 0.0;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        if (r == p || r == q) continue;
        double rp = A[r][p], rq = A[r][q];
        A[r][p] = A[p][r] = c * rp - s * rq;
        A[r][q] = A[q][r] = s * rp + c * rq;
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {
        double vp = V[r][p], vq = V[r][q];
        V[r][p] = c * vp - s * vq;
        V[r][q] = s * vp + c * vq;
    }
}

// Reciprocal by Newton-Raphson (y <- y + y(1 - xy), quadratic convergence)
// from the hardware's fast double approximation (rcp.approx.f64, about 20
// correct bits): two steps take the seed error below double rounding, so the
// result is within 1 ulp of 1/x (checked on the device against 1/x by the
// test suite).  Valid for normal |x| well inside the double range.
IA_DEV double rcp_nr(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double e = fma(-x, y, 1.0);
    y = fma(y, e, y);
    e = fma(-x, y, 1.0);
    return fma(y, e, y);
}

// One more step: the residual of a reciprocal within an ulp is exact, so the
// result rounds like 1 / x (Markstein 1990, "Computation of elementary functions
// on the IBM RISC System/6000 processor"), save for an x whose mantissa is all
// ones, where it may be an ulp off; 0 from 2^1022 on, where the approximation is
// flushed.  Both compared with 1 / x on the device by the test suite.  As long a
// dependent chain as the division operator (51 cycles against 46), but without
// its branch for special operands: with the operator in its place, 64 pairs of
// L 40-300 took 63.2 ms against 61.3, 24 collected pairs 26.3 against 25.5, one
// pair of 64 residues 1.43 against 1.41.
IA_DEV double rcp_cr(double x) {
    const double y = rcp_nr(x);
    return fma(fma(-x, y, 1.0), y, y);
}

// 1 / x for a pair of floats x of [1, 2^126), given -x: the hardware
// approximation y (within 1 ulp) and the residual e = 1 - x y; y + y e, fused,
// is then correctly rounded for every float of that range (compared with
// __frcp_rn over all of them by the test suite).
IA_DEV void rcp_pair(float2 neg_x, float2 &y, float2 &e) {
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(-neg_x.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(-neg_x.y));
    e = __ffma2_rn(neg_x, y, make_float2(1.f, 1.f));
}

// A residue's TM term 1 / (1 + d2 / d0^2) for inv = 1 / d0^2; 0 for an infinite
// distance, NaN for a NaN one.
IA_DEV double tm_term(double d2, double inv) {
    const double x = fma(d2, inv, 1.0);
    return x == INFINITY ? 0.0 : rcp_cr(x);
}

// a / b for y = 1 / b correctly rounded: Markstein's final step (a quotient
// near a / b, its residual, one fused correction), so six quotients by one
// divisor cost one division.  Compared with a / b on the device by the test
// suite: equal, save for a divisor whose mantissa is all ones (no count is),
// where one quotient in a thousand is an ulp off.  The bits matter: the covariance of exactly collinear points
// leaves the rotation about their line to the last bits of its entries.
IA_DEV double div_by(double a, double b, double y) {
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}

IA_DEV void horn_matrix(const double (&H)[3][3], double (&A)[4][4]) {
    A[0][0] = H[0][0] + H[1][1] + H[2][2];
    A[0][1] = A[1][0] = H[1][2] - H[2][1];
    A[0][2] = A[2][0] = H[2][0] - H[0][2];
    A[0][3] = A[3][0] = H[0][1] - H[1][0];
    A[1][1] = H[0][0] - H[1][1] - H[2][2];
    A[1][2] = A[2][1] = H[0][1] + H[1][0];
    A[1][3] = A[3][1] = H[2][0] + H[0][2];
    A[2][2] = -H[0][0] + H[1][1] - H[2][2];
    A[2][3] = A[3][2] = H[1][2] + H[2][1];
    A[3][3] = -H[0][0] - H[1][1] + H[2][2];
}

IA_DEV void set_eye4(double (&V)[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) V[i][j] = (i == j) ? 1.0 : 0.0;
}

// Dominant eigenvector (first index among equal diagonal maxima) -> unit
// quaternion -> rotation (indialign_c/core.h:76-89).
IA_DEV void quat_to_rotation(const double (&A)[4][4], const double (&V)[4][4], double *R) {
    int best = 0;
    double bv = A[0][0];
    if (A[1][1] > bv) { best = 1; bv = A[1][1]; }
    if (A[2][2] > bv) { best = 2; bv = A[2][2]; }
    if (A[3][3] > bv) { best = 3; bv = A[3][3]; }
    double q0, q1, q2, q3;
    q0 = best == 0 ? V[0][0] : best == 1 ? V[0][1] : best == 2 ? V[0][2] : V[0][3];
    q1 = best == 0 ? V[1][0] : best == 1 ? V[1][1] : best == 2 ? V[1][2] : V[1][3];
    q2 = best == 0 ? V[2][0] : best == 1 ? V[2][1] : best == 2 ? V[2][2] : V[2][3];
    q3 = best == 0 ? V[3][0] : best == 1 ? V[3][1] : best == 2 ? V[3][2] : V[3][3];
    double qn = sqrt(q0 * q0 + q1 * q1 + q2 * q2 + q3 * q3);
    if (qn < 1e-12) {
        q0 = 1; q1 = q2 = q3 = 0;
    } else {
        q0 /= qn; q1 /= qn; q2 /= qn; q3 /= qn;
    }
    R[0] = q0 * q0 + q1 * q1 - q2 * q2 - q3 * q3;
    R[1] = 2 * (q1 * q2 + q0 * q3);
    R[2] = 2 * (q1 * q3 - q0 * q2);
    R[3] = 2 * (q1 * q2 - q0 * q3);
    R[4] = q0 * q0 - q1 * q1 + q2 * q2 - q3 * q3;
    R[5] = 2 * (q2 * q3 + q0 * q1);
    R[6] = 2 * (q1 * q3 + q0 * q2);
    R[7] = 2 * (q2 * q3 - q0 * q1);
    R[8] = q0 * q0 - q1 * q1 - q2 * q2 + q3 * q3;
}

// The reference eigen-solve exactly: 8 cyclic sweeps in its pair order with
// correctly rounded divides and square roots (indialign_c/core.h:29-60).
IA_DEV void jacobi_reference(double (&A)[4][4], double (&V)[4][4]) {
    set_eye4(V);
#pragma unroll 1
    for (int sweep = 0; sweep < 8; sweep++) {
        jacobi_rot<0, 1>(A, V);
        jacobi_rot<0, 2>(A, V);
        jacobi_rot<0, 3>(A, V);
        jacobi_rot<1, 2>(A, V);
        jacobi_rot<1, 3>(A, V);
        jacobi_rot<2, 3>(A, V);
    }
}

// Dominant eigenvector of Horn's key matrix F of a covariance H by its
// characteristic polynomial -- the QCP method (Theobald 2005, "Rapid
// calculation of RMSDs using a quaternion-based characteristic polynomial").
// F is traceless, so P(x) = x^4 + c2 x^2 + c1 x + c0 with c2 = -2 |H|^2 (half
// of -tr(F^2)), c1 = -8 det H (a third of -tr(F^3)), c0 = det F.  The largest
// root l1 comes from Halley's method started at sqrt(3/4 tr(F^2)) >= l1 (four
// numbers of sum 0 and square sum s reach at most sqrt(3/4 s)); for a
// polynomial with real roots only, the iterates fall monotonically onto the
// largest root from above, with cubic convergence, so the loop ends once a step
// is below 1e-9 of the scale (3-5 iterations; Newton's method from
// sqrt(tr(F^2)) took 7-9).  P'(l1) is the product of the gaps to the
// other eigenvalues, each at most 2 sqrt(tr(F^2)); when it cannot prove
// l1 - l2 >= 1e-4 sqrt(tr(F^2)), l2 is found by Newton's method on P(x)/(x - l1).
// A top pair closer than that returns false, as does a scale whose sixth power
// would leave the double range: the eigenvector inside a (near-)degenerate pair
// depends on the solver, and the caller reruns the reference's Jacobi sequence.
// Otherwise the eigenvector is the column of adj(F - l1 I) with the largest
// diagonal entry: the adjugate of the symmetric matrix whole (14 two-by-two
// minors, 10 cofactors), so that lanes with different columns do not diverge,
// and the rotation's entries divided by |v|^2 once instead of normalising v.
// A CPU build of the oracle with a characteristic-polynomial solve matched the
// reference build's final scores to 3e-16 on 560 pairs, Jacobi rerunning in
// ~6e-5 of the solves.  The solve is a serial chain of FP64 operations; this
// form took k_bank's launches on one 64-residue pair from 0.75 to 0.68 ms and k_chain
// on 64 pairs of L 40-300 from 60.3 to 57.2 ms.
IA_DEV bool qcp_rotation(const double (&H)[3][3], double *R) {
    double n2 = 0.0;
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) n2 = fma(H[r][c], H[r][c], n2);
    const double p2 = 4.0 * n2;  // tr(F^2)
    if (!(p2 > 1e-80 && p2 < 1e80)) return false;
    const double a01 = H[1][2] - H[2][1], a02 = H[2][0] - H[0][2], a03 = H[0][1] - H[1][0];
    const double a12 = H[0][1] + H[1][0], a13 = H[2][0] + H[0][2], a23 = H[1][2] + H[2][1];
    double a00 = H[0][0] + H[1][1] + H[2][2], a11 = H[0][0] - H[1][1] - H[2][2];
    double a22 = -H[0][0] + H[1][1] - H[2][2], a33 = -H[0][0] - H[1][1] + H[2][2];
    const double detH = H[0][0] * (H[1][1] * H[2][2] - H[1][2] * H[2][1]) -
                        H[0][1] * (H[1][0] * H[2][2] - H[1][2] * H[2][0]) +
                        H[0][2] * (H[1][0] * H[2][1] - H[1][1] * H[2][0]);
    const double c2 = -2.0 * n2, c1 = -8.0 * detH;
    double c0;
    {
        const double b1 = a22 * a33 - a23 * a23, b2 = a12 * a33 - a13 * a23, b3 = a12 * a23 - a13 * a22;
        const double d1 = a11 * a33 - a13 * a13, d2 = a11 * a23 - a12 * a13, d3 = a11 * a22 - a12 * a12;
        c0 = a00 * (a11 * b1 - a12 * b2 + a13 * b3) - a01 * (a01 * b1 - a02 * b2 + a03 * b3) +
             a02 * (a01 * b2 - a02 * d1 + a03 * d2) - a03 * (a01 * b3 - a02 * d2 + a03 * d3);
    }
    // sqrt(p2) to a few parts in 1e7: it starts the iteration, from just above
    // the bound, and scales the thresholds
    double scale;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(scale) : "d"(p2));
    scale *= p2;
    double l1 = 0.86603 * scale;
#pragma unroll 1
    for (int it = 0; it < 64; it++) {
        const double x2 = l1 * l1;
        const double g = fma(fma(x2 + c2, l1, c1), l1, c0);
        const double dg = fma(fma(4.0, x2, 2.0 * c2), l1, c1);
        const double hg = fma(6.0, x2, c2);  // P''/2
        if (!(dg > 0.0)) break;
        const double nx = l1 - g * dg * rcp_nr(fma(dg, dg, -g * hg));
        if (!(nx < l1)) break;
        const bool done = l1 - nx <= 1e-9 * scale;
        l1 = nx;
        if (done) break;
    }
    const double dp = fma(fma(4.0 * l1, l1, 2.0 * c2), l1, c1);  // P'(l1)
    if (!(dp >= 4e-4 * p2 * scale)) {
        // second eigenvalue: largest root of x^3 + l1 x^2 + (c2 + l1^2) x + (c1 + l1 c2 + l1^3)
        const double b2 = l1, b1 = fma(l1, l1, c2), b0 = fma(l1, b1, c1);
        double x = l1;
#pragma unroll 1
        for (int it = 0; it < 128; it++) {
            const double g = fma(fma(x + b2, x, b1), x, b0);
            const double dg = fma(fma(3.0, x, 2.0 * b2), x, b1);
            if (!(dg > 0.0)) break;
            const double nx = x - g * rcp_nr(dg);
            if (!(nx < x)) break;
            const bool done = x - nx <= 1e-16 * scale;
            x = nx;
            if (done) break;
        }
        if (!(l1 - x >= 1e-4 * scale)) return false;
    }
    a00 -= l1;
    a11 -= l1;
    a22 -= l1;
    a33 -= l1;
    const double b1 = a22 * a33 - a23 * a23, b2 = a12 * a33 - a13 * a23, b3 = a12 * a23 - a13 * a22;
    const double d1 = a11 * a33 - a13 * a13, d2 = a11 * a23 - a12 * a13, d3 = a11 * a22 - a12 * a12;
    const double e1 = a02 * a33 - a03 * a23, e2 = a02 * a23 - a03 * a22, e3 = a02 * a13 - a12 * a03;
    const double f1 = a01 * a33 - a13 * a03, f2 = a01 * a13 - a11 * a03, f3 = a01 * a22 - a12 * a02;
    const double f4 = a01 * a12 - a11 * a02, f5 = a01 * a23 - a12 * a03;
    const double k00 = a11 * b1 - a12 * b2 + a13 * b3, k01 = -(a01 * b1 - a02 * b2 + a03 * b3);
    const double k02 = a01 * b2 - a02 * d1 + a03 * d2, k03 = -(a01 * b3 - a02 * d2 + a03 * d3);
    const double k11 = a00 * b1 - a02 * e1 + a03 * e2, k12 = -(a00 * b2 - a01 * e1 + a03 * e3);
    const double k13 = a00 * b3 - a01 * e2 + a02 * e3, k22 = a00 * d1 - a01 * f1 + a03 * f2;
    const double k23 = -(a00 * d2 - a01 * f5 + a02 * f2), k33 = a00 * d3 - a01 * f3 + a02 * f4;
    // adj(F - l1 I) = P'(l1) q q^T: its largest diagonal entry marks the best column
    double v0 = k00, v1 = k01, v2 = k02, v3 = k03, top = fabs(k00);
    if (fabs(k11) > top) { v0 = k01; v1 = k11; v2 = k12; v3 = k13; top = fabs(k11); }
    if (fabs(k22) > top) { v0 = k02; v1 = k12; v2 = k22; v3 = k23; top = fabs(k22); }
    if (fabs(k33) > top) { v0 = k03; v1 = k13; v2 = k23; v3 = k33; }
    const double vv = v0 * v0 + v1 * v1 + v2 * v2 + v3 * v3;
    if (!(vv > 0.0)) return false;
    const double inv = rcp_nr(vv), two = 2.0 * inv;
    R[0] = (v0 * v0 + v1 * v1 - v2 * v2 - v3 * v3) * inv;
    R[1] = two * (v1 * v2 + v0 * v3);
    R[2] = two * (v1 * v3 - v0 * v2);
    R[3] = two * (v1 * v2 - v0 * v3);
    R[4] = (v0 * v0 - v1 * v1 + v2 * v2 - v3 * v3) * inv;
    R[5] = two * (v2 * v3 + v0 * v1);
    R[6] = two * (v1 * v3 + v0 * v2);
    R[7] = two * (v2 * v3 - v0 * v1);
    R[8] = (v0 * v0 - v1 * v1 - v2 * v2 + v3 * v3) * inv;
    return true;
}

// Horn's 4x4 from the 3x3 covariance H -> dominant eigenvector -> rotation
// (indialign_c/core.h:64-90): the characteristic-polynomial solve above, or
// the reference's Jacobi sequence when the top eigenvalue is not separated
// (rare, and large: out of line).
static __device__ __noinline__ void jacobi_rotation(const double (&H)[3][3], double *R) {
    double A[4][4], V[4][4];
    horn_matrix(H, A);
    jacobi_reference(A, V);
    quat_to_rotation(A, V, R);
}
IA_DEV void cov_to_rotation(const double (&H)[3][3], double *R) {
    if (!qcp_rotation(H, R)) jacobi_rotation(H, R);
}

// Raw first and second moments of a selected point set.
struct Moments {
    double sp[3], sq[3], h[9], w;
    IA_DEV void clear() {
#pragma unroll
        for (int i = 0; i < 3; i++) sp[i] = sq[i] = 0.0;
#pragma unroll
        for (int i = 0; i < 9; i++) h[i] = 0.0;
        w = 0.0;
    }
    IA_DEV void add(double px, double py, double pz, double qx, double qy,
                    double qz) {
        sp[0] += px; sp[1] += py; sp[2] += pz;
        sq[0] += qx; sq[1] += qy; sq[2] += qz;
        h[0] += px * qx; h[1] += px * qy; h[2] += px * qz;
        h[3] += py * qx; h[4] += py * qy; h[5] += py * qz;
        h[6] += pz * qx; h[7] += pz * qy; h[8] += pz * qz;
        w += 1.0;
    }
    IA_DEV void add_w(double wi, double px, double py, double pz, double qx,
                      double qy, double qz) {
        double wx = wi * px, wy = wi * py, wz = wi * pz;
        sp[0] += wx; sp[1] += wy; sp[2] += wz;
        sq[0] += wi * qx; sq[1] += wi * qy; sq[2] += wi * qz;
        h[0] += wx * qx; h[1] += wx * qy; h[2] += wx * qz;
        h[3] += wy * qx; h[4] += wy * qy; h[5] += wy * qz;
        h[6] += wz * qx; h[7] += wz * qy; h[8] += wz * qz;
        w += wi;
    }
    // Sum over the 32 lanes, the total on every lane: exchanges that halve the
    // sums a lane carries, then one broadcast each, 34 exchanges instead of the
    // butterfly's 80 (and 16 additions instead of 80), in the butterfly's order
    // of additions.
    IA_DEV void warp_total() {
        const int lane = threadIdx.x & 31;
        double a[16];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            a[i] = sp[i];
            a[3 + i] = sq[i];
        }
#pragma unroll
        for (int i = 0; i < 9; i++) a[6 + i] = h[i];
        a[15] = w;
#pragma unroll
        for (int o = 1, k = 8; k > 0; o <<= 1, k >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < k; i++) {
                const double keep = up ? a[i + k] : a[i], send = up ? a[i] : a[i + k];
                a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        a[0] += __shfl_xor_sync(0xffffffffu, a[0], 16);
        // sum i stands on the lane whose low bits are i's four bits reversed
        auto get = [&](int i) {
            return __shfl_sync(0xffffffffu, a[0], (i >> 3 & 1) | (i >> 1 & 2) | (i << 1 & 4) | (i << 3 & 8));
        };
#pragma unroll
        for (int i = 0; i < 3; i++) {
            sp[i] = get(i);
            sq[i] = get(3 + i);
        }
#pragma unroll
        for (int i = 0; i < 9; i++) h[i] = get(6 + i);
        w = get(15);
    }
    // Butterfly sum over the lanes of `width` (power of two) so that every
    // lane of the group ends with the group total.
    IA_DEV void group_sum(int width) {
        for (int o = 1; o < width; o <<= 1) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
                sp[i] += __shfl_xor_sync(0xffffffffu, sp[i], o);
                sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], o);
            }
#pragma unroll
            for (int i = 0; i < 9; i++) h[i] += __shfl_xor_sync(0xffffffffu, h[i], o);
            w += __shfl_xor_sync(0xffffffffu, w, o);
        }
    }
};

// Kabsch from moments: identity when the weight is below `min_w`
// (3 points for the plain Kabsch, 1e-12 for the weighted one).
static __device__ __noinline__ void kabsch_from_moments(const Moments &m, double min_w, double *R,
                                                  double *t) {
    if (m.w < min_w) {
        set_identity(R, t);
        return;
    }
    double cP[3], cQ[3], H[3][3];
    const double inv_w = rcp_cr(m.w);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        cP[d] = div_by(m.sp[d], m.w, inv_w);
        cQ[d] = div_by(m.sq[d], m.w, inv_w);
    }
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) H[r][c] = m.h[r * 3 + c] - m.sp[r] * cQ[c];
    cov_to_rotation(H, R);
#pragma unroll
    for (int d = 0; d < 3; d++)
        t[d] = cQ[d] - (cP[0] * R[d] + cP[1] * R[3 + d] + cP[2] * R[6 + d]);
}

IA_DEV double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

IA_DEV int warp_sum_int(int v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Compact coordinate views of one pair (pred / native restricted to their
// valid residues), as used by the chain and ranker kernels.
struct Pts {
    const double *P;  // pred compact xyz
    const double *Q;  // native compact xyz
};

// Kabsch over pairs (P[a+i], Q[b+i]), i < cnt (a window), by the warp.
IA_DEV void warp_kabsch_window(const Pts &x, int a, int b, int cnt, double *R, double *t) {
    Moments m;
    m.clear();
    for (int i = threadIdx.x & 31; i < cnt; i += 32) {
        const double *p = x.P + 3 * (a + i), *q = x.Q + 3 * (b + i);
        m.add(p[0], p[1], p[2], q[0], q[1], q[2]);
    }
    m.warp_total();
    kabsch_from_moments(m, 3.0, R, t);
}

}  // namespace ia
