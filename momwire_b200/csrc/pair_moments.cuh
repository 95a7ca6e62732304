// Segment-pair moments and their Galerkin contraction (FP64, sm_100a): the
// arithmetic of the impedance fill (fill.cu), whose phase series and reciprocal
// root the off-edge block sampler (offedge_block.cu) uses too.
//
// A pair's (d+1)^2 moments J[p][P] = sum_qr w_q u_q^p  G(R_qr)  w_r u_r^P are
// computed by ONE thread.  What bounds it is the FP64 pipe (64 lanes a clock
// per SM), so the samples are stripped to what differs between them:
//   * the phase of the first node pair, exp(-j k R_00) / (4 pi), multiplies
//     the finished moments; a sample only needs exp(-j k (R - R_00)), whose
//     argument is at most |k| (h_i + h_j), from a Taylor series as long as that
//     bound asks for (a warp-uniform choice);
//   * one reciprocal square root, without special cases, serves R and 1 / R.
// That is 36 FP64 operations a sample instead of about 62, and no shuffles
// (four lanes a pair, each with a full sine and cosine, and a shuffle
// reduction of all 18 sums took 1.8 times as long).  A thread per observer
// node, its sums contracted later, needs fewer registers but more shared
// memory, and measured slower: 13.1 against 7.6 ms on the 16 x 16 array.
//
// The contraction Z = sum_ab C_m,a . J_ab . C_n,b runs in two stages through
// shared memory: source side first (segment x basis), then observer side
// (basis x basis), a third of the operations and half of the shared-memory
// reads of contracting every basis pair on its own.
#pragma once

#include "common.cuh"
#include "ground_weights.cuh"

namespace mw {

// Staged segment: nq nodes of six doubles -- position, then the folded
// weights w L u^p -- then tangent, centre, squared radius, length.  Nodes are
// read as 16-byte pieces; the stride is twice an odd number of doubles, so
// lanes that read different segments fall on different banks.
constexpr int kNodeDoubles = 6;
template <int D>
__host__ __device__ constexpr int seg_stride(int nq) {
    const int half = (nq * kNodeDoubles + 8) / 2;
    return 2 * (half | 1);
}

// Node q of a segment; the call for node 0 also writes the tail.
template <int D>
__device__ __forceinline__ void stage_node(double* dst, int nq, int q, const double* gt, const double* gw,
                                           const double* sl, const double* sr, const double* tg, double a,
                                           bool mirror, double gz) {
    constexpr int NM = D + 1;
    const double l0 = sl[0], l1 = sl[1], l2 = sl[2];
    const double r0 = sr[0], r1 = sr[1], r2 = sr[2];
    const double dx = r0 - l0, dy = r1 - l1, dz = r2 - l2;
    const double L = sqrt(dx * dx + dy * dy + dz * dz);
    const double t = gt[q];
    const double pz = (1.0 - t) * l2 + t * r2;
    double* node = dst + q * kNodeDoubles;
    node[0] = (1.0 - t) * l0 + t * r0;
    node[1] = (1.0 - t) * l1 + t * r1;
    node[2] = mirror ? 2.0 * gz - pz : pz;
    const double u = t * L;
    double wp = gw[q] * L;
#pragma unroll
    for (int p = 0; p < NM; ++p) {
        node[3 + p] = wp;
        wp *= u;
    }
    if (q != 0) return;
    double* o = dst + nq * kNodeDoubles;
    o[0] = tg[0];
    o[1] = tg[1];
    o[2] = mirror ? -tg[2] : tg[2];
    const double cz = 0.5 * (l2 + r2);
    o[3] = 0.5 * (l0 + r0);
    o[4] = 0.5 * (l1 + r1);
    o[5] = mirror ? 2.0 * gz - cz : cz;
    o[6] = a * a;
    o[7] = L;
}
template <int D>
__device__ __forceinline__ const double* seg_tail(const double* s, int nq) {
    return s + nq * kNodeDoubles;
}

// sin x and cos x for |x| <= kPhaseShort / kPhaseLong from their Taylor
// series (Horner in x^2; coefficients 1/n!), and beyond from sincos.  First
// omitted terms: x^13/13! and x^14/14! at 0.3, x^19/19! and x^18/18! at 0.75
// -- below 3e-17 and 1e-18.
constexpr double kPhaseShort = 0.3, kPhaseLong = 0.75;
enum { kPhaseModeShort = 0, kPhaseModeLong = 1, kPhaseModeAny = 2 };

template <int MODE>
__device__ __forceinline__ void phase_step(double x, double* sx, double* cx) {
    if (MODE == kPhaseModeAny && fabs(x) > kPhaseLong) {
        sincos(x, sx, cx);
        return;
    }
    const double t = x * x;
    double c, s;
    if (MODE == kPhaseModeShort) {
        c = 1.0 / 479001600.0;  // 1/12!
        s = -1.0 / 39916800.0;  // 1/11!
    } else {
        c = 1.0 / 20922789888000.0;  // 1/16!
        c = fma(c, t, -1.0 / 87178291200.0);
        c = fma(c, t, 1.0 / 479001600.0);
        s = 1.0 / 355687428096000.0;  // 1/17!
        s = fma(s, t, -1.0 / 1307674368000.0);
        s = fma(s, t, 1.0 / 6227020800.0);
        s = fma(s, t, -1.0 / 39916800.0);
    }
    c = fma(c, t, -1.0 / 3628800.0);
    c = fma(c, t, 1.0 / 40320.0);
    c = fma(c, t, -1.0 / 720.0);
    c = fma(c, t, 1.0 / 24.0);
    c = fma(c, t, -0.5);
    *cx = fma(c, t, 1.0);
    s = fma(s, t, 1.0 / 362880.0);
    s = fma(s, t, -1.0 / 5040.0);
    s = fma(s, t, 1.0 / 120.0);
    s = fma(s, t, -1.0 / 6.0);
    *sx = fma(s * t, x, x);
}

// 1 / sqrt(x), x > 0 and normal: the hardware's approximation (about 20 bits)
// and one step of Halley's iteration, y (1 + e/2 + 3 e^2/8) with e = 1 - x y^2,
// which triples them.  No special cases, no branch.
__device__ __forceinline__ double rsqrt_pos(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y * y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// sqrt(x) from y = rsqrt_pos(x): x y and one step of Newton's iteration on its
// residual, which is exact, so that the result is rounded (almost always) once.
__device__ __forceinline__ double sqrt_pos(double x, double y) {
    const double r = x * y;
    return fma(0.5 * y, fma(-r, r, x), r);
}

struct Node {
    double x, y, z, w[3];
};
__device__ __forceinline__ Node load_node(const double* p) {
    const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1],
                  c = reinterpret_cast<const double2*>(p)[2];
    return Node{a.x, a.y, b.x, {b.y, c.x, c.y}};
}

// The moments of one segment pair.  a2: squared radius of the reduced
// kernel; ek_a > 0: NEC's coaxial factor with that radius.  NQ > 0: the
// order nq is known at compile time and the source loop unrolls.
template <int D, bool EK, int NQ, int MODE>
__device__ __forceinline__ void pair_moments(const double* si, const double* sj, int nq_rt, double k, double a2,
                                             double ek_a, cd J[D + 1][D + 1]) {
    constexpr int NM = D + 1;
    const int nq = NQ > 0 ? NQ : nq_rt;
    double f0r, f0i, kR0;
    {
        const double dx = si[0] - sj[0], dy = si[1] - sj[1], dz = si[2] - sj[2];
        const double R2 = fma(dz, dz, fma(dy, dy, dx * dx)) + a2;
        kR0 = __dmul_rn(k, R2 * rsqrt_pos(R2));
        double s, c;
        sincos(kR0, &s, &c);
        f0r = c * kInv4Pi;
        f0i = -s * kInv4Pi;
    }
#pragma unroll
    for (int p = 0; p < NM; ++p)
#pragma unroll
        for (int P = 0; P < NM; ++P) J[p][P] = cd{0.0, 0.0};
#pragma unroll 1
    for (int q = 0; q < nq; ++q) {
        const Node ni = load_node(si + q * kNodeDoubles);
        cd acc[NM];
#pragma unroll
        for (int P = 0; P < NM; ++P) acc[P] = cd{0.0, 0.0};
        // a row's phases are those of its first sample, the rounded product
        // k R, plus k (R - R_first)
        double Rq = 0.0, turn = 0.0;
#pragma unroll
        for (int r = 0; r < (NQ > 0 ? NQ : 8); ++r) {
            if (NQ == 0 && r >= nq) break;
            const Node nj = load_node(sj + r * kNodeDoubles);
            const double dx = ni.x - nj.x, dy = ni.y - nj.y, dz = ni.z - nj.z;
            const double R2 = fma(dz, dz, fma(dy, dy, dx * dx)) + a2;
            const double iR = rsqrt_pos(R2), R = R2 * iR;
            if (r == 0) {
                Rq = R;
                turn = __dmul_rn(k, R) - kR0;
            }
            double sx, cx;
            phase_step<MODE>(r == 0 ? turn : fma(k, R - Rq, turn), &sx, &cx);
            cd G{cx * iR, -sx * iR};
            if (EK && ek_a > 0.0) G = G * ek_factor(R, ek_a, k);
#pragma unroll
            for (int P = 0; P < NM; ++P) {
                acc[P].re = fma(nj.w[P], G.re, acc[P].re);
                acc[P].im = fma(nj.w[P], G.im, acc[P].im);
            }
        }
#pragma unroll
        for (int p = 0; p < NM; ++p)
#pragma unroll
            for (int P = 0; P < NM; ++P) {
                J[p][P].re = fma(ni.w[p], acc[P].re, J[p][P].re);
                J[p][P].im = fma(ni.w[p], acc[P].im, J[p][P].im);
            }
    }
#pragma unroll
    for (int p = 0; p < NM; ++p)
#pragma unroll
        for (int P = 0; P < NM; ++P) {
            const cd v = J[p][P];
            J[p][P] = cd{v.re * f0r - v.im * f0i, v.re * f0i + v.im * f0r};
        }
}

// The general orders and phase spans, out of line: their registers are not
// the common path's.
template <int D, bool EK, int NQ, int MODE>
__device__ __noinline__ void pair_moments_far(const double* si, const double* sj, int nq, double k, double a2,
                                              double ek_a, cd* dst) {
    cd J[D + 1][D + 1];
    pair_moments<D, EK, NQ, MODE>(si, sj, nq, k, a2, ek_a, J);
#pragma unroll
    for (int x = 0; x < (D + 1) * (D + 1); ++x) dst[x] = J[x / (D + 1)][x % (D + 1)];
}

// pair_moments into dst[p * NM + P] with the series its warp's arguments
// allow.  Called by whole warps (lanes without work pass `active` = false).
template <int D, bool EK>
__device__ __forceinline__ void pair_moments_any(const double* si, const double* sj, int nq, double k, double a2,
                                                 double ek_a, bool active, cd* dst) {
    constexpr int NM = D + 1;
    // (the sign of k, that of the time convention, is free)
    const double span = active ? fabs(k) * (seg_tail<D>(si, nq)[7] + seg_tail<D>(sj, nq)[7]) : 0.0;
    const bool brief = __all_sync(0xffffffffu, span <= kPhaseShort);
    const bool series = __all_sync(0xffffffffu, span <= kPhaseLong);
    if (!active) return;
    if (nq == 4 && brief) {
        cd J[NM][NM];
        pair_moments<D, EK, 4, kPhaseModeShort>(si, sj, 4, k, a2, ek_a, J);
#pragma unroll
        for (int x = 0; x < NM * NM; ++x) dst[x] = J[x / NM][x % NM];
    } else if (nq == 4 && series) {
        pair_moments_far<D, EK, 4, kPhaseModeLong>(si, sj, 4, k, a2, ek_a, dst);
    } else {
        pair_moments_far<D, EK, 0, kPhaseModeAny>(si, sj, nq, k, a2, ek_a, dst);
    }
}

// Stage 1 for one (observer segment, source basis): the source side of the
// contraction over the basis's wings.  J0: moments of the segment's row of
// pairs (NM^2 per pair), loc: the basis's wing slots, C: its coefficients.
// weight(lb) gives a pair's A and charge weights.
template <int D, class Weight>
__device__ __forceinline__ void contract_source(const cd* J0, const int* loc, const double* C, const Weight& weight,
                                                cd A[D + 1], cd Q[D]) {
    constexpr int NM = D + 1;
#pragma unroll
    for (int p = 0; p < NM; ++p) A[p] = cd{0.0, 0.0};
#pragma unroll
    for (int p = 0; p < D; ++p) Q[p] = cd{0.0, 0.0};
#pragma unroll
    for (int b = 0; b < NM; ++b) {
        const int lb = loc[b];
        if (lb < 0) continue;
        const cd* J = J0 + (size_t)lb * NM * NM;
        double c[NM];
#pragma unroll
        for (int P = 0; P < NM; ++P) c[P] = C[b * NM + P];
        const auto w = weight(lb);
#pragma unroll
        for (int p = 0; p < NM; ++p) {
            cd s{0.0, 0.0}, t{0.0, 0.0};
#pragma unroll
            for (int P = 0; P < NM; ++P) {
                const cd j = J[p * NM + P];
                s.re = fma(c[P], j.re, s.re);
                s.im = fma(c[P], j.im, s.im);
                if (p < D && P < D) {
                    const double d = (P + 1) * c[P + 1 < NM ? P + 1 : 0];
                    t.re = fma(d, j.re, t.re);
                    t.im = fma(d, j.im, t.im);
                }
            }
            w.addA(s, A[p]);
            if (p < D) w.addQ(t, Q[p]);
        }
    }
}

// Pair weights of the contraction: a real A weight (tangent product) with
// unit charge weight, or complex ones (image terms).
struct RealWeight {
    double td;
    __device__ __forceinline__ void addA(cd s, cd& A) const {
        A.re = fma(td, s.re, A.re);
        A.im = fma(td, s.im, A.im);
    }
    __device__ __forceinline__ void addQ(cd t, cd& Q) const { Q = Q + t; }
};
struct ComplexWeight {
    cd a, p;
    __device__ __forceinline__ void addA(cd s, cd& A) const { A = A + a * s; }
    __device__ __forceinline__ void addQ(cd t, cd& Q) const { Q = Q + p * t; }
};

// Stage 2 for one basis pair: the observer side, from stage 1's results
// TA [p][segment] and TQ (`plane` between powers, `pitch` between segments).
template <int D>
__device__ __forceinline__ void contract_observer(const cd* TA, const cd* TQ, int pitch, int plane, const int* loc,
                                                  const double* C, cd* zA, cd* zP) {
    constexpr int NM = D + 1;
    *zA = cd{0.0, 0.0};
    *zP = cd{0.0, 0.0};
#pragma unroll
    for (int a = 0; a < NM; ++a) {
        const int la = loc[a];
        if (la < 0) continue;
#pragma unroll
        for (int p = 0; p < NM; ++p) {
            const double c = C[a * NM + p];
            const cd t = TA[p * plane + la * pitch];
            zA->re = fma(c, t.re, zA->re);
            zA->im = fma(c, t.im, zA->im);
            if (p > 0) {
                const cd u = TQ[(p - 1) * plane + la * pitch];
                zP->re = fma(p * c, u.re, zP->re);
                zP->im = fma(p * c, u.im, zP->im);
            }
        }
    }
}

}  // namespace mw
