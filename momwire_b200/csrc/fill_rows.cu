// Impedance fill of one system together with its complex64 copy (FP64,
// sm_100a): the arithmetic of a fixed order of sums, for systems that are
// solved through complex64 factors.
//
// The reference's sums carry rounding of 1e-13 of an entry (the contraction
// cancels), so two fills that add in different orders round about one entry
// in 200,000 of the copy differently; a large system's refined coefficients
// then differ by up to 6e-8 one by one, whichever fill is the better.  Here the
// order is: source points in turn for each observer point, phases relative to
// that point's first; observer points q, q + 4, then (0, 1), (2, 3), then
// both; basis pairs from the moments one by one.
//
// One CTA owns a pair of 16 x 16 basis tiles (fill.cu has the layout); a
// thread computes a segment pair.  Bound by the FP64 pipe: 62 operations a
// sample against 36 in fill.cu, whose order is free.  Four lanes to a pair,
// each an observer point, and a shuffle reduction of the 18 sums took 13.3 ms
// on the 16 x 16 array (10,496 unknowns) on B200; 11.0 ms so, 11.9 with the full
// sine and cosine in line and every step tested for the series' range.
#include "common.cuh"
#include "fill_args.cuh"
#include "ground_weights.cuh"

namespace mw {
namespace {

// Per-segment staged data: Gauss points (3 nq), weight-folded powers
// w_q L (u_q)^p (nq*(D+1)), tangent, centre, radius.
template <int D>
struct RowStage {
    static constexpr int NM = D + 1;
    __device__ static int stride(int nq) { return nq * 3 + nq * NM + 7; }
};

template <int D>
__device__ __forceinline__ void stage_row_segment(double* dst, int nq, const GLParams& gl,
                                              const double* sl, const double* sr, const double* tg,
                                              double a, bool mirror, double gz) {
    constexpr int NM = D + 1;
    double l0 = sl[0], l1 = sl[1], l2 = sl[2];
    double r0 = sr[0], r1 = sr[1], r2 = sr[2];
    double dx = r0 - l0, dy = r1 - l1, dz = r2 - l2;
    double L = sqrt(dx * dx + dy * dy + dz * dz);
    for (int q = 0; q < nq; ++q) {
        double t = gl.t[q];
        double px = (1.0 - t) * l0 + t * r0;
        double py = (1.0 - t) * l1 + t * r1;
        double pz = (1.0 - t) * l2 + t * r2;
        if (mirror) pz = 2.0 * gz - pz;
        dst[q * 3 + 0] = px;
        dst[q * 3 + 1] = py;
        dst[q * 3 + 2] = pz;
        double u = t * L, wp = gl.w[q] * L;
        for (int p = 0; p < NM; ++p) {
            dst[nq * 3 + q * NM + p] = wp;
            wp *= u;
        }
    }
    int o = nq * 3 + nq * NM;
    dst[o + 0] = tg[0];
    dst[o + 1] = tg[1];
    dst[o + 2] = mirror ? -tg[2] : tg[2];
    double cz = 0.5 * (l2 + r2);
    dst[o + 3] = 0.5 * (l0 + r0);
    dst[o + 4] = 0.5 * (l1 + r1);
    dst[o + 5] = mirror ? 2.0 * gz - cz : cz;
    dst[o + 6] = a;
}

// sin x and cos x for |x| <= kRowPhaseMax from their Taylor series through
// x^17 and x^16 (Horner in x^2; coefficients 1/n!).  At |x| = 0.75 the first
// omitted terms, x^19/19! and x^18/18!, are below 1e-18: full double
// precision.
constexpr double kRowPhaseMax = 0.75;
__device__ __forceinline__ void phase_step_long(double x, double* sx, double* cx) {
    const double t = x * x;
    double c = 1.0 / 20922789888000.0;  // 1/16!
    c = fma(c, t, -1.0 / 87178291200.0);
    c = fma(c, t, 1.0 / 479001600.0);
    c = fma(c, t, -1.0 / 3628800.0);
    c = fma(c, t, 1.0 / 40320.0);
    c = fma(c, t, -1.0 / 720.0);
    c = fma(c, t, 1.0 / 24.0);
    c = fma(c, t, -0.5);
    *cx = fma(c, t, 1.0);
    double s = 1.0 / 355687428096000.0;  // 1/17!
    s = fma(s, t, -1.0 / 1307674368000.0);
    s = fma(s, t, 1.0 / 6227020800.0);
    s = fma(s, t, -1.0 / 39916800.0);
    s = fma(s, t, 1.0 / 362880.0);
    s = fma(s, t, -1.0 / 5040.0);
    s = fma(s, t, 1.0 / 120.0);
    s = fma(s, t, -1.0 / 6.0);
    *sx = fma(s * t, x, x);
}

// (out of line: in line it is most of a pair's code)
__device__ __noinline__ void full_phase(double x, double* s, double* c) { sincos(x, s, c); }

// The sums over the source points of observer point qi, one per source power.
// NQ > 0: the quadrature order is known at compile time (nq == NQ), so the
// source-point loop unrolls and its independent samples interleave.
// NARROW: no phase step of the tile pair exceeds kRowPhaseMax.
template <int D, bool EK, int NQ, bool NARROW>
__device__ __forceinline__ void pair_row(const double* si, const double* sj, int nq_rt, int qi,
                                         double k, bool ek_on, cd accP[D + 1]) {
    constexpr int NM = D + 1;
    const int nq = NQ > 0 ? NQ : nq_rt;
    double a = si[nq * 3 + nq * NM + 6];
    double a2 = a * a;
    double xi = si[qi * 3 + 0], yi = si[qi * 3 + 1], zi = si[qi * 3 + 2];
#pragma unroll
    for (int P = 0; P < NM; ++P) accP[P] = cd{0.0, 0.0};
    if (qi >= nq) return;
    const double* wv = sj + nq * 3;
    double R0 = 0.0, s0 = 0.0, c0 = 1.0;
#pragma unroll
    for (int r = 0; r < (NQ > 0 ? NQ : 8); ++r) {
        if (NQ == 0 && r >= nq) break;
        double dx = xi - sj[r * 3 + 0];
        double dy = yi - sj[r * 3 + 1];
        double dz = zi - sj[r * 3 + 2];
        // (roundings spelled out: which products are fused must not depend on
        // the code around them)
        const double R2 = __dadd_rn(__fma_rn(dz, dz, __fma_rn(dx, dx, __dmul_rn(dy, dy))), a2);
        // one reciprocal square root serves both R and 1/R
        double iR = rsqrt(R2);
        const double R = __dmul_rn(R2, iR);
        double s, c;
        // the first source point's phase in full; the others rotate it by
        // k (R - R0), at most k times a segment length, through that angle's
        // Taylor series (phase_step) -- a full sincos where it is wider
        const double x = __dmul_rn(k, __dsub_rn(R, R0));
        if (r == 0 || (!NARROW && fabs(x) > kRowPhaseMax)) {
            full_phase(k * R, &s, &c);
            if (r == 0) {
                R0 = R;
                s0 = s;
                c0 = c;
            }
        } else {
            double sx, cx;
            phase_step_long(x, &sx, &cx);
            s = __fma_rn(s0, cx, __dmul_rn(c0, sx));
            c = __fma_rn(c0, cx, -__dmul_rn(s0, sx));
        }
        double g = kInv4Pi * iR;
        cd G = cd{c * g, -s * g};
        if (EK && ek_on) G = G * ek_factor(R, a, k);
#pragma unroll
        for (int P = 0; P < NM; ++P) {
            double w = wv[r * NM + P];
            accP[P].re += w * G.re;
            accP[P].im += w * G.im;
        }
    }
}

// Observer point qi's share of the moment (p, P), zero past the rule.
template <int D>
__device__ __forceinline__ cd row_share(const double* si, int nq, int qi, int p, cd acc) {
    if (qi >= nq) return cd{0.0, 0.0};
    const double w = si[nq * 3 + qi * (D + 1) + p];
    return cd{__dmul_rn(w, acc.re), __dmul_rn(w, acc.im)};
}
__device__ __forceinline__ cd add_rn(cd a, cd b) { return cd{__dadd_rn(a.re, b.re), __dadd_rn(a.im, b.im)}; }

// All (D+1)^2 moments of a pair by one thread, to dst: observer points q and
// q + 4 first, then (0, 1), (2, 3), then these two sums.
template <int D, bool EK, int NQ, bool NARROW>
__device__ __forceinline__ void pair_moments_rows(const double* si, const double* sj, int nq, double k, bool ek_on,
                                                  double* dst) {
    constexpr int NM = D + 1, kHalf = NQ == 4 ? 1 : 2;
    cd acc[kHalf][4][NM];
#pragma unroll
    for (int h = 0; h < kHalf; ++h)
#pragma unroll
        for (int q = 0; q < 4; ++q) pair_row<D, EK, NQ, NARROW>(si, sj, nq, q + 4 * h, k, ek_on, acc[h][q]);
#pragma unroll
    for (int p = 0; p < NM; ++p)
#pragma unroll
        for (int P = 0; P < NM; ++P) {
            cd s[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                s[q] = row_share<D>(si, nq, q, p, acc[0][q][P]);
                if (kHalf == 2) s[q] = add_rn(s[q], row_share<D>(si, nq, q + 4, p, acc[kHalf - 1][q][P]));
            }
            const cd J = add_rn(add_rn(s[0], s[1]), add_rn(s[2], s[3]));
            dst[(p * NM + P) * 2 + 0] = J.re;
            dst[(p * NM + P) * 2 + 1] = J.im;
        }
}

// One (row tile, column tile) block of Z.  With allow_mirror the tile pair
// is checked for symmetry (every staged segment of both tiles has the same
// radius: the thin-wire kernel uses the observer radius, so only then is the
// Galerkin block of (tc, tr) the transpose of that of (tr, tc)); a symmetric
// pair also writes the transposed block.  Returns whether it did.
template <int D, bool IMAGE, bool EK>
__device__ __forceinline__ bool fill_rows_tile(const FillArgs& A, const GLParams& gl, double* smem, const int tr,
                                          const int tc, const bool allow_mirror) {
    constexpr int NM = D + 1, NMM = NM * NM;
    const int nq = gl.nq;
    const int SD = RowStage<D>::stride(nq);
    const int SMAX = A.basis.max_tile_seg;
    const int TB = A.basis.max_tile_basis;
    const int ns_r = A.basis.tile_ns[tr], ns_c = A.basis.tile_ns[tc];
    const int nb_r = A.basis.tile_nb[tr], nb_c = A.basis.tile_nb[tc];
    const int fb_r = A.basis.tile_first[tr], fb_c = A.basis.tile_first[tc];
    const double kz = A.k, omz = A.omega;
    const double* table = A.table;
    double* Zb = A.Z;
    float* Z32b = A.Z32;

    double* s_row = smem;                               // SMAX * SD
    double* s_col = s_row + SMAX * SD;                  // SMAX * SD
    double* s_J = s_col + SMAX * SD;                    // SMAX*SMAX*NMM*2
    double* s_W = s_J + (size_t)SMAX * SMAX * NMM * 2;  // image: SMAX*SMAX*4
    double* s_pr = s_W + (IMAGE ? (size_t)SMAX * SMAX * 4 : 0);  // TB*NMM
    double* s_pc = s_pr + TB * NMM;                     // TB*NMM
    double* s_out = s_pc + TB * NMM;                    // TB*TB*2 (mirrored block)
    int* s_int = reinterpret_cast<int*>(s_out + TB * TB * 2);
    int* s_seg_r = s_int;               // SMAX
    int* s_seg_c = s_seg_r + SMAX;      // SMAX
    int* s_edge_r = s_seg_c + SMAX;     // SMAX
    int* s_edge_c = s_edge_r + SMAX;
    int* s_pos_r = s_edge_c + SMAX;
    int* s_pos_c = s_pos_r + SMAX;
    int* s_grp_r = s_pos_c + SMAX;
    int* s_grp_c = s_grp_r + SMAX;
    int* s_loc_r = s_grp_c + SMAX;      // TB*NM
    int* s_loc_c = s_loc_r + TB * NM;   // TB*NM

    const int tid = threadIdx.x;
    const double gz = A.ground.ground_z;

    // ---- staging: segment lists, Gauss points, basis polynomials
    const double r_ref = A.seg.radius[A.basis.tile_seg[(size_t)tr * SMAX]];
    int odd_radius = 0, wide = nq != 4;
    for (int i = tid; i < ns_r; i += blockDim.x) {
        int s = A.basis.tile_seg[(size_t)tr * SMAX + i];
        odd_radius |= A.seg.radius[s] != r_ref;
        s_seg_r[i] = s;
        s_edge_r[i] = A.seg.edge[s];
        s_pos_r[i] = A.seg.pos_in_edge[s];
        s_grp_r[i] = EK ? A.seg.ek_group[s] : 0;
        stage_row_segment<D>(s_row + i * SD, nq, gl, A.seg.seg_l + 3 * s, A.seg.seg_r + 3 * s,
                         A.seg.tangent + 3 * s, A.seg.radius[s], false, 0.0);
    }
    for (int i = tid; i < ns_c; i += blockDim.x) {
        int s = A.basis.tile_seg[(size_t)tc * SMAX + i];
        odd_radius |= A.seg.radius[s] != r_ref;
        {
            // a phase step is at most |k| times the source segment's length
            const double *l = A.seg.seg_l + 3 * s, *r = A.seg.seg_r + 3 * s;
            const double dx = r[0] - l[0], dy = r[1] - l[1], dz = r[2] - l[2];
            wide |= !(fabs(kz) * sqrt(dx * dx + dy * dy + dz * dz) < 0.98 * kRowPhaseMax);
        }
        s_seg_c[i] = s;
        s_edge_c[i] = A.seg.edge[s];
        s_pos_c[i] = A.seg.pos_in_edge[s];
        s_grp_c[i] = EK ? (IMAGE ? A.seg.ek_group_img[s] : A.seg.ek_group[s]) : 0;
        stage_row_segment<D>(s_col + i * SD, nq, gl, A.seg.seg_l + 3 * s, A.seg.seg_r + 3 * s,
                         A.seg.tangent + 3 * s, A.seg.radius[s], IMAGE, gz);
    }
    for (int i = tid; i < nb_r * NMM; i += blockDim.x)
        s_pr[i] = A.basis.polys[(size_t)fb_r * NMM + i];
    for (int i = tid; i < nb_c * NMM; i += blockDim.x)
        s_pc[i] = A.basis.polys[(size_t)fb_c * NMM + i];
    for (int i = tid; i < nb_r * NM; i += blockDim.x) s_loc_r[i] = A.basis.loc[(size_t)fb_r * NM + i];
    for (int i = tid; i < nb_c * NM; i += blockDim.x) s_loc_c[i] = A.basis.loc[(size_t)fb_c * NM + i];
    const bool mirror = __syncthreads_or(odd_radius) == 0 && allow_mirror;
    // the default rule, short segments: unrolled, with no step's own test
    const bool narrow = __syncthreads_or(wide) == 0;

    // ---- phase A: moments of every staged segment pair, a thread each
    const int npair = ns_r * ns_c;
    for (int pidx = tid; pidx < npair; pidx += blockDim.x) {
        const int li = pidx / ns_c, lj = pidx - li * ns_c;
        double* dst = s_J + (size_t)pidx * NMM * 2;
        if (!IMAGE && s_edge_r[li] == s_edge_c[lj]) {
            int e = s_edge_r[li];
            int64_t row = A.e_off[e] + (s_pos_c[lj] - s_pos_r[li]) + A.e_n[e] - 1;
            const double* src = table + row * NMM * 2;
#pragma unroll
            for (int x = 0; x < NMM * 2; ++x) dst[x] = src[x];
        } else {
            const bool ek_on = EK && (s_grp_r[li] == s_grp_c[lj]);
            if (narrow)
                pair_moments_rows<D, EK, 4, true>(s_row + li * SD, s_col + lj * SD, 4, kz, ek_on, dst);
            else
                pair_moments_rows<D, EK, 0, false>(s_row + li * SD, s_col + lj * SD, nq, kz, ek_on, dst);
        }
        if (IMAGE) {
                // per-pair image weights
                const double* si = s_row + li * SD + nq * 3 + nq * NM;
                const double* sj = s_col + lj * SD + nq * 3 + nq * NM;
                cd wA, wP;
                if (A.ground.model == MW_GROUND_REFL) {
                    refl_weights(si + 3, si, sj + 3, sj, A.ground, &wA, &wP);
                } else {
                    double td = si[0] * sj[0] + si[1] * sj[1] + si[2] * sj[2];
                    if (A.ground.model == MW_GROUND_SOMM_IMAGE) {
                        cd et{A.ground.eps_re, A.ground.eps_im};
                        cd c2 = cdiv(cd{et.re - 1.0, et.im}, cd{et.re + 1.0, et.im});
                        wA = td * c2;
                        wP = c2;
                    } else {
                        wA = cd{td, 0.0};
                        wP = cd{1.0, 0.0};
                    }
                }
                double* w = s_W + (size_t)pidx * 4;
                w[0] = wA.re; w[1] = wA.im; w[2] = wP.re; w[3] = wP.im;
        }
    }
    __syncthreads();

    // ---- phase B: Galerkin contraction into the Z tile
    const double wmu = omz * A.mu0;
    const double inv_weps = 1.0 / (omz * A.eps0);
    for (int pp = tid; pp < TB * TB; pp += blockDim.x) {
        int mi = pp % TB, ni = pp / TB;
        if (mi >= nb_r || ni >= nb_c) continue;
        cd zA{0.0, 0.0}, zP{0.0, 0.0};
        const double* Cm = s_pr + mi * NMM;
        const double* Cn = s_pc + ni * NMM;
        for (int a = 0; a < NM; ++a) {
            int la = s_loc_r[mi * NM + a];
            if (la < 0) continue;
            for (int b = 0; b < NM; ++b) {
                int lb = s_loc_c[ni * NM + b];
                if (lb < 0) continue;
                const double* J = s_J + ((size_t)la * ns_c + lb) * NMM * 2;
                cd inA{0.0, 0.0}, inP{0.0, 0.0};
#pragma unroll
                for (int p = 0; p < NM; ++p) {
                    cd rowA{0.0, 0.0};
#pragma unroll
                    for (int P = 0; P < NM; ++P) {
                        double c = Cn[b * NM + P];
                        rowA.re += c * J[(p * NM + P) * 2 + 0];
                        rowA.im += c * J[(p * NM + P) * 2 + 1];
                    }
                    double cm = Cm[a * NM + p];
                    inA.re += cm * rowA.re;
                    inA.im += cm * rowA.im;
                }
#pragma unroll
                for (int p = 1; p < NM; ++p) {
                    cd rowP{0.0, 0.0};
#pragma unroll
                    for (int P = 1; P < NM; ++P) {
                        double c = P * Cn[b * NM + P];
                        rowP.re += c * J[((p - 1) * NM + (P - 1)) * 2 + 0];
                        rowP.im += c * J[((p - 1) * NM + (P - 1)) * 2 + 1];
                    }
                    double cm = p * Cm[a * NM + p];
                    inP.re += cm * rowP.re;
                    inP.im += cm * rowP.im;
                }
                if (IMAGE) {
                    const double* w = s_W + ((size_t)la * ns_c + lb) * 4;
                    zA = zA + cd{w[0], w[1]} * inA;
                    zP = zP + cd{w[2], w[3]} * inP;
                } else {
                    const double* ti = s_row + la * SD + nq * 3 + nq * NM;
                    const double* tj = s_col + lb * SD + nq * 3 + nq * NM;
                    double td = ti[0] * tj[0] + ti[1] * tj[1] + ti[2] * tj[2];
                    zA.re += td * inA.re;
                    zA.im += td * inA.im;
                    zP = zP + inP;
                }
            }
        }
        // j w mu zA + zP / (j w eps)
        double zre = -wmu * zA.im + inv_weps * zP.im;
        double zim = wmu * zA.re - inv_weps * zP.re;
        if (mirror) {
            s_out[(mi * TB + ni) * 2 + 0] = zre;
            s_out[(mi * TB + ni) * 2 + 1] = zim;
        }
        int64_t m = fb_r + mi, n = fb_c + ni;
        double* zp = Zb + m * 2 + n * A.ldz * 2;
        if (IMAGE) {
            zre = zp[0] - zre;
            zim = zp[1] - zim;
        }
        zp[0] = zre;
        zp[1] = zim;
        {
            float* z32 = Z32b + m * 2 + n * A.ldz32 * 2;
            z32[0] = (float)zre;
            z32[1] = (float)zim;
        }
    }
    if (!mirror) return false;
    __syncthreads();
    // the transposed block Z[n, m], column tile index fastest (coalesced)
    for (int pp = tid; pp < TB * TB; pp += blockDim.x) {
        int ni = pp % TB, mi = pp / TB;
        if (mi >= nb_r || ni >= nb_c) continue;
        double zre = s_out[(mi * TB + ni) * 2 + 0];
        double zim = s_out[(mi * TB + ni) * 2 + 1];
        int64_t m = fb_r + mi, n = fb_c + ni;
        double* zp = Zb + n * 2 + m * A.ldz * 2;
        if (IMAGE) {
            zre = zp[0] - zre;
            zim = zp[1] - zim;
        }
        zp[0] = zre;
        zp[1] = zim;
        {
            float* z32 = Z32b + n * 2 + m * A.ldz32 * 2;
            z32[0] = (float)zre;
            z32[1] = (float)zim;
        }
    }
    return true;
}

constexpr int kRowsThreads = 128;

// One block per upper-triangle tile pair (tr <= tc).  A symmetric pair is
// computed once and written to both blocks of Z; otherwise the block also
// computes (tc, tr) itself.  The EK image fill labels direct and mirrored
// segments separately, so it always computes both.
template <int D, bool IMAGE, bool EK>
__global__ void __launch_bounds__(kRowsThreads, 3) fill_rows_kernel(FillArgs A, GLParams gl) {
    extern __shared__ double smem[];
    int tr, tc;
    tri_pair((int64_t)blockIdx.x, tr, tc);
    const bool off_diag = tr != tc;
    const bool mirrored = fill_rows_tile<D, IMAGE, EK>(A, gl, smem, tr, tc, off_diag && !(IMAGE && EK));
    if (off_diag && !mirrored) {
        __syncthreads();
        fill_rows_tile<D, IMAGE, EK>(A, gl, smem, tc, tr, false);
    }
}

static size_t fill_rows_smem(int D, bool image, int nq, int smax, int tb) {
    int NM = D + 1, NMM = NM * NM;
    int SD = nq * 3 + nq * NM + 7;
    size_t dbl = (size_t)2 * smax * SD + (size_t)smax * smax * NMM * 2 + (image ? (size_t)smax * smax * 4 : 0) +
                 (size_t)2 * tb * NMM + (size_t)tb * tb * 2;
    size_t ints = (size_t)8 * smax + (size_t)2 * tb * NM;
    return dbl * 8 + ints * 4;
}

template <int D, bool IMAGE, bool EK>
mw_status launch(const FillArgs& A, const GLParams& gl, double flops, cudaStream_t st) {
    const size_t smem = fill_rows_smem(D, IMAGE, gl.nq, A.basis.max_tile_seg, A.basis.max_tile_basis);
    auto kern = fill_rows_kernel<D, IMAGE, EK>;
    MW_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int64_t nt = A.basis.n_tile;
    const double nb = A.basis.n_basis, tri = (double)(nt + 1) / (2.0 * (double)nt);
    ProfileScope ps(IMAGE ? PC_FILL_IMAGE : PC_FILL, st, tri * flops, nb * nb * 24.0 * (IMAGE ? 2.0 : 1.0));
    kern<<<(unsigned)(nt * (nt + 1) / 2), kRowsThreads, smem, st>>>(A, gl);
    MW_CHECK_CUDA(cudaGetLastError());
    count_launch();
    return MW_OK;
}

}  // namespace

mw_status fill_rows(const FillArgs& A, const GLParams& gl, bool image, bool ek, double flops, cudaStream_t st) {
    const bool d1 = A.basis.degree == 1;
    if (image) {
        if (ek) return d1 ? launch<1, true, true>(A, gl, flops, st) : launch<2, true, true>(A, gl, flops, st);
        return d1 ? launch<1, true, false>(A, gl, flops, st) : launch<2, true, false>(A, gl, flops, st);
    }
    if (ek) return d1 ? launch<1, false, true>(A, gl, flops, st) : launch<2, false, true>(A, gl, flops, st);
    return d1 ? launch<1, false, false>(A, gl, flops, st) : launch<2, false, false>(A, gl, flops, st);
}

}  // namespace mw
