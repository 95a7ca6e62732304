// Galerkin impedance fill for the B-spline thin-wire EFIE (FP64), sm_100a.
//
// Reference algorithm: momwire bspline.py _compute_Z_operator (:3702) with
// _bspline_kernels.py's moment integrals and _accelerators.cpp's assembly.
// Design (B200-first, not a port):
//   * one CTA owns a tile of up to 16 x 16 basis pairs; the segments its
//     bases touch (<= 24 per side) are staged in shared memory as their Gauss
//     points with weight-folded monomials;
//   * phase A computes the (d+1)^2 moments of every touched segment pair, one
//     thread each, straight into shared memory; same-edge pairs read the
//     analytic static + smooth Toeplitz table instead;
//   * phase B contracts moments with the basis polynomials into Z (source
//     side, then observer side) and writes the tile column-major (optionally
//     a complex64 copy for the mixed-precision factorisation).
// The arithmetic of both phases is in pair_moments.cuh.
// The (d+1)^2 x N^2 moment tensor of the reference never exists.
#include <cstdio>

#include "common.cuh"
#include "fill_args.cuh"
#include "pair_moments.cuh"

namespace mw {

static GLParams make_gl(int nq) {
    GLParams g{};
    g.nq = nq;
    const double *t, *w;
    gauss_legendre01(nq, &t, &w);
    for (int i = 0; i < nq; ++i) { g.t[i] = t[i]; g.w[i] = w[i]; }
    gauss_legendre01(20, &t, &w);
    for (int i = 0; i < 20; ++i) { g.x20[i] = 2.0 * t[i] - 1.0; g.w20[i] = 2.0 * w[i]; }
    return g;
}

// fac - fac_static = T1 (3 j kr - kr^2) - T2 (j kr)   (_bspline_kernels.py:225)
__device__ __forceinline__ cd ek_reg_extra(double R, double a, double k) {
    double kr = k * R;
    double ar = a / R;
    double ar2 = ar * ar;
    double t1 = 0.25 * ar2 * ar2;
    double t2 = 0.5 * ar2;
    return cd{-t1 * kr * kr, 3.0 * t1 * kr - t2 * kr};
}

// --------------------------------------------------------------------------
// Same-edge Toeplitz table
// --------------------------------------------------------------------------

// W_pq(t) = int u^p (u - t)^q du over [0,h] ∩ [t, h+t], all terms >= 0.
template <int D>
__device__ __forceinline__ void conv_weights(double h, double t, double W[D + 1][D + 1]) {
    const double binom[3][3] = {{1, 0, 0}, {1, 1, 0}, {1, 2, 1}};
    double at = fabs(t), rest = h - at;
    double tp[D + 1], rp[2 * D + 2];
    tp[0] = 1.0;
    for (int i = 1; i <= D; ++i) tp[i] = tp[i - 1] * at;
    rp[0] = 1.0;
    for (int i = 1; i < 2 * D + 2; ++i) rp[i] = rp[i - 1] * rest;
#pragma unroll
    for (int p = 0; p <= D; ++p)
#pragma unroll
        for (int q = 0; q <= D; ++q) {
            double acc = 0.0;
            if (t >= 0.0) {
                for (int r = 0; r <= p; ++r) {
                    int e = q + r + 1;
                    acc += binom[p][r] * tp[p - r] * rp[e] / e;
                }
            } else {
                for (int r = 0; r <= q; ++r) {
                    int e = p + r + 1;
                    acc += binom[q][r] * tp[q - r] * rp[e] / e;
                }
            }
            W[p][q] = acc;
        }
}

// The static integral of one table row is a sum over Gauss points of
// graded panels on the two half-intervals [-h, 0] and [0, h].  A half whose
// kernel peak c is at least one interval length away is a single 20-point
// panel; otherwise the panels grow geometrically from the end nearest the
// peak: [0, s], [s, 2s], [2s, 4s], ... (s = the radius) until they cover the
// interval.  The peak of every same-edge table entry sits on an end of the
// half interval (c = delta*h with integer delta) or outside it.
__device__ __forceinline__ int half_panels(double lo, double hi, double c, double a, bool& graded,
                                           bool& near_left) {
    const double L = hi - lo;
    const double dist = (c < lo) ? lo - c : (c > hi ? c - hi : 0.0);
    graded = dist < L;
    near_left = fabs(lo - c) <= fabs(hi - c);
    if (!graded) return 1;
    int n = 1;
    for (double s1 = fmax(a, 1e-300); s1 < L; s1 *= 2.0) ++n;
    return n;
}

// Bounds of panel i of a half-interval (see half_panels).
__device__ __forceinline__ void half_panel_bounds(double lo, double hi, double a, bool graded, bool near_left,
                                                  int i, double& x0, double& x1) {
    if (!graded) {
        x0 = lo;
        x1 = hi;
        return;
    }
    const double L = hi - lo, s = fmax(a, 1e-300);
    const double e0 = i == 0 ? 0.0 : fmin(ldexp(s, i - 1), L);
    const double e1 = fmin(ldexp(s, i), L);
    if (near_left) {
        x0 = lo + e0;
        x1 = lo + e1;
    } else {
        x0 = hi - e1;
        x1 = hi - e0;
    }
}

// One Gauss point g of panel [x0, x1] of the static integral:
// acc += half_width w_g K(t - c) W(t), K = 1/R (+ the EK correction).
template <int D, bool EK>
__device__ __forceinline__ void static_point(double x0, double x1, int g, double c, double h, double a,
                                             const GLParams& gl, double acc[D + 1][D + 1]) {
    const double half = 0.5 * (x1 - x0), mid = 0.5 * (x0 + x1);
    const double t = mid + half * gl.x20[g];
    const double x = t - c;
    const double R2 = x * x + a * a;
    const double R = sqrt(R2);
    double K = 1.0 / R;
    if (EK) K += (a * a / (4.0 * R2 * R2 * R)) * (3.0 * a * a - 2.0 * R2);
    double W[D + 1][D + 1];
    conv_weights<D>(h, t, W);
    const double wk = half * gl.w20[g] * K;
#pragma unroll
    for (int p = 0; p <= D; ++p)
#pragma unroll
        for (int q = 0; q <= D; ++q) acc[p][q] += wk * W[p][q];
}

template <int N>
__device__ __forceinline__ void warp_sum(double (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], off);
}

// Table modes: kTableFused writes static + smooth parts for one k per
// blockIdx.y; a frequency batch instead runs kTableStatic once (the static
// part is k-independent: it is written, as the real part, into all n_k
// tables) and then kTableSmoothAdd per k, which adds the smooth part.
enum { kTableFused = 0, kTableStatic = 1, kTableSmoothAdd = 2 };
constexpr int kTableThreads = 128;  // one warp per table row

// One warp per same-edge table row: the lanes split the static quadrature
// points and the nq x nq smooth-part samples, then reduce with shuffles.
template <int D, bool EK>
__global__ void __launch_bounds__(kTableThreads) same_edge_table_kernel(
    int n_edge, const int32_t* __restrict__ n_in_edge, const int64_t* __restrict__ table_off,
    const double* __restrict__ hs, const double* __restrict__ radii, int64_t rows, double k0, GLParams gl,
    double* __restrict__ out, const double* __restrict__ kb, int64_t out_stride, int mode = kTableFused,
    int n_k = 1) {
    constexpr int NM = D + 1, NE = NM * NM * 2;
    const int lane = threadIdx.x & 31;
    const int64_t row = blockIdx.x * (int64_t)(kTableThreads / 32) + (threadIdx.x >> 5);
    if (row >= rows) return;  // uniform per warp
    const double k = kb ? kb[blockIdx.y] : k0;
    double* const out0 = out;
    out += blockIdx.y * out_stride;
    // edge owning this row: last e with table_off[e] <= row
    int lo = 0, hi = n_edge - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (table_off[mid] <= row) lo = mid; else hi = mid - 1;
    }
    const int e = lo;
    const int n = n_in_edge[e];
    const int delta = (int)(row - table_off[e]) - (n - 1);
    const double h = hs[e], a = radii[e];
    const double c = delta * h;

    double st[NM * NM];
#pragma unroll
    for (int i = 0; i < NM * NM; ++i) st[i] = 0.0;
    if (mode != kTableSmoothAdd) {
        bool g0, l0, g1, l1;
        const int n0 = half_panels(-h, 0.0, c, a, g0, l0);
        const int n1 = half_panels(0.0, h, c, a, g1, l1);
        double acc[NM][NM];
#pragma unroll
        for (int p = 0; p < NM; ++p)
#pragma unroll
            for (int q = 0; q < NM; ++q) acc[p][q] = 0.0;
        for (int g = lane; g < 20 * (n0 + n1); g += 32) {
            const int pi = g / 20, gi = g - pi * 20;
            double x0, x1;
            if (pi < n0) half_panel_bounds(-h, 0.0, a, g0, l0, pi, x0, x1);
            else         half_panel_bounds(0.0, h, a, g1, l1, pi - n0, x0, x1);
            static_point<D, EK>(x0, x1, gi, c, h, a, gl, acc);
        }
#pragma unroll
        for (int p = 0; p < NM; ++p)
#pragma unroll
            for (int q = 0; q < NM; ++q) st[p * NM + q] = kInv4Pi * acc[p][q];
        warp_sum(st);
    }
    if (mode == kTableStatic) {
        for (int idx = lane; idx < n_k * NE; idx += 32) {
            const int b = idx / NE, x = idx - b * NE;
            out0[b * out_stride + row * NE + x] = (x & 1) ? 0.0 : st[x >> 1];
        }
        return;
    }

    // smooth part: (exp(-jkR) - 1)/(4 pi R) on nq x nq Gauss points
    double rg[NE];
#pragma unroll
    for (int i = 0; i < NE; ++i) rg[i] = 0.0;
    for (int smp = lane; smp < gl.nq * gl.nq; smp += 32) {
        const int qi = smp / gl.nq, ri = smp - qi * gl.nq;
        const double u = gl.t[qi] * h, wu = gl.w[qi] * h;
        const double v = gl.t[ri] * h, wv = gl.w[ri] * h;
        const double x = u - v - c;
        const double R = sqrt(x * x + a * a);
        double s, co, sh, ch;
        sincos(k * R, &s, &co);
        sincos(0.5 * k * R, &sh, &ch);
        // exp(-jkR) - 1 = -2 sin^2(kR/2) - j sin(kR)
        cd num = cd{-2.0 * sh * sh, -s};
        if (EK) num = num * ek_factor(R, a, k) + ek_reg_extra(R, a, k);
        const double g = kInv4Pi / R;
        const cd G = cd{num.re * g, num.im * g};
        double up = wu;
#pragma unroll
        for (int p = 0; p < NM; ++p) {
            double vp = wv;
#pragma unroll
            for (int P = 0; P < NM; ++P) {
                rg[(p * NM + P) * 2 + 0] += up * vp * G.re;
                rg[(p * NM + P) * 2 + 1] += up * vp * G.im;
                vp *= v;
            }
            up *= u;
        }
    }
    warp_sum(rg);
    if (lane < NE) {
        double* o = out + row * NE + lane;
        // rg[lane] with a lane-dependent index: pick it with a static loop
        double mine = 0.0, stat = 0.0;
#pragma unroll
        for (int i = 0; i < NE; ++i)
            if (i == lane) mine = rg[i];
#pragma unroll
        for (int i = 0; i < NM * NM; ++i)
            if (2 * i == lane) stat = st[i];
        if (mode == kTableSmoothAdd) *o += mine;
        else *o = stat + mine;
    }
}

// --------------------------------------------------------------------------
// Fused fill kernel
// --------------------------------------------------------------------------

// Column bases per contraction round: half a tile, so that three blocks'
// shared memory fits an SM.
constexpr int kFillCols = MW_MAX_TILE_BASIS / 2;

// Shared memory of a tile pair, in elements.
template <int D, bool IMAGE>
struct FillSmem {
    static constexpr int NM = D + 1;
    size_t nJ, nT, nW, bytes;
    __host__ __device__ FillSmem(int nq, int smax, int tb) {
        const size_t pairs = (size_t)smax * smax;
        nJ = pairs * NM * NM;
        nT = (size_t)(NM + D) * smax * (kFillCols + 1);
        nW = IMAGE ? pairs * 2 : 0;
        bytes = (nJ + nT + nW) * sizeof(cd) +
                ((size_t)2 * smax * seg_stride<D>(nq) + (size_t)2 * tb * NM * NM) * sizeof(double) +
                ((size_t)6 * smax + (size_t)2 * tb * NM) * sizeof(int);
    }
};

// One (row tile, column tile) block of Z.  With allow_mirror the tile pair
// is checked for symmetry (every staged segment of both tiles has the same
// radius: the thin-wire kernel uses the observer radius, so only then is the
// Galerkin block of (tc, tr) the transpose of that of (tr, tc)); a symmetric
// pair also writes the transposed block.  Returns whether it did.
template <int D, bool IMAGE, bool EK, int NT>
__device__ __forceinline__ bool fill_tile(const FillArgs& A, const GLParams& gl, double* smem, const int tr,
                                          const int tc, const bool allow_mirror) {
    constexpr int NM = D + 1, NMM = NM * NM;
    const int nq = gl.nq;
    const int SD = seg_stride<D>(nq);
    const int SMAX = A.basis.max_tile_seg;
    const int TB = A.basis.max_tile_basis;
    const int ns_r = A.basis.tile_ns[tr], ns_c = A.basis.tile_ns[tc];
    const int nb_r = A.basis.tile_nb[tr], nb_c = A.basis.tile_nb[tc];
    const int fb_r = A.basis.tile_first[tr], fb_c = A.basis.tile_first[tc];
    const int bz = blockIdx.z;
    const double kz = A.kb ? A.kb[bz] : A.k;
    const double omz = A.omegab ? A.omegab[bz] : A.omega;
    const double* table = A.table ? A.table + bz * A.table_stride : nullptr;
    // z_stride / z32_stride count complex elements (two scalars each)
    double* Zb = A.Z + 2 * bz * A.z_stride;
    float* Z32b = A.Z32 ? A.Z32 + 2 * bz * A.z32_stride : nullptr;

    const FillSmem<D, IMAGE> lay(nq, SMAX, TB);
    cd* s_J = reinterpret_cast<cd*>(smem);            // SMAX*SMAX*NMM moments
    cd* s_T = s_J + lay.nJ;                           // stage 1: (NM + D) planes of SMAX x (kFillCols + 1)
    cd* s_W = s_T + lay.nT;                           // image: the pairs' weights, 2 each
    double* s_row = reinterpret_cast<double*>(s_W + lay.nW);  // SMAX * SD
    double* s_col = s_row + SMAX * SD;                // SMAX * SD
    double* s_pr = s_col + SMAX * SD;                 // TB*NMM
    double* s_pc = s_pr + TB * NMM;                   // TB*NMM
    int* s_edge_r = reinterpret_cast<int*>(s_pc + TB * NMM);  // SMAX each
    int* s_edge_c = s_edge_r + SMAX;
    int* s_pos_r = s_edge_c + SMAX;
    int* s_pos_c = s_pos_r + SMAX;
    int* s_grp_r = s_pos_c + SMAX;
    int* s_grp_c = s_grp_r + SMAX;
    int* s_loc_r = s_grp_c + SMAX;      // TB*NM
    int* s_loc_c = s_loc_r + TB * NM;   // TB*NM

    const int tid = threadIdx.x;
    const double gz = A.ground.ground_z;

    // ---- staging: a thread per segment node, basis tables
    const double r_ref = A.seg.radius[A.basis.tile_seg[(size_t)tr * SMAX]];
    int odd_radius = 0;
    for (int e = tid; e < (ns_r + ns_c) * nq; e += NT) {
        const int g = e / nq, q = e - g * nq;
        const bool c = g >= ns_r;
        const int i = c ? g - ns_r : g;
        const int s = A.basis.tile_seg[(size_t)(c ? tc : tr) * SMAX + i];
        const double a = A.seg.radius[s];
        stage_node<D>((c ? s_col : s_row) + i * SD, nq, q, gl.t, gl.w, A.seg.seg_l + 3 * s, A.seg.seg_r + 3 * s,
                      A.seg.tangent + 3 * s, a, IMAGE && c, gz);
        if (q == 0) {
            odd_radius |= a != r_ref;
            (c ? s_edge_c : s_edge_r)[i] = A.seg.edge[s];
            (c ? s_pos_c : s_pos_r)[i] = A.seg.pos_in_edge[s];
            (c ? s_grp_c : s_grp_r)[i] = EK ? (IMAGE && c ? A.seg.ek_group_img[s] : A.seg.ek_group[s]) : 0;
        }
    }
    for (int i = tid; i < nb_r * NMM; i += NT)
        s_pr[i] = A.basis.polys[(size_t)fb_r * NMM + i];
    for (int i = tid; i < nb_c * NMM; i += NT)
        s_pc[i] = A.basis.polys[(size_t)fb_c * NMM + i];
    for (int i = tid; i < nb_r * NM; i += NT) s_loc_r[i] = A.basis.loc[(size_t)fb_r * NM + i];
    for (int i = tid; i < nb_c * NM; i += NT) s_loc_c[i] = A.basis.loc[(size_t)fb_c * NM + i];
    const bool mirror = __syncthreads_or(odd_radius) == 0 && allow_mirror;

    // ---- phase A: moments of every staged segment pair, one thread each
    const int npair = ns_r * ns_c;
    for (int p0 = 0; p0 < npair; p0 += NT) {
        const int pidx = p0 + tid;
        const bool valid = pidx < npair;
        const int li = valid ? pidx / ns_c : 0;
        const int lj = valid ? pidx - li * ns_c : 0;
        const bool same_edge = !IMAGE && valid && s_edge_r[li] == s_edge_c[lj];
        const double* si = s_row + li * SD;
        const double* sj = s_col + lj * SD;
        const double* ti = seg_tail<D>(si, nq);
        const double a2 = ti[6];
        const double ek_a = EK && s_grp_r[li] == s_grp_c[lj] ? sqrt(a2) : 0.0;
        cd* dst = s_J + (size_t)(valid ? pidx : 0) * NMM;
        pair_moments_any<D, EK>(si, sj, nq, kz, a2, ek_a, valid && !same_edge, dst);
        if (valid) {
            if (same_edge) {
                const int e = s_edge_r[li];
                const int64_t row = A.e_off[e] + (s_pos_c[lj] - s_pos_r[li]) + A.e_n[e] - 1;
                const double* src = table + 2 * row * NMM;
#pragma unroll
                for (int x = 0; x < NMM; ++x) {
                    const double2 v = load_pair(src + 2 * x, A.wide);
                    dst[x] = cd{v.x, v.y};
                }
            }
            if (IMAGE) {
                // per-pair image weights
                const double* tj = seg_tail<D>(sj, nq);
                cd wA, wP;
                if (A.ground.model == MW_GROUND_REFL) {
                    refl_weights(ti + 3, ti, tj + 3, tj, A.ground, &wA, &wP);
                } else {
                    const double td = ti[0] * tj[0] + ti[1] * tj[1] + ti[2] * tj[2];
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
                s_W[2 * pidx] = wA;
                s_W[2 * pidx + 1] = wP;
            }
        }
    }
    __syncthreads();

    // ---- phase B: Galerkin contraction, source side then observer side,
    // kFillCols column bases at a time
    constexpr int pitch = kFillCols + 1;
    const int plane = SMAX * pitch;
    cd* TQ = s_T + NM * plane;
    const double wmu = omz * A.mu0;
    const double inv_weps = 1.0 / (omz * A.eps0);
    // into Z[m, n]: the value, or under a ground what the image term leaves
    auto put = [&](int64_t m, int64_t n, double zre, double zim) {
        double* zp = Zb + m * 2 + n * A.ldz * 2;
        if (IMAGE) {
            const double2 z = load_pair(zp, A.wide);
            zre = z.x - zre;
            zim = z.y - zim;
        }
        store_pair(zp, A.wide, zre, zim);
        if (Z32b) store_pair(Z32b + m * 2 + n * A.ldz32 * 2, A.wide, (float)zre, (float)zim);
    };
    for (int n0 = 0; n0 < nb_c; n0 += kFillCols) {
        const int nc = min(kFillCols, nb_c - n0);
        for (int it = tid; it < ns_r * kFillCols; it += NT) {
            const int la = it / kFillCols, nl = it % kFillCols, ni = n0 + nl;
            if (nl >= nc) continue;
            const double* ti = seg_tail<D>(s_row + la * SD, nq);
            cd a[NM], q[D];
            const cd* J0 = s_J + (size_t)la * ns_c * NMM;
            if constexpr (IMAGE) {
                contract_source<D>(J0, s_loc_c + ni * NM, s_pc + ni * NMM,
                                   [&](int lb) {
                                       return ComplexWeight{s_W[2 * (la * ns_c + lb)], s_W[2 * (la * ns_c + lb) + 1]};
                                   },
                                   a, q);
            } else {
                contract_source<D>(J0, s_loc_c + ni * NM, s_pc + ni * NMM,
                                   [&](int lb) {
                                       const double* tj = seg_tail<D>(s_col + lb * SD, nq);
                                       return RealWeight{ti[0] * tj[0] + ti[1] * tj[1] + ti[2] * tj[2]};
                                   },
                                   a, q);
            }
#pragma unroll
            for (int p = 0; p < NM; ++p) s_T[p * plane + la * pitch + nl] = a[p];
#pragma unroll
            for (int p = 0; p < D; ++p) TQ[p * plane + la * pitch + nl] = q[p];
        }
        __syncthreads();
        // column-major Z: the row basis fastest
        for (int pp = tid; pp < TB * kFillCols; pp += NT) {
            const int mi = pp % TB, nl = pp / TB;
            if (mi >= nb_r || nl >= nc) continue;
            cd zA, zP;
            contract_observer<D>(s_T + nl, TQ + nl, pitch, plane, s_loc_r + mi * NM, s_pr + mi * NMM, &zA, &zP);
            // j w mu zA + zP / (j w eps)
            const double zre = -wmu * zA.im + inv_weps * zP.im, zim = wmu * zA.re - inv_weps * zP.re;
            put(fb_r + mi, fb_c + n0 + nl, zre, zim);
            // the transposed block: a warp holds two column bases, so 32-byte
            // pieces of sixteen columns of Z, which L2 puts together
            if (mirror) put(fb_c + n0 + nl, fb_r + mi, zre, zim);
        }
        if (n0 + kFillCols < nb_c) __syncthreads();
    }
    return mirror;
}

// One block per upper-triangle tile pair (tr <= tc).  A symmetric pair is
// computed once and written to both blocks of Z; otherwise the block also
// computes (tc, tr) itself.  The EK image fill labels direct and mirrored
// segments separately, so it always computes both.
//
// What bounds it: the FP64 pipe in phase A, latency in staging and phase B,
// so the blocks of an SM must be in different phases.  A block is NT threads,
// as many blocks as shared memory lets share an SM, and twelve (or eleven)
// warps at 168 registers in all: the samples need those, and spilling them
// for more warps loses more than it hides (18 warps at 96: 9.7 ms).
// Measured on B200, fill of the 16 x 16 array with its complex64 copy: 13.3
// ms with four lanes per pair and 256 threads, 7.6 with one thread per pair
// and two blocks of 176, 6.7 with three blocks of 128 -- the
// samples' FP64 operations alone take about 4.
template <int D, bool IMAGE, bool EK, int NT>
__global__ void __launch_bounds__(NT, NT == 128 ? 3 : (NT == 192 ? 2 : 1)) fill_kernel(FillArgs A, GLParams gl) {
    extern __shared__ __align__(16) double smem[];
    int tr, tc;
    tri_pair((int64_t)blockIdx.x, tr, tc);
    const bool off_diag = tr != tc;
    const bool mirrored = fill_tile<D, IMAGE, EK, NT>(A, gl, smem, tr, tc, off_diag && !(IMAGE && EK));
    if (off_diag && !mirrored) {
        __syncthreads();
        fill_tile<D, IMAGE, EK, NT>(A, gl, smem, tc, tr, false);
    }
}

// --------------------------------------------------------------------------
// Standalone moment tensor (parity tests; the fill never materialises J)
// --------------------------------------------------------------------------

template <int D>
__global__ void __launch_bounds__(128) offedge_moments_kernel(mw_segments si, mw_segments sj, double k, int mirror,
                                                              double gz, const int32_t* gi, const int32_t* gj,
                                                              GLParams gl, double* __restrict__ out) {
    constexpr int NM = D + 1;
    const int nq = gl.nq;
    const int64_t pair = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t npair = (int64_t)si.n_seg * sj.n_seg;
    const bool valid = pair < npair;
    const int i = valid ? (int)(pair / sj.n_seg) : 0;
    const int j = valid ? (int)(pair - (int64_t)i * sj.n_seg) : 0;
    __align__(16) double bi[seg_stride<D>(8)], bj[seg_stride<D>(8)];
    for (int q = 0; q < nq; ++q) {
        stage_node<D>(bi, nq, q, gl.t, gl.w, si.seg_l + 3 * i, si.seg_r + 3 * i, si.tangent + 3 * i, si.radius[i],
                      false, 0.0);
        stage_node<D>(bj, nq, q, gl.t, gl.w, sj.seg_l + 3 * j, sj.seg_r + 3 * j, sj.tangent + 3 * j, sj.radius[j],
                      mirror != 0, gz);
    }
    const double a2 = seg_tail<D>(bi, nq)[6];
    cd J[NM * NM];
    if (gi && gj)
        pair_moments_any<D, true>(bi, bj, nq, k, a2, valid && gi[i] == gj[j] ? sqrt(a2) : 0.0, valid, J);
    else
        pair_moments_any<D, false>(bi, bj, nq, k, a2, 0.0, valid, J);
    if (!valid) return;
#pragma unroll
    for (int p = 0; p < NM; ++p)
#pragma unroll
        for (int P = 0; P < NM; ++P) {
            const size_t o = (((size_t)p * NM + P) * si.n_seg + i) * sj.n_seg + j;
            out[2 * o + 0] = J[p * NM + P].re;
            out[2 * o + 1] = J[p * NM + P].im;
        }
}

// --------------------------------------------------------------------------
// Host launchers
// --------------------------------------------------------------------------

// Algorithmic flops of one fill: q^2 * 20 per kernel sample group plus the
// (d+1)^2 moment FMAs per segment pair, and the Galerkin contraction per
// basis pair, (d+1)^2 [2 (d+1)^2 + 2 d^2] * 2.
static double fill_flops(int D, int nq, double n_seg, double n_basis) {
    double NM = D + 1;
    double f_pair = nq * nq * 20.0 + NM * NM * nq * nq * 4.0;
    double f_basis = NM * NM * (2.0 * NM * NM + 2.0 * D * D) * 2.0;
    return n_seg * n_seg * f_pair + n_basis * n_basis * f_basis;
}

// The block size by the blocks whose shared memory an SM holds (it grows with
// the square of the largest tile's segment count, 18 for a solver's tiles and
// at most 24): three blocks of 128 threads, two of 192 (the image fill at
// degree 2), or one of 352.
constexpr size_t kFillSmemSM = 227 * 1024;

template <int D, bool IMAGE, bool EK>
static mw_status launch_fill(FillArgs A, const GLParams& gl, cudaStream_t st) {
    A.wide = aligned_to(A.Z, 16) && aligned_to(A.table, 16) && aligned_to(A.Z32, 8);
    // A single system with a complex64 copy is about to be solved through
    // complex64 factors.  Single coefficients of a large one follow the
    // copy's roundings to 6e-8 (16 x 16 array, 10,496 unknowns), and this
    // kernel's sums differ from fill_rows.cu's by 1e-13 of an entry, enough to
    // turn a thousand of them: there Z keeps fill_rows.cu's order of sums,
    // 11.0 ms against 6.7 here.  Sweeps' small systems move by 1e-11.
    if (A.Z32 && A.nbatch == 0) return fill_rows(A, gl, IMAGE, EK, fill_flops(D, gl.nq, A.seg.n_seg, A.basis.n_basis), st);
    const size_t smem = FillSmem<D, IMAGE>(gl.nq, A.basis.max_tile_seg, A.basis.max_tile_basis).bytes;
    const size_t fit = kFillSmemSM / (smem + 1024);
    auto kern = fit >= 3 ? fill_kernel<D, IMAGE, EK, 128>
                         : (fit == 2 ? fill_kernel<D, IMAGE, EK, 192> : fill_kernel<D, IMAGE, EK, 352>);
    const int threads = fit >= 3 ? 128 : (fit == 2 ? 192 : 352);
    MW_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int nbz = A.nbatch > 0 ? A.nbatch : 1;
    const int64_t nt = A.basis.n_tile;
    dim3 grid((unsigned)(nt * (nt + 1) / 2), 1, nbz);
    double nb = A.basis.n_basis;
    // flops of the upper-triangle tile pairs (the mirrored blocks are
    // written, not recomputed, when every segment has one radius)
    const double tri = (double)(nt + 1) / (2.0 * (double)nt);
    ProfileScope ps(IMAGE ? PC_FILL_IMAGE : PC_FILL, st, tri * nbz * fill_flops(D, gl.nq, A.seg.n_seg, nb),
                    nbz * nb * nb * (16.0 + (A.Z32 ? 8.0 : 0.0)) * (IMAGE ? 2.0 : 1.0));
    kern<<<grid, threads, smem, st>>>(A, gl);
    MW_CHECK_CUDA(cudaGetLastError());
    count_launch();
    return MW_OK;
}

}  // namespace mw

using namespace mw;

static mw_status check_common(const mw_basis* b, int n_qp) {
    MW_REQUIRE(b != nullptr, "basis is NULL");
    MW_REQUIRE(b->degree == 1 || b->degree == 2, "degree must be 1 or 2 (got %d)", b->degree);
    MW_REQUIRE(n_qp >= 1 && n_qp <= 8, "n_qp_pair must be in [1, 8] (got %d)", n_qp);
    MW_REQUIRE(b->max_tile_basis >= 1 && b->max_tile_basis <= MW_MAX_TILE_BASIS,
               "max_tile_basis out of range (%d)", b->max_tile_basis);
    MW_REQUIRE(b->max_tile_seg >= 1 && b->max_tile_seg <= MW_MAX_TILE_SEG, "max_tile_seg out of range (%d)",
               b->max_tile_seg);
    MW_REQUIRE(b->n_tile >= 1, "no basis tiles");
    return MW_OK;
}

extern "C" mw_status mw_same_edge_table(const mw_edges* edges, int32_t degree, int32_t n_qp,
                                        int32_t extended_kernel, double k, double* out, void* stream) {
    MW_REQUIRE(edges && out, "NULL argument");
    MW_REQUIRE(degree == 1 || degree == 2, "degree must be 1 or 2 (got %d)", degree);
    MW_REQUIRE(n_qp >= 1 && n_qp <= 8, "n_qp_pair must be in [1, 8] (got %d)", n_qp);
    if (edges->table_rows == 0) return MW_OK;
    GLParams gl = make_gl(n_qp);
    const int threads = kTableThreads, rows_per_block = kTableThreads / 32;
    int64_t blocks = (edges->table_rows + rows_per_block - 1) / rows_per_block;
    cudaStream_t st = as_stream(stream);
    ProfileScope ps(PC_TABLE, st);
#define MW_TBL(DD, EE)                                                                                 \
    same_edge_table_kernel<DD, EE><<<(unsigned)blocks, threads, 0, st>>>(                                \
        edges->n_edge, edges->n_in_edge, edges->table_off, edges->h, edges->radius, edges->table_rows, k, \
        gl, out, nullptr, 0)
    if (degree == 1) { if (extended_kernel) MW_TBL(1, true); else MW_TBL(1, false); }
    else             { if (extended_kernel) MW_TBL(2, true); else MW_TBL(2, false); }
#undef MW_TBL
    MW_CHECK_CUDA(cudaGetLastError());
    count_launch();
    return MW_OK;
}

extern "C" mw_status mw_offedge_moments(const mw_segments* seg_i, const mw_segments* seg_j, int32_t degree,
                                        int32_t n_qp, double k, int32_t mirror, double ground_z,
                                        const int32_t* groups_i, const int32_t* groups_j, double* out,
                                        void* stream) {
    MW_REQUIRE(seg_i && seg_j && out, "NULL argument");
    MW_REQUIRE(degree == 1 || degree == 2, "degree must be 1 or 2 (got %d)", degree);
    MW_REQUIRE(n_qp >= 1 && n_qp <= 8, "n_qp_pair must be in [1, 8] (got %d)", n_qp);
    int64_t npair = (int64_t)seg_i->n_seg * seg_j->n_seg;
    if (npair == 0) return MW_OK;
    GLParams gl = make_gl(n_qp);
    int threads = 128;
    int64_t blocks = (npair + threads - 1) / threads;
    cudaStream_t st = as_stream(stream);
    if (degree == 1)
        offedge_moments_kernel<1><<<(unsigned)blocks, threads, 0, st>>>(*seg_i, *seg_j, k, mirror, ground_z,
                                                                        groups_i, groups_j, gl, out);
    else
        offedge_moments_kernel<2><<<(unsigned)blocks, threads, 0, st>>>(*seg_i, *seg_j, k, mirror, ground_z,
                                                                        groups_i, groups_j, gl, out);
    MW_CHECK_CUDA(cudaGetLastError());
    count_launch();
    return MW_OK;
}

extern "C" mw_status mw_fill_z(const mw_segments* seg, const mw_basis* basis, const double* table,
                               const mw_edges* edges, const mw_freq* freq, int32_t n_qp, double* Z, int64_t ldz,
                               float* Z32, int64_t ldz32, void* stream) {
    MW_REQUIRE(seg && basis && table && edges && freq && Z, "NULL argument");
    mw_status s = check_common(basis, n_qp);
    if (s != MW_OK) return s;
    MW_REQUIRE(ldz >= basis->n_basis, "ldz < n_basis");
    MW_REQUIRE(Z32 == nullptr || ldz32 >= basis->n_basis, "ldz32 < n_basis");
    FillArgs A{};
    A.seg = *seg;
    A.basis = *basis;
    A.table = table;
    A.e_n = edges->n_in_edge;
    A.e_off = edges->table_off;
    A.k = freq->k;
    A.omega = freq->omega;
    A.eps0 = freq->eps0;
    A.mu0 = freq->mu0;
    A.Z = Z;
    A.ldz = ldz;
    A.Z32 = Z32;
    A.ldz32 = ldz32;
    GLParams gl = make_gl(n_qp);
    cudaStream_t st = as_stream(stream);
    bool ek = seg->ek_group != nullptr;
    if (basis->degree == 1) return ek ? launch_fill<1, false, true>(A, gl, st) : launch_fill<1, false, false>(A, gl, st);
    return ek ? launch_fill<2, false, true>(A, gl, st) : launch_fill<2, false, false>(A, gl, st);
}

extern "C" mw_status mw_fill_z_image(const mw_segments* seg, const mw_basis* basis, const mw_ground* ground,
                                     const mw_freq* freq, int32_t n_qp, double* Z, int64_t ldz, float* Z32,
                                     int64_t ldz32, void* stream) {
    MW_REQUIRE(seg && basis && ground && freq && Z, "NULL argument");
    mw_status s = check_common(basis, n_qp);
    if (s != MW_OK) return s;
    MW_REQUIRE(ground->model >= MW_GROUND_PEC && ground->model <= MW_GROUND_SOMM_IMAGE,
               "ground model %d has no image term", ground->model);
    MW_REQUIRE(ldz >= basis->n_basis, "ldz < n_basis");
    bool ek = seg->ek_group != nullptr;
    MW_REQUIRE(!ek || seg->ek_group_img != nullptr, "EK image fill needs ek_group_img labels");
    FillArgs A{};
    A.seg = *seg;
    A.basis = *basis;
    A.ground = *ground;
    A.k = freq->k;
    A.omega = freq->omega;
    A.eps0 = freq->eps0;
    A.mu0 = freq->mu0;
    A.Z = Z;
    A.ldz = ldz;
    A.Z32 = Z32;
    A.ldz32 = ldz32;
    GLParams gl = make_gl(n_qp);
    cudaStream_t st = as_stream(stream);
    if (basis->degree == 1) return ek ? launch_fill<1, true, true>(A, gl, st) : launch_fill<1, true, false>(A, gl, st);
    return ek ? launch_fill<2, true, true>(A, gl, st) : launch_fill<2, true, false>(A, gl, st);
}

extern "C" mw_status mw_fill_z_batch(const mw_segments* seg, const mw_basis* basis, const mw_edges* edges,
                                     int32_t n_k, const double* k_dev, const double* omega_dev, double eps0,
                                     double mu0, int32_t n_qp, int32_t extended_kernel, double ground_z,
                                     int32_t pec_ground, double* table, double* Z, int64_t ldz, int64_t z_stride,
                                     float* Z32, int64_t ldz32, int64_t z32_stride, void* stream) {
    MW_REQUIRE(seg && basis && edges && k_dev && omega_dev && table && Z, "NULL argument");
    MW_REQUIRE(n_k >= 1 && n_k <= 65535, "n_k out of range (%d)", n_k);
    mw_status s = check_common(basis, n_qp);
    if (s != MW_OK) return s;
    MW_REQUIRE(ldz >= basis->n_basis && z_stride >= ldz * basis->n_basis, "bad Z layout");
    MW_REQUIRE(Z32 == nullptr || (ldz32 >= basis->n_basis && z32_stride >= ldz32 * basis->n_basis), "bad Z32 layout");
    const int d = basis->degree;
    const int64_t tstride = edges->table_rows * (d + 1) * (d + 1) * 2;
    GLParams gl = make_gl(n_qp);
    cudaStream_t st = as_stream(stream);
    if (edges->table_rows > 0) {
        ProfileScope ps(PC_TABLE, st);
        const int threads = kTableThreads, rows_per_block = kTableThreads / 32;
        const unsigned bx = (unsigned)((edges->table_rows + rows_per_block - 1) / rows_per_block);
        const bool ek = extended_kernel != 0;
        // the k-independent static part once into every table, then the
        // smooth part per k
#define MW_TBL_B(DD, EE, GRID, MODE)                                                                            \
    same_edge_table_kernel<DD, EE><<<GRID, threads, 0, st>>>(edges->n_edge, edges->n_in_edge, edges->table_off, \
                                                             edges->h, edges->radius, edges->table_rows, 0.0, gl,   \
                                                             table, k_dev, tstride, MODE, n_k)
        for (int mode : {(int)kTableStatic, (int)kTableSmoothAdd}) {
            dim3 grid(bx, mode == kTableStatic ? 1u : (unsigned)n_k);
            if (d == 1) { if (ek) MW_TBL_B(1, true, grid, mode); else MW_TBL_B(1, false, grid, mode); }
            else        { if (ek) MW_TBL_B(2, true, grid, mode); else MW_TBL_B(2, false, grid, mode); }
            MW_CHECK_CUDA(cudaGetLastError());
            count_launch();
        }
#undef MW_TBL_B
    }
    FillArgs A{};
    A.seg = *seg;
    A.basis = *basis;
    A.table = table;
    A.e_n = edges->n_in_edge;
    A.e_off = edges->table_off;
    A.eps0 = eps0;
    A.mu0 = mu0;
    A.Z = Z;
    A.ldz = ldz;
    A.Z32 = Z32;
    A.ldz32 = ldz32;
    A.kb = k_dev;
    A.omegab = omega_dev;
    A.table_stride = tstride;
    A.z_stride = z_stride;
    A.z32_stride = z32_stride;
    A.nbatch = n_k;
    const bool ek = seg->ek_group != nullptr;
    s = (d == 1) ? (ek ? launch_fill<1, false, true>(A, gl, st) : launch_fill<1, false, false>(A, gl, st))
                 : (ek ? launch_fill<2, false, true>(A, gl, st) : launch_fill<2, false, false>(A, gl, st));
    if (s != MW_OK || !pec_ground) return s;
    MW_REQUIRE(!ek || seg->ek_group_img != nullptr, "EK image fill needs ek_group_img labels");
    A.ground.model = MW_GROUND_PEC;
    A.ground.ground_z = ground_z;
    return (d == 1) ? (ek ? launch_fill<1, true, true>(A, gl, st) : launch_fill<1, true, false>(A, gl, st))
                    : (ek ? launch_fill<2, true, true>(A, gl, st) : launch_fill<2, true, false>(A, gl, st));
}
