// Off-edge Galerkin block sampler (FP64), sm_100a.
//
// The reference's H-matrix and array-block solvers compress the far field
// with adaptive cross approximation: they ask for arbitrary rows, columns
// and blocks Z[I, J] of the impedance matrix between two basis sets, and
// its C++ assembler (bspline_assemble_offedge_block[_refl][_ek],
// _accelerators.cpp:1977-2680) evaluates them by plain n_qp x n_qp
// Gauss quadrature of every wing pair -- no same-edge treatment (the
// sampled blocks are well separated) -- fused with the Galerkin combine:
//   Z[m, n] = j w mu sum_ab w_A(a,b) I_A + sum_ab w_Phi(a,b) I_Phi / (j w eps)
//   I_A   = sum_qr w_q w_r  f_m,a(u_q) f_n,b(u_r)  G(R_qr)
//   I_Phi = sum_qr w_q w_r  f'_m,a(u_q) f'_n,b(u_r) G(R_qr)
// with G = exp(-jkR) / (4 pi R), R = sqrt(|x - y|^2 + a^2), f the wing's
// polynomial in local arc length; w_A = the tangent dot and w_Phi = 1, or
// for the reflection-coefficient image (J side passed pre-mirrored) the
// Fresnel dyad and w_Phi = c0 + c1 rho_v; under the extended kernel G takes
// NEC's coaxial factor on pairs with equal non-negative group labels.
//
// Design: one CTA per 16 x 16 block of entries.  The segments its bases' wings
// touch are listed once per side (neighbouring bases share them: 18 instead
// of 48), staged as quadrature nodes, and every pair of listed segments is
// sampled once, by one thread; the bases are then contracted through their
// values at the nodes, source side first, observer segments by the stripe.
// Index sets whose 16 bases touch more than kObSegs segments are taken 8 or 4
// bases at a time.
// The entries of a far block are what is left when the charges of a basis's
// wings cancel, 1e-2 of the terms and less, so the terms have to be as good as
// they can be: samples at the rounded phase k R with R a square root rounded
// once, bases as node values.  Moments of u^p v^P contracted with the
// polynomials' coefficients, and phases from R as it comes out of the
// reciprocal root, were off by 1.1e-13 of the block's norm (1025 x 1311,
// degree 2) and 1.7e-13 (103 x 150, degree 1); this is off by 3.4e-14 and
// 2.5e-14, as a warp per entry was.
// What bounds it is latency: the samples' dependent FP64 operations and the two
// barriers of a stripe, with twelve warps an SM (issue 45 %, FP64 pipe 36 %).
// Measured on B200, a 1025 x 1311 block at degree 2: 4.83 ms with one warp per
// entry, which evaluated every segment pair's samples up to nine times, 0.25
// ms now (0.24 with moments).  Output row-major, Z[m * ldz + n], like the
// reference's (nI, nJ) array.
#include "common.cuh"
#include "ground_weights.cuh"
#include "pair_moments.cuh"

namespace mw {

constexpr int kObMaxQ = 8;
constexpr int kObTile = 16;      // entries of a CTA's block, per side
constexpr int kObSegs = 18;      // segments a side may list
constexpr int kObThreads = 128;

struct ObSide {
    const int32_t* supp;
    const double* polys;
    const double* seg_l;
    const double* seg_r;
    const double* tan;
    const int32_t* group;
};

struct ObArgs {
    ObSide I, J;
    int nI, nJ, d1;
    double a2, k, omega, eps0, mu0;
    int nq;
    double t[kObMaxQ], w[kObMaxQ];
    double reach;  // times two segments' lengths: bound of a phase step between a pair's samples
    int refl;
    double er, ei, c0r, c0i, c1r, c1i;
    double a_ek;  // > 0: extended kernel on eligible pairs
    double* Z;
    int64_t ldz;
    bool wide;  // Z is aligned to its complex entries
};

// Lists of a CTA, then (in the kernel) what depends on the rule's order.
template <int D>
struct ObShared {
    static constexpr int NM = D + 1;
    int list[2][kObSegs];
    int grp[2][kObSegs];
    int loc[2][kObTile * NM];
    int all[kObTile * NM], fresh[kObTile * NM];
    int count;
};

// A staged segment: nq node positions, then tangent, centre, length.  The
// stride is odd, so that lanes that read different segments fall on different
// banks.
__host__ __device__ constexpr int ob_seg_stride(int nq) { return (nq * 3 + 7) | 1; }

// (shared memory, 16 bytes at a time)
__device__ __forceinline__ cd ld_cd(const cd* p) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    return cd{v.x, v.y};
}
__device__ __forceinline__ void st_cd(cd* p, cd v) { *reinterpret_cast<double2*>(p) = make_double2(v.re, v.im); }

// Dynamic shared memory: sample slots of a pair (one more than nq^2: lanes of
// different pairs on different banks) and of a stripe's source sums.  At the
// usual order 4 three CTAs share an SM (68 KB at most), at 8 two (107).
template <int D, bool REFL>
struct ObSmem {
    static constexpr int NM = D + 1;
    int pairs, rows, slot;  // segment pairs and observer segments of a stripe, samples per pair
    size_t nG, nT, nW, nSeg, nF, bytes;
    __host__ __device__ explicit ObSmem(int nq) {
        pairs = nq <= 4 ? kObThreads : kObThreads / 2;
        rows = nq <= 4 ? 8 : 4;
        slot = nq * nq + 1;
        nG = (size_t)pairs * slot;
        nT = (size_t)2 * nq * rows * kObTile;
        nW = (size_t)pairs * (REFL ? 2 : 1);
        nSeg = (size_t)2 * kObSegs * ob_seg_stride(nq);
        nF = (size_t)2 * kObTile * NM * nq;
        bytes = sizeof(cd) * (nG + nT + nW + nF) + sizeof(double) * nSeg + sizeof(ObShared<D>);
    }
};

// Lists the segments that the `nb` bases from b0 on touch, in order of first
// mention, and the bases' wing slots in that list; returns how many there
// are (the list is complete if at most kObSegs).  Called by the whole block.
template <int D>
__device__ __forceinline__ int ob_list(ObShared<D>& S, int side, const ObSide& X, int b0, int nb) {
    constexpr int NM = D + 1;
    const int tid = threadIdx.x, n = nb * NM;
    __syncthreads();
    if (tid < n) S.all[tid] = X.supp[(size_t)b0 * NM + tid];
    if (tid == 0) S.count = 0;
    __syncthreads();
    int first = -1;  // first mention of this entry's segment
    if (tid < n && S.all[tid] >= 0) {
        first = tid;
        for (int u = tid - 1; u >= 0; --u)
            if (S.all[u] == S.all[tid]) first = u;
    }
    if (tid < n) S.fresh[tid] = first == tid;
    __syncthreads();
    int slot = -1;
    if (first >= 0) {
        slot = 0;
        for (int u = 0; u < first; ++u) slot += S.fresh[u];
        atomicMax(&S.count, slot + 1);
        if (slot < kObSegs) S.list[side][slot] = S.all[tid];
    }
    if (tid < n) S.loc[side][tid] = slot;
    __syncthreads();
    return S.count;
}

// The nq^2 samples 4 pi G(R) of one segment pair, observer node major.  The first
// sample's phase is taken in full and multiplies the others, whose own steps
// are at most |k| (h_i + h_j) (ObArgs::reach: more where the caller's nodes
// leave the segments).
template <bool EK, int NQ, int MODE>
__device__ __forceinline__ void ob_samples(const double* xi, const double* xj, int nq_rt, double k, double a2,
                                           double a_ek, cd* G) {
    constexpr int kMax = NQ > 0 ? NQ : kObMaxQ;
    const int nq = NQ > 0 ? NQ : nq_rt;
    double y[NQ > 0 ? 3 * NQ : 1];  // the source nodes, in registers where their number is known
    if (NQ > 0) {
#pragma unroll
        for (int x = 0; x < 3 * NQ; ++x) y[x] = xj[x];
    }
    auto distance = [&](double x0, double x1, double x2, int r, double* iR) {
        const double* p = NQ > 0 ? y + 3 * r : xj + 3 * r;
        const double dx = x0 - p[0], dy = x1 - p[1], dz = x2 - p[2];
        const double R2 = fma(dz, dz, fma(dy, dy, dx * dx)) + a2;
        *iR = rsqrt_pos(R2);
        return sqrt_pos(R2, *iR);
    };
    double iR, s, c;
    const double kR0 = __dmul_rn(k, distance(xi[0], xi[1], xi[2], 0, &iR));
    sincos(kR0, &s, &c);
    const cd f{c, -s};
#pragma unroll 1
    for (int q = 0; q < nq; ++q) {
        const double x0 = xi[3 * q], x1 = xi[3 * q + 1], x2 = xi[3 * q + 2];
        cd g[kMax];
#pragma unroll
        for (int r = 0; r < kMax; ++r) {
            if (NQ == 0 && r >= nq) break;
            const double R = distance(x0, x1, x2, r, &iR);
            double sx, cx;
            phase_step<MODE>(__dmul_rn(k, R) - kR0, &sx, &cx);
            g[r] = cd{cx * iR, -sx * iR};
            if (EK && a_ek > 0.0) g[r] = g[r] * ek_factor(R, a_ek, k);
            if (NQ == 0) st_cd(G + q * nq + r, f * g[r]);
        }
        if (NQ > 0) {
#pragma unroll
            for (int r = 0; r < kMax; ++r) st_cd(G + q * nq + r, f * g[r]);
        }
    }
}

// The general orders and phase spans, out of line: their registers are not
// the common path's.
template <bool EK, int NQ, int MODE>
__device__ __noinline__ void ob_samples_far(const double* xi, const double* xj, int nq, double k, double a2,
                                            double a_ek, cd* G) {
    ob_samples<EK, NQ, MODE>(xi, xj, nq, k, a2, a_ek, G);
}

template <int D, bool REFL, bool EK>
__global__ void __launch_bounds__(kObThreads, 3) offedge_block_kernel(ObArgs A) {
    constexpr int NM = D + 1;
    extern __shared__ __align__(16) unsigned char ob_smem[];
    const int tid = threadIdx.x, nq = A.nq, SD = ob_seg_stride(nq);
    const ObSmem<D, REFL> lay(nq);
    cd* const sG = reinterpret_cast<cd*>(ob_smem);  // [pair][q][r]
    cd* const sT = sG + lay.nG;                     // [A, charge][q][row of the stripe][column basis]
    cd* const sW = sT + lay.nT;                     // the pairs' weights
    // [side][wing][q][basis]: value and derivative, times w L
    double2* const sF = reinterpret_cast<double2*>(sW + lay.nW);
    double* const sSeg = reinterpret_cast<double*>(sF + lay.nF);
    ObShared<D>& S = *reinterpret_cast<ObShared<D>*>(sSeg + lay.nSeg);
    auto seg = [&](int side, int i) { return sSeg + (side * kObSegs + i) * SD; };
    auto nodal = [&](int side, int b, int q, int n) -> double2& { return sF[((side * NM + b) * nq + q) * kObTile + n]; };
    const int n_jt = (A.nJ - 1) / kObTile + 1;
    const int mb = (int)(blockIdx.x / n_jt) * kObTile, nb = (int)(blockIdx.x % n_jt) * kObTile;
    const int m_end = min(A.nI - mb, kObTile) + mb, n_end = min(A.nJ - nb, kObTile) + nb;
    // (the kernel's 1 / (4 pi) goes last: it would round every sample)
    const double om_mu = A.omega * A.mu0 * kInv4Pi, inv_om_eps = kInv4Pi / (A.omega * A.eps0);
    int mstep = kObTile, nstep = kObTile;
    for (int m0 = mb; m0 < m_end; m0 += mstep) {
        int ns_i = ob_list<D>(S, 0, A.I, m0, min(mstep, m_end - m0));
        while (ns_i > kObSegs) {  // (four bases list at most 4 NM <= 12)
            mstep /= 2;
            ns_i = ob_list<D>(S, 0, A.I, m0, min(mstep, m_end - m0));
        }
        const int nm = min(mstep, m_end - m0);
        for (int n0 = nb; n0 < n_end; n0 += nstep) {
            int ns_j = ob_list<D>(S, 1, A.J, n0, min(nstep, n_end - n0));
            while (ns_j > kObSegs) {
                nstep /= 2;
                ns_j = ob_list<D>(S, 1, A.J, n0, min(nstep, n_end - n0));
            }
            const int nn = min(nstep, n_end - n0);
            // ---- the listed segments' nodes
            for (int e = tid; e < (ns_i + ns_j) * nq; e += kObThreads) {
                const int g = e / nq, q = e - g * nq;
                const int side = g >= ns_i, i = side ? g - ns_i : g, s = S.list[side][i];
                const ObSide& X = side ? A.J : A.I;
                const double *l = X.seg_l + 3 * (size_t)s, *r = X.seg_r + 3 * (size_t)s;
                double* o = seg(side, i);
                const double t = A.t[q];
#pragma unroll
                for (int c = 0; c < 3; ++c) o[3 * q + c] = (1.0 - t) * l[c] + t * r[c];
                if (q != 0) continue;
                o += 3 * nq;
                const double dx = r[0] - l[0], dy = r[1] - l[1], dz = r[2] - l[2];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    o[c] = X.tan[3 * (size_t)s + c];
                    o[3 + c] = 0.5 * (l[c] + r[c]);
                }
                o[6] = sqrt(dx * dx + dy * dy + dz * dz);
                S.grp[side][i] = EK ? X.group[s] : 0;
            }
            __syncthreads();
            // ---- the bases' values and derivatives at the nodes
            for (int e = tid; e < (nm + nn) * NM * nq; e += kObThreads) {
                const int side = e >= nm * NM * nq, x = side ? e - nm * NM * nq : e;
                const int w = x / nq, q = x - w * nq, l = S.loc[side][w];
                if (l < 0) continue;
                const double* c = (side ? A.J.polys + (size_t)n0 * NM * NM : A.I.polys + (size_t)m0 * NM * NM) + w * NM;
                const double L = seg(side, l)[3 * nq + 6], u = A.t[q] * L, wl = A.w[q] * L;
                double v = c[D], dv = D * c[D];
#pragma unroll
                for (int p = D - 1; p >= 0; --p) v = fma(v, u, c[p]);
#pragma unroll
                for (int p = D - 1; p >= 1; --p) dv = fma(dv, u, p * c[p]);
                nodal(side, w % NM, q, w / NM) = make_double2(wl * v, wl * dv);
            }
            cd zA[2] = {}, zP[2] = {};  // entries tid and tid + kObThreads of the block
            const int rows = max(1, min(lay.rows, lay.pairs / max(ns_j, 1)));
            for (int g0 = 0; g0 < ns_i; g0 += rows) {
                const int nr = min(rows, ns_i - g0);
                // ---- a stripe's samples and weights, a pair to a thread
                const bool valid = tid < nr * ns_j;
                const int li = valid ? g0 + tid / ns_j : 0, lj = valid ? tid % ns_j : 0;
                const double *xi = seg(0, li), *xj = seg(1, lj), *ti = xi + 3 * nq, *tj = xj + 3 * nq;
                const double span = valid ? A.reach * (ti[6] + tj[6]) : 0.0;
                const bool brief = __all_sync(0xffffffffu, span <= kPhaseShort);
                const bool series = __all_sync(0xffffffffu, span <= kPhaseLong);
                if (valid) {
                    const bool ek = EK && S.grp[0][li] >= 0 && S.grp[0][li] == S.grp[1][lj];
                    const double a_ek = ek ? A.a_ek : 0.0;
                    cd* G = sG + (size_t)tid * lay.slot;
                    if (nq == 4 && brief)
                        ob_samples<EK, 4, kPhaseModeShort>(xi, xj, 4, A.k, A.a2, a_ek, G);
                    else if (nq == 4 && series)
                        ob_samples_far<EK, 4, kPhaseModeLong>(xi, xj, 4, A.k, A.a2, a_ek, G);
                    else
                        ob_samples_far<EK, 0, kPhaseModeAny>(xi, xj, nq, A.k, A.a2, a_ek, G);
                    if constexpr (REFL) {
                        cd wa, rv;
                        refl_dyad(ti + 3, ti, tj + 3, tj, A.er, A.ei, &wa, &rv);
                        sW[2 * tid] = wa;
                        sW[2 * tid + 1] = cd{A.c0r, A.c0i} + cd{A.c1r, A.c1i} * rv;
                    } else {
                        sW[tid].re = ti[0] * tj[0] + ti[1] * tj[1] + ti[2] * tj[2];
                    }
                }
                __syncthreads();
                // ---- source side: per observer node and column basis
                for (int it = tid; it < nr * nq * kObTile; it += kObThreads) {
                    const int n = it % kObTile, q = it / kObTile % nq, row = it / (kObTile * nq);
                    if (n >= nn) continue;
                    // (node by node over the wings: their charges, of opposite
                    // signs, then never add up to more than one wing's term)
                    int pair[NM];
                    cd s[NM], t[NM];
#pragma unroll
                    for (int b = 0; b < NM; ++b) {
                        const int lb = S.loc[1][n * NM + b];
                        pair[b] = lb < 0 ? -1 : row * ns_j + lb;
                        s[b] = t[b] = cd{0.0, 0.0};
                    }
#pragma unroll 4
                    for (int r = 0; r < nq; ++r)
#pragma unroll
                        for (int b = 0; b < NM; ++b) {
                            if (pair[b] < 0) continue;
                            const cd g = ld_cd(sG + (size_t)pair[b] * lay.slot + q * nq + r);
                            const double2 f = nodal(1, b, r, n);
                            cd& c = t[REFL ? b : 0];
                            s[b].re = fma(f.x, g.re, s[b].re);
                            s[b].im = fma(f.x, g.im, s[b].im);
                            c.re = fma(f.y, g.re, c.re);
                            c.im = fma(f.y, g.im, c.im);
                        }
                    cd a{0.0, 0.0}, p = REFL ? cd{0.0, 0.0} : t[0];
#pragma unroll
                    for (int b = 0; b < NM; ++b) {
                        if (pair[b] < 0) continue;
                        if constexpr (REFL) {
                            a = a + sW[2 * pair[b]] * s[b];
                            p = p + sW[2 * pair[b] + 1] * t[b];
                        } else {
                            a = a + sW[pair[b]].re * s[b];
                        }
                    }
                    cd* T = sT + (q * lay.rows + row) * kObTile + n;
                    st_cd(T, a);
                    st_cd(T + nq * lay.rows * kObTile, p);
                }
                __syncthreads();
                // ---- observer side: the entries' share of this stripe
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int e = tid + h * kObThreads, m = e / kObTile, n = e % kObTile;
                    if (m >= nm || n >= nn) continue;
#pragma unroll
                    for (int a = 0; a < NM; ++a) {
                        const int row = S.loc[0][m * NM + a] - g0;
                        if (row < 0 || row >= nr) continue;
#pragma unroll 4
                        for (int q = 0; q < nq; ++q) {
                            const cd* T = sT + (q * lay.rows + row) * kObTile + n;
                            const cd t = ld_cd(T), p = ld_cd(T + nq * lay.rows * kObTile);
                            const double2 f = nodal(0, a, q, m);
                            zA[h].re = fma(f.x, t.re, zA[h].re);
                            zA[h].im = fma(f.x, t.im, zA[h].im);
                            zP[h].re = fma(f.y, p.re, zP[h].re);
                            zP[h].im = fma(f.y, p.im, zP[h].im);
                        }
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int e = tid + h * kObThreads, m = e / kObTile, n = e % kObTile;  // the column basis fastest
                if (m >= nm || n >= nn) continue;
                store_pair(A.Z + 2 * ((int64_t)(m0 + m) * A.ldz + n0 + n), A.wide,
                           -om_mu * zA[h].im + zP[h].im * inv_om_eps, om_mu * zA[h].re - zP[h].re * inv_om_eps);
            }
        }
    }
}

template <int D, bool REFL, bool EK>
static mw_status ob_launch(const ObArgs& A, cudaStream_t st) {
    auto kern = offedge_block_kernel<D, REFL, EK>;
    const size_t smem = ObSmem<D, REFL>(A.nq).bytes;
    MW_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int64_t tiles = ((int64_t)A.nI + kObTile - 1) / kObTile * (((int64_t)A.nJ + kObTile - 1) / kObTile);
    kern<<<(unsigned)tiles, kObThreads, smem, st>>>(A);
    MW_CHECK_CUDA(cudaGetLastError());
    return MW_OK;
}

template <int D>
static mw_status ob_pick(const ObArgs& A, bool ek, cudaStream_t st) {
    if (A.refl) return ek ? ob_launch<D, true, true>(A, st) : ob_launch<D, true, false>(A, st);
    return ek ? ob_launch<D, false, true>(A, st) : ob_launch<D, false, false>(A, st);
}

}  // namespace mw

using namespace mw;

extern "C" mw_status mw_offedge_block(int32_t degree, const mw_block_side* I, const mw_block_side* J,
                                      double a_squared, const mw_freq* freq, int32_t n_qp, const double* gl_t,
                                      const double* gl_w, const mw_block_refl* refl, double a_ek, double* Z,
                                      int64_t ldz, void* stream) {
    MW_REQUIRE(I && J && freq && gl_t && gl_w, "NULL argument");
    MW_REQUIRE(degree == 1 || degree == 2, "max_d must be 1 or 2, got %d", degree);
    MW_REQUIRE(n_qp >= 1 && n_qp <= kObMaxQ, "n_qp > %d not supported (got %d)", kObMaxQ, n_qp);
    MW_REQUIRE(I->n_basis >= 0 && J->n_basis >= 0, "negative basis count");
    MW_REQUIRE(ldz >= (J->n_basis > 0 ? J->n_basis : 1), "ldz smaller than the J-side basis count");
    if (I->n_basis == 0 || J->n_basis == 0) return MW_OK;
    MW_REQUIRE(Z && I->supp && I->polys && I->seg_l && I->seg_r && I->tangent && J->supp && J->polys && J->seg_l &&
                   J->seg_r && J->tangent,
               "NULL side table");
    MW_REQUIRE(!(a_ek > 0.0) || (I->ek_group && J->ek_group), "the extended kernel needs both sides' group labels");
    ObArgs A{};
    A.I = ObSide{I->supp, I->polys, I->seg_l, I->seg_r, I->tangent, I->ek_group};
    A.J = ObSide{J->supp, J->polys, J->seg_l, J->seg_r, J->tangent, J->ek_group};
    A.nI = I->n_basis;
    A.nJ = J->n_basis;
    A.d1 = degree + 1;
    A.a2 = a_squared;
    A.k = freq->k;
    A.omega = freq->omega;
    A.eps0 = freq->eps0;
    A.mu0 = freq->mu0;
    A.nq = n_qp;
    double spread = 1.0;  // of the nodes, in segment lengths (the caller's rule need not stay on [0, 1])
    for (int i = 0; i < n_qp; ++i) {
        A.t[i] = gl_t[i];
        A.w[i] = gl_w[i];
        spread = fmax(spread, fabs(gl_t[i] - gl_t[0]));
    }
    A.reach = fabs(A.k) * spread;
    A.refl = refl != nullptr;
    if (refl) {
        A.er = refl->eps_re;
        A.ei = refl->eps_im;
        A.c0r = refl->phi_c0_re;
        A.c0i = refl->phi_c0_im;
        A.c1r = refl->phi_c1_re;
        A.c1i = refl->phi_c1_im;
    }
    A.a_ek = a_ek;
    A.Z = Z;
    A.ldz = ldz;
    A.wide = aligned_to(Z, 16);
    MW_REQUIRE((int64_t)A.nI * A.nJ / 8 < (1ll << 31), "block too large");
    const bool ek = a_ek > 0.0 && A.I.group != nullptr && A.J.group != nullptr;
    cudaStream_t st = as_stream(stream);
    ProfileScope ps(PC_FILL, st, 0.0, 16.0 * (double)A.nI * A.nJ);
    const mw_status s = degree == 1 ? ob_pick<1>(A, ek, st) : ob_pick<2>(A, ek, st);
    if (s != MW_OK) return s;
    count_launch();
    return MW_OK;
}
