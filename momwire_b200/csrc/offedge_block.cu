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
// integrated once, by one thread, before the bases are contracted -- the
// arithmetic of the impedance fill (pair_moments.cuh).  Index sets whose 16
// bases touch more than kObSegs segments are taken 8 or 4 bases at a time.
// What bounds it is the FP64 pipe.  Measured on B200, a 1025 x 1311 block at
// degree 2: 4.83 ms with one warp per entry, which evaluated every segment
// pair's samples up to nine times, 0.24 ms now.  Output row-major,
// Z[m * ldz + n], like the reference's (nI, nJ) array.
#include "common.cuh"
#include "ground_weights.cuh"
#include "pair_moments.cuh"

namespace mw {

constexpr int kObMaxQ = 8;
constexpr int kObTile = 16;      // entries of a CTA's block, per side
constexpr int kObSegs = 18;      // segments a side may list
constexpr int kObThreads = 128;  // three CTAs an SM, as the fill

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
    int refl;
    double er, ei, c0r, c0i, c1r, c1i;
    double a_ek;  // > 0: extended kernel on eligible pairs
    double* Z;
    int64_t ldz;
};

template <int D>
struct ObShared {
    static constexpr int NM = D + 1;
    cd J[kObSegs * kObSegs * NM * NM];
    cd T[(NM + D) * kObSegs * (kObTile / 2 + 1)];
    double seg[2][kObSegs * seg_stride<D>(kObMaxQ)];
    double C[2][kObTile * NM * NM];
    int list[2][kObSegs];
    int grp[2][kObSegs];
    int loc[2][kObTile * NM];
    int all[kObTile * NM], fresh[kObTile * NM];
    int count;
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

template <int D, bool REFL, bool EK>
__global__ void __launch_bounds__(kObThreads, 3) offedge_block_kernel(ObArgs A) {
    constexpr int NM = D + 1, NMM = NM * NM;
    extern __shared__ __align__(16) unsigned char ob_smem[];
    ObShared<D>& S = *reinterpret_cast<ObShared<D>*>(ob_smem);
    const int tid = threadIdx.x, nq = A.nq, SD = seg_stride<D>(nq);
    const int n_jt = (A.nJ - 1) / kObTile + 1;
    const int mb = (int)(blockIdx.x / n_jt) * kObTile, nb = (int)(blockIdx.x % n_jt) * kObTile;
    const int m_end = min(A.nI - mb, kObTile) + mb, n_end = min(A.nJ - nb, kObTile) + nb;
    const double om_mu = A.omega * A.mu0, inv_om_eps = 1.0 / (A.omega * A.eps0);
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
            // ---- staging
            for (int e = tid; e < (ns_i + ns_j) * nq; e += kObThreads) {
                const int g = e / nq, q = e - g * nq;
                const bool c = g >= ns_i;
                const int i = c ? g - ns_i : g, s = S.list[c][i];
                const ObSide& X = c ? A.J : A.I;
                stage_node<D>(S.seg[c] + i * SD, nq, q, A.t, A.w, X.seg_l + 3 * (size_t)s, X.seg_r + 3 * (size_t)s,
                              X.tan + 3 * (size_t)s, 0.0, false, 0.0);
                if (q == 0) S.grp[c][i] = EK ? X.group[s] : 0;
            }
            for (int i = tid; i < nm * NMM; i += kObThreads) S.C[0][i] = A.I.polys[(size_t)m0 * NMM + i];
            for (int i = tid; i < nn * NMM; i += kObThreads) S.C[1][i] = A.J.polys[(size_t)n0 * NMM + i];
            __syncthreads();
            // ---- the listed pairs' moments
            for (int p0 = 0; p0 < ns_i * ns_j; p0 += kObThreads) {
                const int pidx = p0 + tid;
                const bool valid = pidx < ns_i * ns_j;
                const int li = valid ? pidx / ns_j : 0, lj = valid ? pidx - li * ns_j : 0;
                const bool ek = EK && S.grp[0][li] >= 0 && S.grp[0][li] == S.grp[1][lj];
                pair_moments_any<D, EK>(S.seg[0] + li * SD, S.seg[1] + lj * SD, nq, A.k, A.a2, ek ? A.a_ek : 0.0,
                                        valid, S.J + (size_t)(valid ? pidx : 0) * NMM);
            }
            __syncthreads();
            // ---- contraction, source side then observer side
            constexpr int cols = kObTile / 2, pitch = cols + 1, plane = kObSegs * pitch;
            cd* TQ = S.T + NM * plane;
            for (int c0 = 0; c0 < nn; c0 += cols) {
                const int nc = min(cols, nn - c0);
                for (int it = tid; it < ns_i * cols; it += kObThreads) {
                    const int la = it / cols, nl = it % cols, ni = c0 + nl;
                    if (nl >= nc) continue;
                    const double* ti = seg_tail<D>(S.seg[0] + la * SD, nq);
                    cd a[NM], q[D];
                    const cd* J0 = S.J + (size_t)la * ns_j * NMM;
                    if constexpr (REFL) {
                        contract_source<D>(J0, S.loc[1] + ni * NM, S.C[1] + ni * NMM,
                                           [&](int lb) {
                                               const double* tj = seg_tail<D>(S.seg[1] + lb * SD, nq);
                                               ComplexWeight w;
                                               cd rv;
                                               refl_dyad(ti + 3, ti, tj + 3, tj, A.er, A.ei, &w.a, &rv);
                                               w.p = cd{A.c0r, A.c0i} + cd{A.c1r, A.c1i} * rv;
                                               return w;
                                           },
                                           a, q);
                    } else {
                        contract_source<D>(J0, S.loc[1] + ni * NM, S.C[1] + ni * NMM,
                                           [&](int lb) {
                                               const double* tj = seg_tail<D>(S.seg[1] + lb * SD, nq);
                                               return RealWeight{ti[0] * tj[0] + ti[1] * tj[1] + ti[2] * tj[2]};
                                           },
                                           a, q);
                    }
#pragma unroll
                    for (int p = 0; p < NM; ++p) S.T[p * plane + la * pitch + nl] = a[p];
#pragma unroll
                    for (int p = 0; p < D; ++p) TQ[p * plane + la * pitch + nl] = q[p];
                }
                __syncthreads();
                for (int pp = tid; pp < nm * cols; pp += kObThreads) {
                    const int mi = pp / cols, nl = pp % cols;  // row-major Z: the column basis fastest
                    if (nl >= nc) continue;
                    cd zA, zP;
                    contract_observer<D>(S.T + nl, TQ + nl, pitch, plane, S.loc[0] + mi * NM, S.C[0] + mi * NMM, &zA,
                                         &zP);
                    double2* out = reinterpret_cast<double2*>(A.Z + 2 * ((int64_t)(m0 + mi) * A.ldz + n0 + c0 + nl));
                    *out = make_double2(-om_mu * zA.im + zP.im * inv_om_eps, om_mu * zA.re - zP.re * inv_om_eps);
                }
                __syncthreads();
            }
        }
    }
}

template <int D, bool REFL, bool EK>
static mw_status ob_launch(const ObArgs& A, cudaStream_t st) {
    auto kern = offedge_block_kernel<D, REFL, EK>;
    MW_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ObShared<D>)));
    const int64_t tiles = ((int64_t)A.nI + kObTile - 1) / kObTile * (((int64_t)A.nJ + kObTile - 1) / kObTile);
    kern<<<(unsigned)tiles, kObThreads, sizeof(ObShared<D>), st>>>(A);
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
    for (int i = 0; i < n_qp; ++i) {
        A.t[i] = gl_t[i];
        A.w[i] = gl_w[i];
    }
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
    MW_REQUIRE((int64_t)A.nI * A.nJ / 8 < (1ll << 31), "block too large");
    const bool ek = a_ek > 0.0 && A.I.group != nullptr && A.J.group != nullptr;
    cudaStream_t st = as_stream(stream);
    ProfileScope ps(PC_FILL, st, 0.0, 16.0 * (double)A.nI * A.nJ);
    const mw_status s = degree == 1 ? ob_pick<1>(A, ek, st) : ob_pick<2>(A, ek, st);
    if (s != MW_OK) return s;
    count_launch();
    return MW_OK;
}
