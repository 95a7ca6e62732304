// Static-pivot panel of the complex64 LU (sm_100a).
//
// The mixed-precision path factors Z in complex64 and refines the solution
// against the FP64 Z, so its factors need only be a good preconditioner,
// not LAPACK's partial-pivoting factors.  Pivoting is therefore restricted
// to the rows of each 128 x 128 diagonal block ("static pivoting", Li and
// Demmel 1998: factor with pivots chosen locally, recover accuracy by
// iterative refinement): the panel no longer needs a pivot search over all
// the rows below it, so it has no grid-wide exchange per column.  A panel is
//   sp_diag_kernel  one CTA factors the diagonal block in shared memory,
//                   without interchanges where it can and with partial
//                   pivoting among its own rows where it must, and
//   sp_l21_kernel   every row below is solved against the block's upper
//                   factor, L21 = A21 U11^-1, eight rows to a warp.
// The growth the restriction allows is measured: sp_l21_kernel raises the
// largest |L21| (|re| + |im|) into PanelWs::lmax_bits, and an exact zero
// pivot sets it to +inf.  The caller refactors with full partial pivoting
// when it exceeds its bound, and the FP64 refinement checks the result.
// Galerkin thin-wire impedance matrices are strongly diagonal: partial
// pivoting rarely leaves the diagonal block on them (no interchange at all
// on the planar dipole arrays, a few per cent of columns on Yagis, where
// the local pivot's |L| stays below 3).
#include "common.cuh"
#include "tc_layout.cuh"
#include "waits.cuh"

namespace mw {

constexpr int kSpB = 128;          // diagonal block order
constexpr int kSpDiagThreads = 512;  // 128 rows x 4 groups of 32 columns
constexpr int kSpUStride = kSpB + 2;  // complex elements per shared-memory row of U (16-byte aligned)

namespace {

// (mul_rn, submul_rn: the forms are chosen per position so that the factors
// are, bit for bit, those of 32-column panels and chunks, whatever the width
// used here)

__device__ __forceinline__ cf crcp_sp(cf z) {
    // 1 / z with z scaled by its larger component (|z|^2 neither overflows
    // nor underflows); two reciprocals instead of Smith's three divisions
    const float s = fmaxf(fabsf(z.re), fabsf(z.im));
    if (s < 1e-30f) return cdiv(cone<cf>(), z);
    const float rs = __frcp_rn(s);
    const float a = z.re * rs, b = z.im * rs;
    const float t = rs * __frcp_rn(a * a + b * b);
    return cf{a * t, -b * t};
}

__device__ __forceinline__ float cabs1f(cf z) { return fabsf(z.re) + fabsf(z.im); }

constexpr int kSpLD = kSpB + 2;  // column stride of the staged block (complex; 16-byte aligned columns)
constexpr int kSpPW = 32;        // panel width inside the block
constexpr size_t kSpDiagSmem = sizeof(cf) * (size_t)kSpB * kSpLD;

// U12 = L11^-1 A12 on the rows of the panel at c0 (unit lower L11), one
// thread per later column; `t` is the caller's index among the threads
// that take part (the others pass t < 0).
__device__ __forceinline__ void sp_u12(cf* S, int c0, int jb, int t) {
    const int t0 = c0 + kSpPW;
    const int nt = jb - t0;
    if (t < 0 || t >= nt) return;
    cf* col = S + (t0 + t) * kSpLD + c0;
    cf x[kSpPW];
#pragma unroll
    for (int i = 0; i < kSpPW; ++i) x[i] = col[i];
#pragma unroll
    for (int i = 1; i < kSpPW; ++i) {
        cf v = x[i];
#pragma unroll
        for (int jj = 0; jj < i; ++jj) v = v - S[(c0 + jj) * kSpLD + c0 + i] * x[jj];
        x[i] = v;
    }
#pragma unroll
    for (int i = 0; i < kSpPW; ++i) col[i] = x[i];
}

// A22 -= L21 U12 over rows and columns c0+32 .. jb-1 in 4 x 2 register
// tiles (all threads of the block).
__device__ __forceinline__ void sp_a22(cf* S, int c0, int jb, int tid) {
    const int t0 = c0 + kSpPW;
    const int nt = jb - t0;
    if (nt <= 0) return;
    const int ntr = (nt + 3) / 4, ntc = (nt + 1) / 2;
    for (int tile = tid; tile < ntr * ntc; tile += kSpDiagThreads) {
        const int i0 = t0 + 4 * (tile % ntr), jc = t0 + 2 * (tile / ntr);
        cf acc[4][2];
#pragma unroll
        for (int b2 = 0; b2 < 2; ++b2)
#pragma unroll
            for (int a4 = 0; a4 < 4; ++a4) acc[a4][b2] = S[(jc + b2) * kSpLD + i0 + a4];
#pragma unroll 4
        for (int jj = 0; jj < kSpPW; ++jj) {
            const cf* lcol = S + (c0 + jj) * kSpLD + i0;
            const float4 l01 = *reinterpret_cast<const float4*>(lcol);
            const float4 l23 = *reinterpret_cast<const float4*>(lcol + 2);
            const cf l[4] = {cf{l01.x, l01.y}, cf{l01.z, l01.w}, cf{l23.x, l23.y}, cf{l23.z, l23.w}};
            const cf u0 = S[jc * kSpLD + c0 + jj], u1 = S[(jc + 1) * kSpLD + c0 + jj];
#pragma unroll
            for (int a4 = 0; a4 < 4; ++a4) {
                acc[a4][0] = acc[a4][0] - l[a4] * u0;
                acc[a4][1] = acc[a4][1] - l[a4] * u1;
            }
        }
#pragma unroll
        for (int b2 = 0; b2 < 2; ++b2)
#pragma unroll
            for (int a4 = 0; a4 < 4; ++a4) S[(jc + b2) * kSpLD + i0 + a4] = acc[a4][b2];
    }
}

// The later columns of a factored 32-column panel: U12, then A22 (all
// threads; the caller synchronises after it).
__device__ __forceinline__ void sp_trailing(cf* S, int c0, int jb, int tid) {
    if (jb - (c0 + kSpPW) <= 0) return;
    sp_u12(S, c0, jb, tid);
    __syncthreads();
    sp_a22(S, c0, jb, tid);
}

// Factor A[j0 .. j0+jb) x [j0 .. j0+jb) in place, pivots among these rows
// only: a blocked LU of the block staged in shared memory (column major).
//   first   without interchanges, 16 columns at a time (sp_nopivot): the
//           first warp factors the 16 x 16 sub-block in registers (sp_sub16)
//           while the others still apply the panel before to the rest of the
//           block; then the rows below and the columns right of the sub-block
//           are solved, a thread each.  Two block barriers per panel.  Kept
//           when every pivot is nonzero and every |l| (|re| + |im|) stays
//           within kSpNoPivotBound -- on the strongly diagonal Galerkin
//           blocks partial pivoting would keep the diagonal anyway, and the
//           factors are then the same.
//   else    the block is staged again and factored with partial pivoting
//           among its rows, 32 columns at a time: thread (r, s) holds row r's
//           panel columns 8s .. 8s+7, every thread takes part in every
//           column, rows are interchanged physically (registers for the
//           panel, shared memory for the other columns); two block barriers
//           per column, then the panel's U12 and A22 updates (sp_trailing).
// What bounds it is the chain of 128 columns: a reciprocal, a trip through
// shared memory, a multiplier, an update.  32-column panels whose diagonal
// sub-block one warp factored in shared memory while fifteen waited, then
// rows, U12 and A22 in turn, took 162 us a block on B200; 67 us so, of
// which 7 are the trips from and to global memory, 28 the sub-blocks, 13 the
// rows and columns beside them and the rest the first panels' updates, for
// which one SM's FP32 rate is the bound.
constexpr float kSpNoPivotBound = 2.0f;

constexpr int kSpNW = 16;  // columns of a panel without interchanges

// A 4 x 4 tile, rows i0, i0 + 1, i1, i1 + 1 (even) of columns jc .. jc + 3,
// of A -= L U over inner columns c0 .. c0 + 15, every entry's products in
// column order.
template <bool FIRST>
__device__ __noinline__ void sp_rank16_tile(cf* S, int c0, int i0, int i1, int jc) {
    cf acc[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int a4 = 0; a4 < 4; a4 += 2) {
            const float4 v = *reinterpret_cast<const float4*>(S + (jc + q) * kSpLD + (a4 ? i1 : i0));
            acc[a4][q] = cf{v.x, v.y};
            acc[a4 + 1][q] = cf{v.z, v.w};
        }
#pragma unroll 2
    for (int jj = 0; jj < kSpNW; ++jj) {
        const cf* lcol = S + (c0 + jj) * kSpLD;
        const float4 l01 = *reinterpret_cast<const float4*>(lcol + i0);
        const float4 l23 = *reinterpret_cast<const float4*>(lcol + i1);
        const cf l[4] = {cf{l01.x, l01.y}, cf{l01.z, l01.w}, cf{l23.x, l23.y}, cf{l23.z, l23.w}};
        cf u[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) u[q] = S[(jc + q) * kSpLD + c0 + jj];
#pragma unroll
        for (int a4 = 0; a4 < 4; ++a4)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[a4][q] = submul_rn<FIRST>(acc[a4][q], l[a4], u[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int a4 = 0; a4 < 4; a4 += 2)
            *reinterpret_cast<float4*>(S + (jc + q) * kSpLD + (a4 ? i1 : i0)) =
                make_float4(acc[a4][q].re, acc[a4][q].im, acc[a4 + 1][q].re, acc[a4 + 1][q].im);
}

// The tiles of rows [r0, r1) x columns [q0, q1) (row counts multiples of 8)
// by `nt` threads (this one the t-th); a tile's row pairs lie half the rows
// apart, so that a warp's loads are contiguous.
template <bool FIRST>
__device__ __forceinline__ void sp_rank16(cf* S, int c0, int r0, int r1, int q0, int q1, int t, int nt) {
    const int ntr = (r1 - r0) / 4, ntc = (q1 - q0) / 4;
    for (int tile = t; tile < ntr * ntc; tile += nt) {
        const int i0 = r0 + 2 * (tile % ntr);
        sp_rank16_tile<FIRST>(S, c0, i0, i0 + 2 * ntr, q0 + 4 * (tile / ntr));
    }
}

// All of rows, columns >= t0 but the 16 x 16 sub-block at t0 itself, which
// the first warp keeps up to date.
__device__ __forceinline__ void sp_rank16_rest(cf* S, int c0, int jr, int t, int nt) {
    const int t0 = c0 + kSpNW, t1 = t0 + kSpNW;
    // positions within the 32-column group of c0 take the second form
    if (t0 / kSpPW == c0 / kSpPW) {
        sp_rank16<false>(S, c0, t1, jr, t0, t1, t, nt);
        sp_rank16<false>(S, c0, t0, t1, t1, jr, nt - 1 - t, nt);
    } else {
        sp_rank16<true>(S, c0, t1, jr, t0, t1, t, nt);
        sp_rank16<true>(S, c0, t0, t1, t1, jr, nt - 1 - t, nt);
    }
    sp_rank16<true>(S, c0, t1, jr, t1, jr, t, nt);
}

// The sub-block's registers brought up to date with the panel at cp.
template <bool FIRST>
__device__ __forceinline__ void sp_sub16_update(const cf* S, int c0, int cp, int r, int h, cf (&a)[kSpNW / 2]) {
#pragma unroll 2
    for (int jj = 0; jj < kSpNW; ++jj) {
        const cf l = S[(cp + jj) * kSpLD + c0 + r];
#pragma unroll
        for (int x = 0; x < kSpNW / 2; ++x)
            a[x] = submul_rn<FIRST>(a[x], l, S[(c0 + 2 * x + h) * kSpLD + cp + jj]);
    }
}

// The 16 x 16 sub-block at c0 by one warp: lane (r, h) holds row r's columns
// of parity h in registers, brought up to date with the panel before (cp =
// its first column, < 0: none) on the way in.  Pivot, pivot row and the
// row's own entry pass by shuffles; every lane computes the reciprocal.  The
// loop over column pairs stays rolled, the slots turning by one each time
// (eight turns put them back): unrolled it ran five times slower, waiting for
// instructions that one warp executes once.  True when a pivot is zero or a
// multiplier exceeds the bound.
__device__ __forceinline__ bool sp_sub16(cf* S, int c0, int cp, cf* s_inv) {
    const int lane = threadIdx.x & 31, r = lane & 15, h = lane >> 4;
    constexpr int kX = kSpNW / 2;
    cf a[kX];
#pragma unroll
    for (int x = 0; x < kX; ++x) a[x] = S[(c0 + 2 * x + h) * kSpLD + c0 + r];
    if (cp >= 0) {
        if (cp / kSpPW == c0 / kSpPW)
            sp_sub16_update<false>(S, c0, cp, r, h, a);
        else
            sp_sub16_update<true>(S, c0, cp, r, h, a);
    }
    bool bad = false;
    float lmax = 0.0f;
#pragma unroll 1
    for (int t = 0; t < kX; ++t) {
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            const int j = 2 * t + o;  // held by lanes 16 o + r in slot 0
            const cf piv{__shfl_sync(0xffffffffu, a[0].re, 16 * o + j), __shfl_sync(0xffffffffu, a[0].im, 16 * o + j)};
            const cf v{__shfl_sync(0xffffffffu, a[0].re, 16 * o + r), __shfl_sync(0xffffffffu, a[0].im, 16 * o + r)};
            const float pa = cabs1f(piv);
            bad = bad || !(pa > 0.0f);
            const cf inv = pa > 0.0f ? crcp_sp(piv) : cone<cf>();
            if (lane == j) s_inv[c0 + j] = inv;
            const cf l = mul_rn<true>(v, inv);
            const bool below = r > j;
#pragma unroll
            for (int x = 0; x < kX; ++x) {
                // slot x holds column 2 (t + x) + h, or a finished one
                const cf u{__shfl_sync(0xffffffffu, a[x].re, 16 * h + j),
                           __shfl_sync(0xffffffffu, a[x].im, 16 * h + j)};
                const cf w = submul_rn<false>(a[x], l, u);
                const bool later = x == 0 ? h > o : t + x < kX;
                if (below && later) a[x] = w;
            }
            if (below && h == o) a[0] = l;
            if (below) lmax = fmaxf(lmax, cabs1f(l));
        }
        const cf turn = a[0];
#pragma unroll
        for (int x = 0; x + 1 < kX; ++x) a[x] = a[x + 1];
        a[kX - 1] = turn;
    }
#pragma unroll
    for (int x = 0; x < kX; ++x) S[(c0 + 2 * x + h) * kSpLD + c0 + r] = a[x];
    // NaN-safe: a NaN multiplier fails the comparison
    return bad || !(lmax <= kSpNoPivotBound);
}

// A row below the sub-block at c0 (ROW: a U11 = x, reciprocal pivots in inv)
// or a column right of it (L11 t = x), in place; entry x at p + x * step, and
// the sub-block's entry (i, j) at S[(c0 + j) * kSpLD + c0 + i].  Four entries
// are finished at a time, then leave the others up to date, in registers that
// turn by four.  Returns the largest |re| + |im| of a row's result.
template <bool ROW>
__device__ __forceinline__ float sp_solve16(const cf* S, int c0, cf* p, int step, const cf* inv, bool near) {
    cf a[kSpNW];
    float lmax = 0.0f;
    const cf* D = S + c0 * kSpLD + c0;
#pragma unroll
    for (int x = 0; x < kSpNW; ++x) a[x] = p[x * step];
#pragma unroll 1
    for (int b = 0; b < kSpNW; b += 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (ROW) {
                const cf d = inv[b + j];
                a[j] = near ? mul_rn<true>(a[j], d) : mul_rn<false>(a[j], d);
                lmax = fmaxf(lmax, cabs1f(a[j]));
            }
#pragma unroll
            for (int x = j + 1; x < 4; ++x)
                a[x] = ROW ? submul_rn<false>(a[x], a[j], D[(b + x) * kSpLD + b + j])
                           : submul_rn<false>(a[x], D[(b + j) * kSpLD + b + x], a[j]);
        }
#pragma unroll
        for (int g = 4; g < kSpNW; g += 4) {
            if (b + g >= kSpNW) break;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int x = g; x < g + 4; ++x)
                    a[x] = ROW ? submul_rn<false>(a[x], a[j], D[(b + x) * kSpLD + b + j])
                               : submul_rn<false>(a[x], D[(b + j) * kSpLD + b + x], a[j]);
        }
        cf turn[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) turn[x] = a[x];
#pragma unroll
        for (int x = 0; x + 4 < kSpNW; ++x) a[x] = a[x + 4];
#pragma unroll
        for (int x = 0; x < 4; ++x) a[kSpNW - 4 + x] = turn[x];
    }
#pragma unroll
    for (int x = 0; x < kSpNW; ++x) p[x * step] = a[x];
    return lmax;
}

// The block in S without interchanges (all threads); false when a pivot is
// zero or a multiplier exceeds the bound (S is then half factored).  Rows and
// columns from jb on must hold the identity.  s_bad: two flags, cleared.
__device__ __forceinline__ bool sp_nopivot(cf* S, int jb, cf* s_inv, int* s_bad) {
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (uniform, and known to be)
    const int jr = (jb + kSpNW - 1) / kSpNW * kSpNW;
    for (int c0 = 0; c0 < jr; c0 += kSpNW) {
        const int left = jr - c0;
        if (warp == 0) {
            if (sp_sub16(S, c0, c0 - kSpNW, s_inv)) s_bad[0] = 1;
        } else if (c0 > 0) {
            // once the rest is quicker than the sub-block, the warps that
            // share the first one's scheduler (every fourth) leave it alone
            if (left > 80)
                sp_rank16_rest(S, c0 - kSpNW, jr, tid - 32, kSpDiagThreads - 32);
            else if (warp & 3)
                sp_rank16_rest(S, c0 - kSpNW, jr, (warp - 1 - warp / 4) * 32 + (tid & 31), kSpDiagThreads / 4 * 3);
        }
        __syncthreads();
        if (s_bad[0]) return false;
        const int t0 = c0 + kSpNW;
        if (t0 >= jr) break;
        // L below the sub-block (a row to a thread), U right of it (a column
        // to a thread)
        if (tid < kSpB) {
            const int R = t0 + tid;
            if (R < jr) {
                const float lmax =
                    sp_solve16<true>(S, c0, S + c0 * kSpLD + R, kSpLD, s_inv + c0, R / kSpPW == c0 / kSpPW);
                if (!(lmax <= kSpNoPivotBound)) s_bad[1] = 1;
            }
        } else if (tid < 2 * kSpB) {
            const int q = t0 + tid - kSpB;
            if (q < jr) sp_solve16<false>(S, c0, S + q * kSpLD + c0, 1, nullptr, false);
        }
        __syncthreads();
        if (s_bad[1]) return false;
    }
    return true;
}

__global__ void __launch_bounds__(kSpDiagThreads, 1)
    sp_diag_kernel(cf* __restrict__ A, int64_t lda, int64_t j0, int jb, int32_t* __restrict__ ipiv,
                   int32_t* __restrict__ info, cf* __restrict__ inv_diag, int32_t* __restrict__ perm, PanelWs* ws) {
    extern __shared__ __align__(16) unsigned char sp_diag_smem[];
    cf* S = reinterpret_cast<cf*>(sp_diag_smem);  // S[col * kSpLD + row]
    __shared__ cf s_col[2][kSpB];                 // column c of every row (by column parity)
    __shared__ unsigned long long s_key[2][4];
    __shared__ __align__(16) cf s_u[2][kSpPW];    // the pivot row's panel values
    __shared__ cf s_rc[2][kSpPW];                 // row c's panel values before the interchange
    __shared__ int s_row_at[kSpB];                // original row at each position
    __shared__ cf s_inv[kSpB];
    __shared__ int s_bad[2];
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    for (int base = 0; base < kSpB * kSpB; base += 16 * kSpDiagThreads) {
        cf t[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const int idx = base + u * kSpDiagThreads + tid;
            const int rr = idx % kSpB, col = idx / kSpB;
            // (a partial block's padding: the identity)
            t[u] = (rr < jb && col < jb) ? A[(j0 + rr) + (j0 + col) * lda] : cf{rr == col ? 1.0f : 0.0f, 0.0f};
        }
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const int idx = base + u * kSpDiagThreads + tid;
            S[(idx / kSpB) * kSpLD + idx % kSpB] = t[u];
        }
    }
    if (tid < 2) s_bad[tid] = 0;
    __syncthreads();
    if (sp_nopivot(S, jb, s_inv, s_bad)) {
        for (int c = tid; c < jb; c += kSpDiagThreads) {
            ipiv[j0 + c] = (int32_t)(j0 + c + 1);
            inv_diag[c] = s_inv[c];
            perm[c] = c;
        }
    } else {
        // ---- partial pivoting among the block's rows, from the block as
        // it came
        __syncthreads();
        for (int base = 0; base < kSpB * kSpB; base += 8 * kSpDiagThreads) {
            cf t[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int idx = base + u * kSpDiagThreads + tid;
                const int rr = idx % kSpB, col = idx / kSpB;
                t[u] = (rr < jb && col < jb) ? A[(j0 + rr) + (j0 + col) * lda] : cf{0.0f, 0.0f};
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int idx = base + u * kSpDiagThreads + tid;
                S[(idx / kSpB) * kSpLD + idx % kSpB] = t[u];
            }
        }
        if (tid < kSpB) s_row_at[tid] = tid;
        __syncthreads();
        const int r = tid & (kSpB - 1);
        const int sg = tid >> 7;  // panel column group: columns 8 sg .. 8 sg + 7 of the panel
        const int wig = (tid >> 5) & 3;
        for (int c0 = 0; c0 < jb; c0 += kSpPW) {
            const int nck = (jb - c0) < kSpPW ? (jb - c0) : kSpPW;
            cf pr[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) pr[q] = S[(c0 + 8 * sg + q) * kSpLD + r];
#pragma unroll 1
            for (int cc = 0; cc < nck; ++cc) {
                const int c = c0 + cc, scol = cc >> 3, qc = cc & 7, par = cc & 1;
                if (sg == scol) {
                    cf v = pr[0];
#pragma unroll
                    for (int q = 1; q < 8; ++q)
                        if (q == qc) v = pr[q];
                    s_col[par][r] = v;
                    // largest |re| + |im| among rows c .. jb-1, then the smallest
                    // row (LAPACK's icamax); the low bits carry the row
                    unsigned long long key = 0;
                    if (r >= c && r < jb)
                        key = ((unsigned long long)__float_as_uint(cabs1f(v)) << 32) |
                              ((unsigned long long)(0xFFFFu - (unsigned int)r) << 16) | (unsigned long long)r;
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) {
                        const unsigned long long o = __shfl_xor_sync(0xffffffffu, key, off);
                        key = o > key ? o : key;
                    }
                    if (lane == 0) s_key[par][wig] = key;
                }
                __syncthreads();
                unsigned long long best = s_key[par][0];
#pragma unroll
                for (int w = 1; w < 4; ++w) best = s_key[par][w] > best ? s_key[par][w] : best;
                const int p = (int)(best & 0xFFFFull);
                const bool zero = (best >> 32) == 0ull;
                const cf inv = zero ? cone<cf>() : crcp_sp(s_col[par][p]);
                if (r == p) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) s_u[par][8 * sg + q] = pr[q];
                }
                if (r == c) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) s_rc[par][8 * sg + q] = pr[q];
                }
                // the interchange in the columns outside the panel, one column
                // per thread
                if (p != c && tid < kSpB && (tid < c0 || tid >= c0 + kSpPW)) {
                    cf* col = S + tid * kSpLD;
                    const cf t0 = col[c];
                    col[c] = col[p];
                    col[p] = t0;
                }
                if (tid == 0) {
                    ipiv[j0 + c] = (int32_t)(j0 + p + 1);
                    if (zero) {
                        if (info[0] == 0) info[0] = (int32_t)(j0 + c + 1);
                        atomicExch(&ws->lmax_bits, 0x7f800000u);  // +inf: the block is singular
                    }
                    inv_diag[c] = inv;
                    const int t0 = s_row_at[c];
                    s_row_at[c] = s_row_at[p];
                    s_row_at[p] = t0;
                }
                __syncthreads();  // s_u, s_rc complete
                if (r == c) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) pr[q] = s_u[par][8 * sg + q];
                } else if (r == p) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) pr[q] = s_rc[par][8 * sg + q];
                }
                if (r > c && r < jb && !zero) {
                    // row p now holds row c's old values
                    const cf l = (r == p ? s_col[par][c] : s_col[par][r]) * inv;
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int pc = 8 * sg + q;
                        if (pc == cc) pr[q] = l;
                        else if (pc > cc) pr[q] = pr[q] - l * s_u[par][pc];
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) S[(c0 + 8 * sg + q) * kSpLD + r] = pr[q];
            __syncthreads();
            sp_trailing(S, c0, jb, tid);
            __syncthreads();
        }

        // the block's rows in pivot order: position i holds original row s_row_at[i]
        if (tid < jb) perm[tid] = s_row_at[tid];
    }
    __syncthreads();
#pragma unroll 8
    for (int base = 0; base < kSpB * kSpB; base += kSpDiagThreads) {
        const int idx = base + tid;
        const int rr = idx % kSpB, col = idx / kSpB;
        if (rr < jb && col < jb) A[(j0 + rr) + (j0 + col) * lda] = S[col * kSpLD + rr];
    }
}

// Rows [row0, row0 + jb) of columns [col0, col0 + ncols) rearranged in
// place, row row0 + i taking the old row row0 + perm[i]: one warp per
// column, all of the column's rows read before any is written.  Applies a
// diagonal block's interchanges to the columns beside it in one parallel
// pass (the interchanges never leave the block).
__global__ void __launch_bounds__(256) sp_permute_kernel(cf* __restrict__ A, int64_t lda, int64_t row0, int jb,
                                                         int64_t col0, int64_t ncols,
                                                         const int32_t* __restrict__ perm) {
    const int lane = threadIdx.x & 31;
    const int64_t col = col0 + (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (col >= col0 + ncols) return;
    cf* a = A + col * lda + row0;
    cf v[kSpB / 32];
#pragma unroll
    for (int u = 0; u < kSpB / 32; ++u) {
        const int i = lane + 32 * u;
        v[u] = i < jb ? a[perm[i]] : cf{0.0f, 0.0f};
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kSpB / 32; ++u) {
        const int i = lane + 32 * u;
        if (i < jb) a[i] = v[u];
    }
}

// L21 = A21 U11^-1 for the rows below the diagonal block.  A warp solves
// eight rows by itself, no barrier after U11 is staged: 16 columns at a time,
// eight lanes to a row pair, lane (p, f) holding columns 2f, 2f + 1 of rows
// 2p, 2p + 1.  The columns solved before are removed first (x from the
// warp's strip of shared memory, U11 row-major there), then the chunk is
// solved with x_j passed on by shuffles.  The CTA takes as many rows as
// spread the panel evenly over the chip, up to kSpL21Warps warps' worth; its
// other warps only help to stage U11 (64 KB from L2).  Bound by the FP32
// pipe: 6 operations per update, 128 x 128 / 2 updates a row.  The largest
// |L21| goes to ws->lmax_bits.
// Four warps to 32 rows, handing solved chunks of 32 columns over through
// block barriers, took 61 us a launch on B200 (mean over a 2835-unknown
// matrix); 25 us so.
constexpr int kSpChunk = 16;      // columns at a time
constexpr int kSpWarpRows = 8;    // rows of a warp
constexpr int kSpL21Warps = 11;   // warps of a CTA: the strips of x fill the shared memory beside U11
constexpr int kSpSMs = 148;
constexpr int kSpL21Threads = 32 * kSpL21Warps;
constexpr size_t kSpL21Smem =
    sizeof(cf) * ((size_t)kSpB * kSpUStride + kSpB + (size_t)kSpL21Warps * kSpWarpRows * kSpUStride);

__device__ __forceinline__ void load2(const cf* __restrict__ src, cf (&v)[2]) {
    const float4 w = *reinterpret_cast<const float4*>(src);
    v[0] = cf{w.x, w.y};
    v[1] = cf{w.z, w.w};
}

// Columns [j0, j1) (even) of x removed from the lane's entries; x0 and x1 are
// its two rows in the strip, u its columns of U11.  NEAR: the columns lie in
// the chunk's own group of 32.
template <bool NEAR>
__device__ __forceinline__ void sp_l21_remove(cf (&a)[2][2], const cf* x0, const cf* x1, const cf* u, int j0, int j1) {
#pragma unroll 2
    for (int j = j0; j < j1; j += 2) {
        cf x[2][2], ua[2], ub[2];
        load2(x0 + j, x[0]);
        load2(x1 + j, x[1]);
        load2(u + (size_t)j * kSpUStride, ua);
        load2(u + (size_t)(j + 1) * kSpUStride, ub);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            a[r][0] = submul_rn<NEAR>(a[r][0], x[r][0], ua[0]);
            a[r][1] = submul_rn<false>(a[r][1], x[r][0], ua[1]);
            a[r][0] = submul_rn<NEAR>(a[r][0], x[r][1], ub[0]);
            a[r][1] = submul_rn<false>(a[r][1], x[r][1], ub[1]);
        }
    }
}

__global__ void __launch_bounds__(kSpL21Threads, 1)
    sp_l21_kernel(cf* __restrict__ A, int64_t lda, int64_t j0, int jb, int64_t row_end, int64_t row_pad, int rows_cta,
                  const cf* __restrict__ inv_diag, PanelWs* ws, float* __restrict__ a_hi, float* __restrict__ a_lo) {
    extern __shared__ __align__(16) unsigned char sp_smem[];
    cf* sU = reinterpret_cast<cf*>(sp_smem);       // [kSpB][kSpUStride]
    cf* sX = sU + (size_t)kSpB * kSpUStride;       // [rows of the CTA][kSpUStride]
    cf* sInv = sX + (size_t)kSpL21Warps * kSpWarpRows * kSpUStride;  // [kSpB]
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int p = lane >> 3, f = lane & 7;
    const int64_t base_row = j0 + jb + (int64_t)blockIdx.x * rows_cta;
    const int64_t row = base_row + warp * kSpWarpRows + 2 * p;
    const bool work = warp * kSpWarpRows < rows_cta && base_row + warp * kSpWarpRows < row_pad;
    const int nchunks = (jb + kSpChunk - 1) / kSpChunk;
    cf nxt[2][2];
    auto fetch = [&](int k) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int col = kSpChunk * k + 2 * f + c;
#pragma unroll
            for (int r = 0; r < 2; ++r)
                nxt[r][c] = (work && row + r < row_end && col < jb) ? A[row + r + (j0 + col) * lda] : cf{0.0f, 0.0f};
        }
    };
    fetch(0);
    // staged with eight loads in flight per thread before the stores
    constexpr int kU = 8;
    for (int base = 0; base < kSpB * kSpB; base += kU * kSpL21Threads) {
        cf t[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int idx = base + u * kSpL21Threads + tid;
            const int j = idx % kSpB, col = idx / kSpB;  // coalesced down each column
            t[u] = (idx < kSpB * kSpB && j <= col && col < jb) ? A[(j0 + j) + (j0 + col) * lda] : cf{0.0f, 0.0f};
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int idx = base + u * kSpL21Threads + tid;
            if (idx < kSpB * kSpB) sU[(idx % kSpB) * kSpUStride + idx / kSpB] = t[u];
        }
    }
    for (int j = tid; j < kSpB; j += blockDim.x) sInv[j] = j < jb ? inv_diag[j] : cf{0.0f, 0.0f};
    __syncthreads();
    if (!work) return;
    cf* x0 = sX + (size_t)(warp * kSpWarpRows + 2 * p) * kSpUStride;
    cf* x1 = x0 + kSpUStride;
    const int n_ks = tc_n_ks(jb);
    float lmax = 0.0f;
    for (int k = 0; k < nchunks; ++k) {
        const int c0 = kSpChunk * k, g0 = c0 / kSpPW * kSpPW;
        cf a[2][2] = {{nxt[0][0], nxt[0][1]}, {nxt[1][0], nxt[1][1]}};
        if (k + 1 < nchunks) fetch(k + 1);
        const cf* u = sU + c0 + 2 * f;
        sp_l21_remove<false>(a, x0, x1, u, 0, g0);
        sp_l21_remove<true>(a, x0, x1, u, g0, c0);
#pragma unroll
        for (int j = 0; j < kSpChunk; ++j) {
            cf uj[2], x[2];
            load2(u + (size_t)(c0 + j) * kSpUStride, uj);
            const cf inv = sInv[c0 + j];
            const int src = (lane & ~7) | (j / 2);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const cf t = mul_rn<false>(a[r][j & 1], inv);
                if (f == j / 2) a[r][j & 1] = t;
                x[r] = cf{__shfl_sync(0xffffffffu, t.re, src), __shfl_sync(0xffffffffu, t.im, src)};
                if (2 * f > j) a[r][0] = submul_rn<true>(a[r][0], x[r], uj[0]);
                if (2 * f + 1 > j) a[r][1] = submul_rn<false>(a[r][1], x[r], uj[1]);
            }
        }
        *reinterpret_cast<float4*>(x0 + c0 + 2 * f) = make_float4(a[0][0].re, a[0][0].im, a[0][1].re, a[0][1].im);
        *reinterpret_cast<float4*>(x1 + c0 + 2 * f) = make_float4(a[1][0].re, a[1][0].im, a[1][1].re, a[1][1].im);
        __syncwarp();
        // a packed row: each complex l is the 2 x 2 block [[re, -im], [im, re]]
        // of the trailing updates' operand (rows from j0 + jb, inner dimension
        // jb); rows past the matrix and columns past jb hold zeros, so that
        // the tiles they pad contribute nothing
        const int64_t kap4 = 2 * (c0 + 2 * f);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const cf v0 = a[r][0], v1 = a[r][1];
            lmax = fmaxf(lmax, fmaxf(cabs1f(v0), cabs1f(v1)));
            if (row + r < row_end) {
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    if (c0 + 2 * f + c < jb) A[row + r + (j0 + c0 + 2 * f + c) * lda] = a[r][c];
            }
            if (a_hi != nullptr && kap4 < (int64_t)n_ks * TC_KS) {
                const int64_t rho = 2 * (row + r - (j0 + jb));
                tc_store_a4(a_hi, a_lo, n_ks, rho, kap4, make_float4(v0.re, -v0.im, v1.re, -v1.im));
                tc_store_a4(a_hi, a_lo, n_ks, rho + 1, kap4, make_float4(v0.im, v0.re, v1.im, v1.re));
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, off));
    // NaN-safe: a NaN compares false and raises the bound to +inf
    if (lane == 0) atomicMax(&ws->lmax_bits, (lmax == lmax) ? __float_as_uint(lmax) : 0x7f800000u);
}

// U12 = L11^-1 P A12 for many columns right of the diagonal block: the rows in
// the block's order (perm), the unit lower solve and the packed B operand of
// the update that follows, in one pass.  The mirror image of sp_l21_kernel: a
// warp solves eight columns by itself, 16 rows at a time, eight lanes to a
// column pair; the columns stay in the warp's strip of shared memory from the
// gather to the end.  Every entry takes its products in row order, in the
// form of the leaves it replaces.  Bound by the FP32 pipe, as L21.  Beside the
// row permutation, two leaves of 64 rows with a warp to four columns took
// 100 us for 10,240 columns on B200 (5 + 36 + 59, one after the other before
// each trailing update); 33 us so, 24 for 2,500 columns.
__global__ void __launch_bounds__(kSpL21Threads, 1)
    sp_u12_kernel(const cf* __restrict__ L, int64_t ldl, int jb, cf* __restrict__ X, int64_t ldx, int64_t ncols,
                  int cols_cta, const int32_t* __restrict__ perm, float* __restrict__ b_hi,
                  float* __restrict__ b_lo) {
    extern __shared__ __align__(16) unsigned char sp_smem[];
    cf* sL = reinterpret_cast<cf*>(sp_smem);  // sL[j * kSpUStride + i] = L(i, j)
    cf* sX = sL + (size_t)kSpB * kSpUStride;  // [columns of the CTA][kSpUStride]
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int p = lane >> 3, f = lane & 7;
    const int64_t base_col = (int64_t)blockIdx.x * cols_cta + warp * kSpWarpRows;
    const bool work = warp * kSpWarpRows < cols_cta && base_col < ncols;
    cf* strip = sX + (size_t)warp * kSpWarpRows * kSpUStride;
    if (work) {
#pragma unroll
        for (int h = 0; h < kSpB; h += 32) {
            const int i = h + lane;
            const int src = i < jb ? perm[i] : 0;
            cf t[kSpWarpRows];
#pragma unroll
            for (int c = 0; c < kSpWarpRows; ++c)
                t[c] = (i < jb && base_col + c < ncols) ? X[src + (base_col + c) * ldx] : cf{0.0f, 0.0f};
#pragma unroll
            for (int c = 0; c < kSpWarpRows; ++c) strip[c * kSpUStride + i] = t[c];
        }
    }
    constexpr int kU = 8;
    for (int base = 0; base < kSpB * kSpB; base += kU * kSpL21Threads) {
        cf t[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int idx = base + u * kSpL21Threads + tid;
            const int i = idx % kSpB, j = idx / kSpB;
            t[u] = (idx < kSpB * kSpB && i > j && i < jb) ? L[i + (int64_t)j * ldl] : cf{0.0f, 0.0f};
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int idx = base + u * kSpL21Threads + tid;
            if (idx < kSpB * kSpB) sL[(idx / kSpB) * kSpUStride + idx % kSpB] = t[u];
        }
    }
    __syncthreads();
    if (!work) return;
    cf* x0 = strip + (size_t)(2 * p) * kSpUStride;
    cf* x1 = x0 + kSpUStride;
    const int64_t col = base_col + 2 * p;
    const int n_ks = tc_n_ks(jb);
    const int nchunks = (jb + kSpChunk - 1) / kSpChunk;
    for (int k = 0; k < nchunks; ++k) {
        const int r0 = kSpChunk * k + 2 * f;  // this lane's rows r0, r0 + 1 of columns col, col + 1
        cf a[2][2];
        load2(x0 + r0, a[0]);
        load2(x1 + r0, a[1]);
#pragma unroll 2
        for (int j = 0; j < kSpChunk * k; j += 2) {
            cf x[2][2], la[2], lb[2];
            load2(x0 + j, x[0]);
            load2(x1 + j, x[1]);
            load2(sL + (size_t)j * kSpUStride + r0, la);
            load2(sL + (size_t)(j + 1) * kSpUStride + r0, lb);
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    a[c][r] = submul_rn<false>(a[c][r], la[r], x[c][0]);
                    a[c][r] = submul_rn<false>(a[c][r], lb[r], x[c][1]);
                }
        }
#pragma unroll
        for (int j = 0; j < kSpChunk; ++j) {
            cf lj[2];
            load2(sL + (size_t)(kSpChunk * k + j) * kSpUStride + r0, lj);
            const int src = (lane & ~7) | (j / 2);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const cf v = a[c][j & 1];
                const cf x{__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src)};
#pragma unroll
                for (int r = 0; r < 2; ++r)
                    if (2 * f + r > j) a[c][r] = submul_rn<false>(a[c][r], lj[r], x);
            }
        }
        *reinterpret_cast<float4*>(x0 + r0) = make_float4(a[0][0].re, a[0][0].im, a[0][1].re, a[0][1].im);
        *reinterpret_cast<float4*>(x1 + r0) = make_float4(a[1][0].re, a[1][0].im, a[1][1].re, a[1][1].im);
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            if (col + c >= ncols) continue;
#pragma unroll
            for (int r = 0; r < 2; ++r)
                if (r0 + r < jb) X[r0 + r + (col + c) * ldx] = a[c][r];
            if (b_hi != nullptr && 2 * r0 < n_ks * TC_KS)
                tc_store_b4(b_hi, b_lo, n_ks, col + c, 2 * r0,
                            make_float4(a[c][0].re, a[c][0].im, a[c][1].re, a[c][1].im));
        }
    }
}

}  // namespace

// U12 of a static-pivot panel: L11^-1 P X for the jb <= 128 rows at X, ncols
// columns, L11 at L (unit lower), the block's row order in `perm`; with
// `pack_b` set also as the packed B operand of the update with inner dimension
// jb.
mw_status static_u12_c64(const cf* L, int64_t ldl, int jb, cf* X, int64_t ldx, int64_t ncols, const int32_t* perm,
                         const TcPlanes* pack_b, cudaStream_t st) {
    MW_REQUIRE(jb >= 1 && jb <= kSpB, "static panel width %d outside 1..%d", jb, kSpB);
    if (ncols <= 0) return MW_OK;
    static bool configured = false;
    if (!configured) {
        MW_CHECK_CUDA(cudaFuncSetAttribute(sp_u12_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)kSpL21Smem));
        configured = true;
    }
    const int64_t full = (int64_t)kSpL21Warps * kSpWarpRows * kSpSMs;
    const int64_t ctas = (ncols + full - 1) / full * kSpSMs;
    const int64_t per_cta = (ncols + ctas * kSpWarpRows - 1) / (ctas * kSpWarpRows) * kSpWarpRows;
    ProfileScope ps(PC_TRSM, st, 4.0 * (double)jb * jb * ncols, 16.0 * (double)jb * ncols);
    sp_u12_kernel<<<(unsigned)((ncols + per_cta - 1) / per_cta), kSpL21Threads, kSpL21Smem, st>>>(
        L, ldl, jb, X, ldx, ncols, (int)per_cta, perm, pack_b ? pack_b->b_hi : nullptr,
        pack_b ? pack_b->b_lo : nullptr);
    MW_CHECK_CUDA(cudaGetLastError());
    count_launch();
    return MW_OK;
}

// The panel of columns [j0, j0+jb) (jb <= 128) over rows [j0, n): the
// diagonal block factored with pivots among its own rows, then L21.
// `inv_diag`: 128 complex64 of device scratch for the reciprocal pivots;
// `perm` (128 int32) receives the block's rows in pivot order; with
// `pack_a` set, L21 is also written as the packed A operand (hi / lo
// planes) of the updates that follow.
mw_status static_panel_c64(cf* A, int64_t lda, int64_t n, int64_t j0, int jb, int32_t* ipiv, int32_t* info,
                           PanelWs* ws, cf* inv_diag, int32_t* perm, const TcPlanes* pack_a, cudaStream_t st) {
    MW_REQUIRE(jb >= 1 && jb <= kSpB, "static panel width %d outside 1..%d", jb, kSpB);
    static bool configured = false;
    if (!configured) {
        MW_CHECK_CUDA(cudaFuncSetAttribute(sp_l21_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)kSpL21Smem));
        MW_CHECK_CUDA(cudaFuncSetAttribute(sp_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)kSpDiagSmem));
        configured = true;
    }
    {
        ProfileScope ps(PC_PANEL, st, 8.0 * (double)jb * jb * jb / 3.0, 16.0 * (double)jb * jb);
        sp_diag_kernel<<<1, kSpDiagThreads, kSpDiagSmem, st>>>(A, lda, j0, jb, ipiv, info, inv_diag, perm, ws);
        count_launch();
    }
    {
        const int64_t rows = n - j0 - jb;
        ProfileScope ps(PC_L21, st, 4.0 * (double)rows * jb * jb, 16.0 * (double)rows * jb);
        if (rows > 0) {
            // the packed operand's last tile is written whole (64 rows), and
            // the rows are spread evenly over whole waves of CTAs, one to an SM
            const int64_t pad = (rows + 63) / 64 * 64, full = (int64_t)kSpL21Warps * kSpWarpRows * kSpSMs;
            const int64_t ctas = (pad + full - 1) / full * kSpSMs;
            const int64_t per_cta = (pad + ctas * kSpWarpRows - 1) / (ctas * kSpWarpRows) * kSpWarpRows;
            const unsigned grid = (unsigned)((pad + per_cta - 1) / per_cta);
            sp_l21_kernel<<<grid, kSpL21Threads, kSpL21Smem, st>>>(
                A, lda, j0, jb, n, j0 + jb + pad, (int)per_cta, inv_diag, ws, pack_a ? pack_a->a_hi : nullptr,
                pack_a ? pack_a->a_lo : nullptr);
            count_launch();
        }
    }
    MW_CHECK_CUDA(cudaGetLastError());
    return MW_OK;
}

// Every block's interchanges applied to the columns left of it (the L
// factors of the earlier blocks), all blocks in one launch: blockIdx.y + 1
// is the block, blockIdx.x a chunk of eight columns.  `perm_all` holds the
// n rows in pivot order, block by block.
__global__ void __launch_bounds__(256) sp_left_permute_kernel(cf* __restrict__ A, int64_t lda, int64_t n,
                                                              const int32_t* __restrict__ perm_all) {
    const int64_t j0 = ((int64_t)blockIdx.y + 1) * kSpB;
    const int jb = (int)((n - j0) < kSpB ? (n - j0) : kSpB);
    const int lane = threadIdx.x & 31;
    const int64_t col = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (col >= j0) return;
    const int32_t* perm = perm_all + j0;
    cf* a = A + col * lda + j0;
    cf v[kSpB / 32];
#pragma unroll
    for (int u = 0; u < kSpB / 32; ++u) {
        const int i = lane + 32 * u;
        v[u] = i < jb ? a[perm[i]] : cf{0.0f, 0.0f};
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kSpB / 32; ++u) {
        const int i = lane + 32 * u;
        if (i < jb) a[i] = v[u];
    }
}

void static_left_permute_c64(cf* A, int64_t lda, int64_t n, const int32_t* perm_all, cudaStream_t st) {
    const int64_t nb = (n + kSpB - 1) / kSpB;
    if (nb < 2) return;
    const int64_t last0 = (nb - 1) * kSpB;  // widest left part
    ProfileScope ps(PC_LASWP, st, 0.0, sizeof(cf) * (double)n * n);
    dim3 grid((unsigned)((last0 + 7) / 8), (unsigned)(nb - 1));
    sp_left_permute_kernel<<<grid, 256, 0, st>>>(A, lda, n, perm_all);
    count_launch();
}

// Every block's interchanges applied to columns [0, ncols) of B (n rows, a
// solve's right-hand sides): the whole row permutation of a static-pivot
// factorisation in one parallel pass (the interchanges never leave their
// block).  blockIdx.y is the block, one warp per column.
__global__ void __launch_bounds__(256) sp_block_permute_kernel(cf* __restrict__ B, int64_t ldb, int64_t n,
                                                               int64_t ncols, const int32_t* __restrict__ perm_all) {
    const int64_t j0 = (int64_t)blockIdx.y * kSpB;
    const int jb = (int)((n - j0) < kSpB ? (n - j0) : kSpB);
    const int lane = threadIdx.x & 31;
    const int64_t col = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (col >= ncols) return;
    const int32_t* perm = perm_all + j0;
    cf* a = B + col * ldb + j0;
    cf v[kSpB / 32];
#pragma unroll
    for (int u = 0; u < kSpB / 32; ++u) {
        const int i = lane + 32 * u;
        v[u] = i < jb ? a[perm[i]] : cf{0.0f, 0.0f};
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kSpB / 32; ++u) {
        const int i = lane + 32 * u;
        if (i < jb) a[i] = v[u];
    }
}

void static_rows_permute_c64(cf* B, int64_t ldb, int64_t n, int64_t ncols, const int32_t* perm_all,
                             cudaStream_t st) {
    const int64_t nb = (n + kSpB - 1) / kSpB;
    if (nb < 1 || ncols <= 0) return;
    ProfileScope ps(PC_LASWP, st, 0.0, 2.0 * sizeof(cf) * (double)n * ncols);
    dim3 grid((unsigned)((ncols + 7) / 8), (unsigned)nb);
    sp_block_permute_kernel<<<grid, 256, 0, st>>>(B, ldb, n, ncols, perm_all);
    count_launch();
}

// The block's interchanges applied to columns [col0, col0 + ncols).
void static_permute_c64(cf* A, int64_t lda, int64_t row0, int jb, int64_t col0, int64_t ncols, const int32_t* perm,
                        cudaStream_t st) {
    if (ncols <= 0) return;
    ProfileScope ps(PC_LASWP, st, 0.0, 2.0 * sizeof(cf) * (double)jb * ncols);
    sp_permute_kernel<<<(unsigned)((ncols + 7) / 8), 256, 0, st>>>(A, lda, row0, jb, col0, ncols, perm);
    count_launch();
}

}  // namespace mw
