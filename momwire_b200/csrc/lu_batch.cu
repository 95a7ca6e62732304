// Batched mixed-precision solves for frequency sweeps (sm_100a).
//
// The swept port solve of the reference (bspline.py:4181-4440:
// _swept_batched_z_chunks + _solve_with_kcl_swept_ports, a stacked
// numpy.linalg.solve over the k axis) factorises one small complex matrix per
// frequency.  Here a whole batch of same-order matrices (one structure at
// many frequencies) is factorised together in complex64:
//   panel   one CTA per matrix, the panel (rows j0..n, 8-32 columns) in
//           registers, a row to a thread, or in shared memory where the
//           threads run out;
//   update  the batched tcgen05 3xTF32 update of cgemm_tc.cu over all
//           matrices' tiles in one persistent launch;
// then every matrix is solved and refined in FP64 against its own Z
// (X += LU32 \ (B - Z X)) until the largest relative correction of the whole
// batch is below tol.
#include <cmath>
#include <vector>

#include "common.cuh"
#include "tc_layout.cuh"

namespace mw {

mw_status cgemm_tc_update_batched(int64_t m, int64_t n, int64_t k, int batch, const cf* A, int64_t lda, int64_t sa,
                                  const cf* B, int64_t ldb, int64_t sb, cf* C, int64_t ldc, int64_t sc, void* ws,
                                  size_t ws_bytes, int* err, cudaStream_t st, int max_ctas);
size_t cgemm_tc_workspace_batched(int64_t m, int64_t n, int64_t k, int batch);
void tc_batched_b_planes(void* ws, int64_t m, int64_t n, int64_t k, int batch, float** b_hi, float** b_lo,
                         int64_t* p_stride);

constexpr int kBNB = 16;       // default panel width of the batched factorisation
constexpr int kBNBMax = 32;    // widest panel of the batched factorisation (<= kBOuter)
constexpr int kBOuter = 64;    // block of the batched factorisation: the trailing update's k
constexpr int kBSB = 64;       // block size of the batched triangular solves
constexpr int kBThreads = 256;

__device__ __forceinline__ void amax_merge(double& v, int& i, double v2, int i2) {
    if (v2 > v || (v2 == v && i2 < i)) {
        v = v2;
        i = i2;
    }
}

// One CTA factors the panel rows [j0, n) x columns [j0, j0+jb) of its matrix.
__global__ void __launch_bounds__(kBThreads) panel1_kernel(cf* A, int64_t lda, int64_t stride, int n, int j0, int jb,
                                                           int32_t* ipiv, int32_t* info) {
    extern __shared__ __align__(16) unsigned char p1_smem[];
    cf* slab = reinterpret_cast<cf*>(p1_smem);
    __shared__ double s_v[kBThreads / 32];
    __shared__ int s_i[kBThreads / 32];
    __shared__ int s_p;
    __shared__ double s_pv;
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    A += (int64_t)b * stride;
    ipiv += (int64_t)b * n;
    const int m = n - j0;
    for (int q = tid; q < m * jb; q += blockDim.x) {
        const int i = q % m, x = q / m;
        slab[x * m + i] = A[(j0 + i) + (int64_t)(j0 + x) * lda];
    }
    __syncthreads();
    for (int jj = 0; jj < jb; ++jj) {
        double best = -1.0;
        int bi = 0x7fffffff;
        for (int i = jj + tid; i < m; i += blockDim.x) amax_merge(best, bi, cabs1(slab[jj * m + i]), i);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            amax_merge(best, bi, __shfl_xor_sync(0xffffffffu, best, off), __shfl_xor_sync(0xffffffffu, bi, off));
        if (lane == 0) {
            s_v[warp] = best;
            s_i[warp] = bi;
        }
        __syncthreads();
        if (warp == 0) {
            best = lane < kBThreads / 32 ? s_v[lane] : -1.0;
            bi = lane < kBThreads / 32 ? s_i[lane] : 0x7fffffff;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
                amax_merge(best, bi, __shfl_xor_sync(0xffffffffu, best, off), __shfl_xor_sync(0xffffffffu, bi, off));
            if (lane == 0) {
                s_p = bi < m ? bi : jj;  // nothing but NaN: no interchange
                s_pv = best;
                ipiv[j0 + jj] = j0 + s_p + 1;
            }
        }
        __syncthreads();
        const int p = s_p;
        if (p != jj)
            for (int x = tid; x < jb; x += blockDim.x) {
                const cf t = slab[x * m + jj];
                slab[x * m + jj] = slab[x * m + p];
                slab[x * m + p] = t;
            }
        __syncthreads();
        if (s_pv == 0.0) {
            if (tid == 0 && info[b] == 0) info[b] = j0 + jj + 1;
            continue;
        }
        const cf inv = cdiv(cf{1.f, 0.f}, slab[jj * m + jj]);
        // rows in the threads: scale the multiplier and update its row
        for (int i = jj + 1 + tid; i < m; i += blockDim.x) {
            const cf l = slab[jj * m + i] * inv;
            slab[jj * m + i] = l;
            for (int x = jj + 1; x < jb; ++x) slab[x * m + i] = slab[x * m + i] - l * slab[x * m + jj];
        }
        __syncthreads();
    }
    for (int q = tid; q < m * jb; q += blockDim.x) {
        const int i = q % m, x = q / m;
        A[(j0 + i) + (int64_t)(j0 + x) * lda] = slab[x * m + i];
    }
}

// The panel with a row to a thread, its W columns (>= jb) in registers: slot 0
// is the current column, the slots turn by one per column (W turns put them
// back).  Each warp offers its largest entry with that row; after one barrier
// every thread knows the pivot.  Bound by the chain of jb columns (the pivot
// search over m <= NT rows, a complex reciprocal) and, with one or two CTAs an
// SM, by the slots' updates.  From the slab in shared memory with four
// barriers a column this took 75 us at m = 437, jb = 16, 192 matrices, on
// B200; 30 us so.  Entry for entry the slab's operations (mul_rn and
// submul_rn spell its roundings out).
template <int W, int NT>
__global__ void __launch_bounds__(NT) panel_rows_kernel(cf* A, int64_t lda, int64_t stride, int n, int j0, int jb,
                                                        int32_t* ipiv, int32_t* info) {
    __shared__ __align__(16) cf s_cand[2][NT / 32][W];  // a warp's candidate row
    __shared__ __align__(16) cf s_cur[2][W];            // row jj itself
    __shared__ unsigned s_hi[2][32], s_lo[2][32];
    __shared__ int s_row[2][32];
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0), warps = blockDim.x / 32;
    A += (int64_t)b * stride + j0 + tid + (int64_t)j0 * lda;
    ipiv += (int64_t)b * n;
    const int m = n - j0;
    const bool live = tid < m;
    cf a[W];
#pragma unroll
    for (int x = 0; x < W; ++x) a[x] = (live && x < jb) ? A[x * lda] : cf{0.f, 0.f};
#pragma unroll 1
    for (int jj = 0; jj < W; ++jj) {
        cf last = a[0];
        bool upd = false;
        cf l{0.f, 0.f};
        const cf* u = s_cand[0][0];
        if (jj < jb) {
            const int par = jj & 1;
            // (a NaN is never the pivot; 0 marks rows that are no candidates)
            const double v = cabs1(a[0]);
            const unsigned long long key =
                (live && tid >= jj && v >= 0.0) ? (unsigned long long)__double_as_longlong(v) + 1ull : 0ull;
            const unsigned kh = (unsigned)(key >> 32), kl = (unsigned)key;
            const unsigned mh = __reduce_max_sync(0xffffffffu, kh);
            const unsigned ml = __reduce_max_sync(0xffffffffu, kh == mh ? kl : 0u);
            const int src = __ffs(__ballot_sync(0xffffffffu, kh == mh && kl == ml)) - 1;
            if (lane == src) {
                s_hi[par][warp] = kh;
                s_lo[par][warp] = kl;
                s_row[par][warp] = tid;
#pragma unroll
                for (int x = 0; x < W; ++x) s_cand[par][warp][x] = a[x];
            }
            if (tid == jj) {
#pragma unroll
                for (int x = 0; x < W; ++x) s_cur[par][x] = a[x];
            }
            __syncthreads();
            const unsigned wh = lane < warps ? s_hi[par][lane] : 0u, wl = lane < warps ? s_lo[par][lane] : 0u;
            const unsigned bh = __reduce_max_sync(0xffffffffu, wh);
            const unsigned bl = __reduce_max_sync(0xffffffffu, wh == bh ? wl : 0u);
            const int bw = __ffs(__ballot_sync(0xffffffffu, wh == bh && wl == bl)) - 1;
            const bool none = (bh | bl) == 0u;  // nothing but NaN: no interchange
            const bool zero = bh == 0u && bl == 1u;
            const int p = none ? jj : s_row[par][bw];
            u = none ? s_cur[par] : s_cand[par][bw];
            if (tid == 0) {
                ipiv[j0 + jj] = j0 + p + 1;
                if (zero && info[b] == 0) info[b] = j0 + jj + 1;
            }
            if (p != jj) {
                if (tid == jj) {
#pragma unroll
                    for (int x = 0; x < W; ++x) a[x] = u[x];
                } else if (tid == p) {
#pragma unroll
                    for (int x = 0; x < W; ++x) a[x] = s_cur[par][x];
                }
            }
            last = a[0];
            upd = tid > jj && !zero;
            if (!zero) {
                l = mul_rn<true>(a[0], cdiv(cf{1.f, 0.f}, u[0]));
                if (upd) last = l;
            }
        }
#pragma unroll
        for (int x = 1; x < W; ++x) {
            cf t = a[x];
            if (x + jj < jb) {  // a column of the panel still ahead
                const cf w = submul_rn<false>(t, l, u[x]);
                if (upd) t = w;
            }
            a[x - 1] = t;
        }
        a[W - 1] = last;
    }
    if (live) {
#pragma unroll
        for (int x = 0; x < W; ++x)
            if (x < jb) A[x * lda] = a[x];
    }
}

// The launch of a panel: rows in registers where a thread each is enough, the
// slab in shared memory otherwise.
static void panel_batched(cf* A, int64_t lda, int64_t stride, int n, int j0, int jb, int32_t* ipiv, int32_t* info,
                          int batch, cudaStream_t st) {
    const int m = n - j0, nt = (m + 31) / 32 * 32;
    // (768 threads leave 85 registers a thread and no spill; 1,024 leave 64: 59
    // against 65 us a panel of 16 columns and 513 to 768 rows)
    if (jb <= 8 && m <= 1024)
        panel_rows_kernel<8, 1024><<<batch, nt, 0, st>>>(A, lda, stride, n, j0, jb, ipiv, info);
    else if (jb <= 16 && m <= 512)
        panel_rows_kernel<16, 512><<<batch, nt, 0, st>>>(A, lda, stride, n, j0, jb, ipiv, info);
    else if (jb <= 16 && m <= 768)
        panel_rows_kernel<16, 768><<<batch, nt, 0, st>>>(A, lda, stride, n, j0, jb, ipiv, info);
    else if (jb <= 16 && m <= 1024)
        panel_rows_kernel<16, 1024><<<batch, nt, 0, st>>>(A, lda, stride, n, j0, jb, ipiv, info);
    else if (jb <= 32 && m <= 512)
        panel_rows_kernel<32, 512><<<batch, nt, 0, st>>>(A, lda, stride, n, j0, jb, ipiv, info);
    else
        panel1_kernel<<<batch, kBThreads, (size_t)m * jb * sizeof(cf), st>>>(A, lda, stride, n, j0, jb, ipiv, info);
    count_launch();
}

template <class T>
__global__ void laswp_batched_kernel(T* A, int64_t lda, int64_t stride, int col0, int ncols, const int32_t* ipiv,
                                     int n, int k1, int k2) {
    const int col = col0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= col0 + ncols) return;
    T* a = A + (int64_t)blockIdx.y * stride + (int64_t)col * lda;
    const int32_t* pv = ipiv + (int64_t)blockIdx.y * n;
    for (int i = k1; i < k2; ++i) {
        const int p = pv[i] - 1;
        if (p != i) {
            const T t = a[i];
            a[i] = a[p];
            a[p] = t;
        }
    }
}

// X <- L^-1 X for the unit lower jb x jb (jb <= NB) diagonal block at T, a
// column of X to a thread, in registers; batch on blockIdx.y.  Four rows are
// finished at a time, then leave the rows below up to date, the registers
// turning by four; L is read as broadcasts from shared memory.  The solved rows
// also go out as the packed B operand of the update that follows (inner
// dimension jb; rows past it hold zeros), which saves that its packing pass:
// 1.7 ms of packing against 0.35 here in a sweep of 24 Yagis.  Bound by the
// FP32 pipe (6 operations per entry of L and column).  A warp per column with
// a shuffle per row took 330 us for 64 x 373, 192 matrices, on B200; 74 us so (mean of the
// Yagi sweep's launches), 81 with the packed operand.
// submul_rn's form is that kernel's.
constexpr int kTrsmThreads = 64;
template <int NB>
__global__ void __launch_bounds__(kTrsmThreads) trsm_lower_batched_kernel(const cf* Tm, int64_t ldt, int64_t ts, cf* X,
                                                                          int64_t ldx, int64_t xs, int jb, int ncols,
                                                                          float* b_hi, float* b_lo,
                                                                          int64_t b_pstride) {
    constexpr int kRows = 16;
    __shared__ __align__(16) cf sL[NB][NB];                       // sL[k][i] = L(i, k)
    __shared__ cf sX[kTrsmThreads / 32][32][kRows + 1];           // a warp's columns, kRows rows of them
    Tm += (int64_t)blockIdx.y * ts;
    X += (int64_t)blockIdx.y * xs;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
#pragma unroll 8
    for (int q = tid; q < NB * NB; q += kTrsmThreads) {
        const int i = q % NB, k = q / NB;
        sL[k][i] = (i < jb && k < i) ? Tm[i + (int64_t)k * ldt] : cf{0.f, 0.f};
    }
    const int col0 = blockIdx.x * kTrsmThreads + 32 * warp;
    cf a[NB];
    // coalesced: lanes along the rows, 32 / kRows columns at a time
    constexpr int kPer = 32 / kRows;
    const int lr = lane % kRows, lc = lane / kRows;
#pragma unroll
    for (int h = 0; h < NB; h += kRows) {
#pragma unroll 8
        for (int c = 0; c < 32; c += kPer) {
            const int col = col0 + c + lc;
            sX[warp][c + lc][lr] =
                (h + lr < jb && col < ncols) ? X[h + lr + (int64_t)col * ldx] : cf{0.f, 0.f};
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < kRows; ++r) a[h + r] = sX[warp][lane][r];
        __syncwarp();
    }
    __syncthreads();
#pragma unroll 1
    for (int b = 0; b < NB; b += 4) {
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int x = j + 1; x < 4; ++x) a[x] = submul_rn<true>(a[x], sL[b + j][b + x], a[j]);
#pragma unroll
        for (int g = 4; g < NB; g += 4) {
            if (b + g >= NB) break;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 l01 = *reinterpret_cast<const float4*>(&sL[b + j][b + g]);
                const float4 l23 = *reinterpret_cast<const float4*>(&sL[b + j][b + g + 2]);
                a[g] = submul_rn<true>(a[g], cf{l01.x, l01.y}, a[j]);
                a[g + 1] = submul_rn<true>(a[g + 1], cf{l01.z, l01.w}, a[j]);
                a[g + 2] = submul_rn<true>(a[g + 2], cf{l23.x, l23.y}, a[j]);
                a[g + 3] = submul_rn<true>(a[g + 3], cf{l23.z, l23.w}, a[j]);
            }
        }
        cf turn[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) turn[x] = a[x];
#pragma unroll
        for (int x = 0; x + 4 < NB; ++x) a[x] = a[x + 4];
#pragma unroll
        for (int x = 0; x < 4; ++x) a[NB - 4 + x] = turn[x];
    }
    if (col0 + lane < ncols) {
        const int n_ks = tc_n_ks(jb);
        b_hi += blockIdx.y * b_pstride;
        b_lo += blockIdx.y * b_pstride;
#pragma unroll
        for (int i = 0; i < NB; i += 2)
            if (2 * i < n_ks * TC_KS)
                tc_store_b4(b_hi, b_lo, n_ks, col0 + lane, 2 * i,
                            make_float4(a[i].re, a[i].im, a[i + 1].re, a[i + 1].im));
    }
#pragma unroll
    for (int h = 0; h < NB; h += kRows) {
        __syncwarp();
#pragma unroll
        for (int r = 0; r < kRows; ++r) sX[warp][lane][r] = a[h + r];
        __syncwarp();
#pragma unroll 8
        for (int c = 0; c < 32; c += kPer) {
            const int col = col0 + c + lc;
            if (h + lr < jb && col < ncols) X[h + lr + (int64_t)col * ldx] = sX[warp][c + lc][lr];
        }
    }
}

// m: rows of the update that follows, whose workspace tc_ws takes the packed
// operand.
static void trsm_lower_batched(const cf* Tm, int64_t ldt, int64_t ts, cf* X, int64_t ldx, int64_t xs, int jb, int ncols,
                               int batch, int m, void* tc_ws, cudaStream_t st) {
    float *b_hi, *b_lo;
    int64_t bp;
    tc_batched_b_planes(tc_ws, m, ncols, jb, batch, &b_hi, &b_lo, &bp);
    const dim3 grid((unsigned)((ncols + kTrsmThreads - 1) / kTrsmThreads), (unsigned)batch);
    if (jb <= 16)
        trsm_lower_batched_kernel<16><<<grid, kTrsmThreads, 0, st>>>(Tm, ldt, ts, X, ldx, xs, jb, ncols, b_hi, b_lo, bp);
    else if (jb <= 32)
        trsm_lower_batched_kernel<32><<<grid, kTrsmThreads, 0, st>>>(Tm, ldt, ts, X, ldx, xs, jb, ncols, b_hi, b_lo, bp);
    else
        trsm_lower_batched_kernel<64><<<grid, kTrsmThreads, 0, st>>>(Tm, ldt, ts, X, ldx, xs, jb, ncols, b_hi, b_lo, bp);
    count_launch();
}

// B <- U^-1 L^-1 P B for one matrix and up to C of its right-hand sides per
// CTA (right-hand sides on blockIdx.x, batch on blockIdx.y), the right-hand
// sides in shared memory.  Per 64-row block: a warp per column solves the
// diagonal block (lane = rows r and r + 32), then every row outside it takes
// the 64 products, summed from zero in column order, off at once.  The next
// diagonal block is on its way (cp.async) meanwhile, and each thread's first
// row has half its entries in registers before the block is solved: what
// bounds it is latency, 2 n / 64 times a block's chain of 64 rows and a row's
// loads, then the factors' one pass through HBM (8 n^2 bytes a matrix).  As a
// block solve and a row update per launch it took 460 us (mean of the solves of
// a sweep over 24 Yagis x 64 frequencies) on B200; 225 us so.
constexpr int kGsThreads = 256;
constexpr int kGsAhead = 32;  // entries of a row in registers ahead of time
constexpr size_t kGsSmemMax = 200 * 1024;
template <int C>
__global__ void __launch_bounds__(kGsThreads, 2) getrs_batched_kernel(const cf* LU, int64_t lda, int64_t stride, int n,
                                                                      const int32_t* ipiv, cf* B, int nr, bool wide) {
    extern __shared__ __align__(16) unsigned char gs_smem[];
    cf* sT = reinterpret_cast<cf*>(gs_smem);  // [2][64][64], sT[k * 64 + i] = T(i, k)
    cf* sX = sT + 2 * kBSB * kBSB;            // [C][n]
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int c0 = blockIdx.x * C, nc = min(C, nr - c0);
    LU += (int64_t)blockIdx.y * stride;
    ipiv += (int64_t)blockIdx.y * n;
    B += (int64_t)blockIdx.y * n * nr + (int64_t)c0 * n;
    const int nblk = (n + kBSB - 1) / kBSB;
    auto block_of = [&](int step) { return (step >= nblk ? 2 * nblk - 1 - step : step) * kBSB; };
    auto issue = [&](int step) {
        const int j0 = block_of(step), jb = min(kBSB, n - j0);
        const unsigned dst = (unsigned)__cvta_generic_to_shared(sT + (step & 1) * kBSB * kBSB);
        const cf* src = LU + j0 + (int64_t)j0 * lda;
        for (int q = tid; q < kBSB * kBSB; q += kGsThreads) {
            const int i = q % kBSB, k = q / kBSB;
            if (i >= jb || k >= jb) continue;
            const cf* from = src + i + (int64_t)k * lda;
            if (wide) {
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 8u * q), "l"(from) : "memory");
            } else {  // factors aligned to their floats only
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 8u * q), "l"(&from->re) : "memory");
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 8u * q + 4u), "l"(&from->im)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    issue(0);
    for (int q = tid; q < C * n; q += kGsThreads) sX[q] = q < nc * n ? B[q] : cf{0.f, 0.f};
    __syncthreads();
    if (warp < nc) {
        cf* x = sX + warp * n;
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane, p = i < n ? ipiv[i] - 1 : i;
            unsigned todo = __ballot_sync(0xffffffffu, p != i);
            while (todo) {
                const int r = __ffs(todo) - 1;
                todo &= todo - 1;
                const int q = __shfl_sync(0xffffffffu, p, r);
                if (lane == 0) {
                    const cf t = x[i0 + r];
                    x[i0 + r] = x[q];
                    x[q] = t;
                }
                __syncwarp();
            }
        }
    }
#pragma unroll 1
    for (int step = 0; step < 2 * nblk; ++step) {
        const bool upper = step >= nblk;
        const int j0 = block_of(step), jb = min(kBSB, n - j0);
        // the rows still to be solved
        const int lo = upper ? 0 : j0 + jb, hi = upper ? j0 : n;
        const cf* panel = LU + (int64_t)j0 * lda;
        int i = lo + tid;
        cf t[kGsAhead];
        auto ahead = [&]() {
#pragma unroll
            for (int l = 0; l < kGsAhead; ++l)
                t[l] = (i < hi && l < jb) ? panel[i + (int64_t)l * lda] : cf{0.f, 0.f};
        };
        ahead();
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (step + 1 < 2 * nblk) issue(step + 1);
        if (warp < nc) {
            const cf* T = sT + (step & 1) * kBSB * kBSB;
            cf* x = sX + warp * n + j0;
            cf x0 = lane < jb ? x[lane] : cf{0.f, 0.f};
            cf x1 = lane + 32 < jb ? x[lane + 32] : cf{0.f, 0.f};
            auto pass = [&](cf v, int src) {
                return cf{__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src)};
            };
            if (!upper) {
                const int ka = min(jb, 32);
#pragma unroll 4
                for (int k = 0; k < ka; ++k) {
                    const cf xk = pass(x0, k);
                    const cf w0 = submul_rn<true>(x0, T[k * kBSB + lane], xk);
                    const cf w1 = submul_rn<true>(x1, T[k * kBSB + lane + 32], xk);
                    if (lane > k && lane < jb) x0 = w0;
                    if (lane + 32 < jb) x1 = w1;
                }
#pragma unroll 4
                for (int k = 32; k < jb; ++k) {
                    const cf xk = pass(x1, k - 32);
                    const cf w1 = submul_rn<true>(x1, T[k * kBSB + lane + 32], xk);
                    if (lane + 32 > k && lane + 32 < jb) x1 = w1;
                }
            } else {
                // reciprocals of the diagonal
                const cf one = cone<cf>();
                const cf d0 = lane < jb ? cdiv(one, T[lane * (kBSB + 1)]) : one;
                const cf d1 = lane + 32 < jb ? cdiv(one, T[(lane + 32) * (kBSB + 1)]) : one;
#pragma unroll 4
                for (int k = jb - 1; k >= 32; --k) {
                    if (lane == k - 32) x1 = mul_rn<false>(x1, d1);
                    const cf xk = pass(x1, k - 32);
                    const cf w1 = submul_rn<true>(x1, T[k * kBSB + lane + 32], xk);
                    x0 = submul_rn<true>(x0, T[k * kBSB + lane], xk);
                    if (lane + 32 < k) x1 = w1;
                }
#pragma unroll 4
                for (int k = min(jb, 32) - 1; k >= 0; --k) {
                    if (lane == k) x0 = mul_rn<false>(x0, d0);
                    const cf xk = pass(x0, k);
                    const cf w0 = submul_rn<true>(x0, T[k * kBSB + lane], xk);
                    if (lane < k) x0 = w0;
                }
            }
            if (lane < jb) x[lane] = x0;
            if (lane + 32 < jb) x[lane + 32] = x1;
        }
        __syncthreads();
        while (i < hi) {
            cf acc[C];
#pragma unroll
            for (int c = 0; c < C; ++c) acc[c] = cf{0.f, 0.f};
            auto take = [&](cf v, int l) {
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const cf p = mul_rn<false>(v, sX[c * n + j0 + l]);
                    acc[c] = cf{__fadd_rn(acc[c].re, p.re), __fadd_rn(acc[c].im, p.im)};
                }
            };
#pragma unroll 1
            for (int h = 0; h < kBSB; h += kGsAhead / 2) {
                // t: entries h .. h + 31; the first half is used up and refilled
#pragma unroll
                for (int l = 0; l < kGsAhead / 2; ++l)
                    if (h + l < jb) take(t[l], h + l);
#pragma unroll
                for (int l = 0; l < kGsAhead / 2; ++l) {
                    t[l] = t[l + kGsAhead / 2];
                    const int q = h + kGsAhead + l;
                    t[l + kGsAhead / 2] = q < jb ? panel[i + (int64_t)q * lda] : cf{0.f, 0.f};
                }
            }
#pragma unroll
            for (int c = 0; c < C; ++c) sX[c * n + i] = sX[c * n + i] - acc[c];
            i += kGsThreads;
            if (i < hi) ahead();
        }
    }
    __syncthreads();
    for (int q = tid; q < nc * n; q += kGsThreads) B[q] = sX[q];
}

// R = B - Z X  (complex128; B shared across the batch when bs == 0)
__global__ void resid_batched_kernel(const cd* Z, int64_t ldz, int64_t zs, const cd* X, int64_t ldx, int64_t xs,
                                     const cd* B, int64_t ldb, int64_t bs, cd* R, int64_t ldr, int64_t rs, int n,
                                     int nr) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Z += (int64_t)blockIdx.y * zs;
    X += (int64_t)blockIdx.y * xs;
    B += (int64_t)blockIdx.y * bs;
    R += (int64_t)blockIdx.y * rs;
    for (int c = 0; c < nr; ++c) {
        double ar = 0.0, ai = 0.0;
        const cd* x = X + (int64_t)c * ldx;
        for (int j = 0; j < n; ++j) {
            const cd z = Z[i + (int64_t)j * ldz];
            const cd v = x[j];
            ar = fma(z.re, v.re, ar);
            ar = fma(-z.im, v.im, ar);
            ai = fma(z.re, v.im, ai);
            ai = fma(z.im, v.re, ai);
        }
        const cd bb = B[i + (int64_t)c * ldb];
        R[i + (int64_t)c * ldr] = cd{bb.re - ar, bb.im - ai};
    }
}

// The first residual, R32 = B rounded (X = 0; B with its own leading dimension
// and stride), one launch for the batch.
__global__ void narrow_rhs_batched_kernel(const cd* B, int64_t ldb, int64_t bs, cf* R32, int n, int nr,
                                          int64_t total) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t col = q / n;
        const cd v = B[(col / nr) * bs + (col % nr) * ldb + (q - col * n)];
        R32[q] = cf{(float)v.re, (float)v.im};
    }
}

__global__ void narrow_batched_kernel(const cd* R, cf* R32, int64_t total) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x)
        R32[q] = cf{(float)R[q].re, (float)R[q].im};
}

// X += C; per-matrix max |C| and max |X| (|re| + |im|) into cm / xm.
__global__ void accum_batched_kernel(const cf* C, cd* X, int64_t per, double* cm, double* xm) {
    const int b = blockIdx.y;
    double mc = 0.0, mx = 0.0;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < per; q += (int64_t)gridDim.x * blockDim.x) {
        const cf c = C[b * per + q];
        cd x = X[b * per + q];
        x.re += (double)c.re;
        x.im += (double)c.im;
        X[b * per + q] = x;
        mc = fmax(mc, fabs((double)c.re) + fabs((double)c.im));
        mx = fmax(mx, fabs(x.re) + fabs(x.im));
    }
    for (int off = 16; off > 0; off >>= 1) {
        mc = fmax(mc, __shfl_xor_sync(0xffffffffu, mc, off));
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(reinterpret_cast<unsigned long long*>(cm + b), (unsigned long long)__double_as_longlong(mc));
        atomicMax(reinterpret_cast<unsigned long long*>(xm + b), (unsigned long long)__double_as_longlong(mx));
    }
}

static size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

struct BatchWs {
    void* tc;
    size_t tc_bytes;
    int* tc_err;
    cd* R;
    cf* R32;
    double* norms;  // [2][batch]
};

static size_t batch_ws_bytes(int n, int nrhs, int batch) {
    return al256(cgemm_tc_workspace_batched(n, n, kBOuter, batch)) + 256 + al256((size_t)batch * n * nrhs * 16) +
           al256((size_t)batch * n * nrhs * 8) + al256((size_t)batch * 16);
}

static BatchWs batch_ws(void* ws, int n, int nrhs, int batch) {
    char* w = static_cast<char*>(ws);
    BatchWs b;
    b.tc = w;
    b.tc_bytes = cgemm_tc_workspace_batched(n, n, kBOuter, batch);
    w += al256(b.tc_bytes);
    b.tc_err = reinterpret_cast<int*>(w);
    w += 256;
    b.R = reinterpret_cast<cd*>(w);
    w += al256((size_t)batch * n * nrhs * 16);
    b.R32 = reinterpret_cast<cf*>(w);
    w += al256((size_t)batch * n * nrhs * 8);
    b.norms = reinterpret_cast<double*>(w);
    return b;
}

static mw_status cgetrf_batched(int n, int batch, cf* A, int64_t lda, int64_t stride, int32_t* ipiv, int32_t* info,
                                const BatchWs& w, int pw, cudaStream_t st) {
    const size_t slab_max = (size_t)n * pw * sizeof(cf);
    MW_REQUIRE(slab_max <= 200 * 1024, "order %d too large for a batched panel of %d columns", n, pw);
    static bool attr = false;
    if (!attr) {
        MW_CHECK_CUDA(cudaFuncSetAttribute(panel1_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr = true;
    }
    // Blocked right-looking factorisation: kBOuter-column blocks, each
    // factored as pw-column panels (one CTA per matrix) whose updates stay
    // inside the block; the rest of the matrix then takes the block's row
    // interchanges, one triangular solve and ONE tensor-core update with
    // k = kBOuter (a pw-wide k would underuse the tensor pipe).
    for (int J0 = 0; J0 < n; J0 += kBOuter) {
        const int bw = (n - J0) < kBOuter ? (n - J0) : kBOuter;
        for (int j0 = J0; j0 < J0 + bw; j0 += pw) {
            const int jb = (J0 + bw - j0) < pw ? (J0 + bw - j0) : pw;
            {
                ProfileScope ps(PC_PANEL, st, 4.0 * (double)(n - j0) * jb * jb * batch);
                panel_batched(A, lda, stride, n, j0, jb, ipiv, info, batch, st);
            }
            if (j0 > 0) {
                ProfileScope ps(PC_LASWP, st);
                laswp_batched_kernel<cf><<<dim3((j0 + 127) / 128, batch), 128, 0, st>>>(A, lda, stride, 0, j0, ipiv,
                                                                                        n, j0, j0 + jb);
                count_launch();
            }
            const int inner = J0 + bw - j0 - jb;  // block columns right of this panel
            if (inner > 0) {
                {
                    ProfileScope ps(PC_LASWP, st);
                    laswp_batched_kernel<cf><<<dim3((inner + 127) / 128, batch), 128, 0, st>>>(
                        A, lda, stride, j0 + jb, inner, ipiv, n, j0, j0 + jb);
                }
                cf* A11 = A + j0 + (int64_t)j0 * lda;
                cf* A12 = A + j0 + (int64_t)(j0 + jb) * lda;
                {
                    ProfileScope ps(PC_TRSM, st, 4.0 * (double)jb * jb * inner * batch);
                    trsm_lower_batched(A11, lda, stride, A12, lda, stride, jb, inner, batch, n - j0 - jb, w.tc, st);
                }
                count_launch();
                mw_status s = cgemm_tc_update_batched(n - j0 - jb, inner, jb, batch, A + (j0 + jb) + (int64_t)j0 * lda,
                                                      lda, stride, nullptr, 0, 0,
                                                      A + (j0 + jb) + (int64_t)(j0 + jb) * lda, lda, stride, w.tc,
                                                      w.tc_bytes, w.tc_err, st, 0);
                if (s != MW_OK) return s;
            }
        }
        const int right = n - J0 - bw;
        if (right > 0) {
            {
                ProfileScope ps(PC_LASWP, st);
                laswp_batched_kernel<cf><<<dim3((right + 127) / 128, batch), 128, 0, st>>>(
                    A, lda, stride, J0 + bw, right, ipiv, n, J0, J0 + bw);
            }
            cf* A11 = A + J0 + (int64_t)J0 * lda;
            cf* A12 = A + J0 + (int64_t)(J0 + bw) * lda;
            {
                ProfileScope ps(PC_TRSM, st, 4.0 * (double)bw * bw * right * batch);
                trsm_lower_batched(A11, lda, stride, A12, lda, stride, bw, right, batch, right, w.tc, st);
            }
            count_launch();
            mw_status s = cgemm_tc_update_batched(right, right, bw, batch, A + (J0 + bw) + (int64_t)J0 * lda, lda,
                                                  stride, nullptr, 0, 0, A + (J0 + bw) + (int64_t)(J0 + bw) * lda,
                                                  lda, stride, w.tc, w.tc_bytes, w.tc_err, st, 0);
            if (s != MW_OK) return s;
        }
        MW_CHECK_CUDA(cudaGetLastError());
    }
    return MW_OK;
}

// In-place solve of the batch's B (n x nr each, column-major, ld n).
template <int C>
static mw_status getrs_launch(int n, int nr, int batch, const cf* LU, int64_t lda, int64_t stride, const int32_t* ipiv,
                              cf* B, cudaStream_t st) {
    static bool attr = false;
    if (!attr) {
        MW_CHECK_CUDA(cudaFuncSetAttribute(getrs_batched_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)kGsSmemMax));
        attr = true;
    }
    const size_t smem = sizeof(cf) * ((size_t)2 * kBSB * kBSB + (size_t)C * n);
    getrs_batched_kernel<C><<<dim3((unsigned)((nr + C - 1) / C), (unsigned)batch), kGsThreads, smem, st>>>(
        LU, lda, stride, n, ipiv, B, nr, aligned_to(LU, 8));
    count_launch();
    MW_CHECK_CUDA(cudaGetLastError());
    return MW_OK;
}

static mw_status cgetrs_batched(int n, int nr, int batch, const cf* LU, int64_t lda, int64_t stride,
                                const int32_t* ipiv, cf* B, cudaStream_t st) {
    ProfileScope ps(PC_ZGEMM, st, 8.0 * (double)n * n * nr * batch);  // the whole batched getrs
    // as many right-hand sides a CTA as there are (to 8), where they fit
    // beside the block; n <= 3200 (panels of 8 columns) leaves room for four
    auto fits = [&](int c) { return sizeof(cf) * ((size_t)2 * kBSB * kBSB + (size_t)c * n) <= kGsSmemMax; };
    if (nr > 4 && fits(8)) return getrs_launch<8>(n, nr, batch, LU, lda, stride, ipiv, B, st);
    if (nr > 2 && fits(4)) return getrs_launch<4>(n, nr, batch, LU, lda, stride, ipiv, B, st);
    if (nr > 1 && fits(2)) return getrs_launch<2>(n, nr, batch, LU, lda, stride, ipiv, B, st);
    return getrs_launch<1>(n, nr, batch, LU, lda, stride, ipiv, B, st);
}

}  // namespace mw

using namespace mw;

extern "C" size_t mw_zgesv_mixed_batched_workspace_size(int32_t n, int32_t nrhs, int32_t batch) {
    return batch_ws_bytes(n, nrhs, batch);
}

extern "C" mw_status mw_zgesv_mixed_batched(int32_t n, int32_t nrhs, int32_t batch, int32_t panel_width,
                                            const double* Z, int64_t ldz,
                                            int64_t z_stride, float* Z32, int64_t ldz32, int64_t z32_stride,
                                            int32_t* ipiv, int32_t* info, const double* B, int64_t ldb,
                                            int64_t b_stride, double* X, double tol, int32_t max_iter, void* workspace,
                                            size_t workspace_bytes, int32_t* iterations, double* last_correction,
                                            void* stream) {
    MW_REQUIRE(n >= 1 && nrhs >= 1 && batch >= 1 && batch <= 65535, "bad sizes");
    MW_REQUIRE(Z && Z32 && ipiv && info && B && X && workspace, "NULL argument");
    MW_REQUIRE(ldz >= n && ldz32 >= n && ldb >= n, "leading dimension too small");
    MW_REQUIRE(workspace_bytes >= batch_ws_bytes(n, nrhs, batch), "workspace too small");
    cudaStream_t st = as_stream(stream);
    BatchWs w = batch_ws(workspace, n, nrhs, batch);
    MW_CHECK_CUDA(cudaMemsetAsync(info, 0, sizeof(int32_t) * batch, st));
    MW_CHECK_CUDA(cudaMemsetAsync(w.tc_err, 0, sizeof(int), st));
    cf* Z32c = reinterpret_cast<cf*>(Z32);
    const int pw = panel_width > 0 ? panel_width : kBNB;
    MW_REQUIRE((pw == 8 || pw == 16 || pw == 32) && pw <= kBNBMax, "panel_width must be 8, 16 or 32 (got %d)", pw);
    mw_status s = cgetrf_batched(n, batch, Z32c, ldz32, z32_stride, ipiv, info, w, pw, st);
    if (s != MW_OK) return s;
    const int64_t per = (int64_t)n * nrhs;
    const int64_t tot = per * batch;
    cd* Xc = reinterpret_cast<cd*>(X);
    const cd* Zc = reinterpret_cast<const cd*>(Z);
    const cd* Bc = reinterpret_cast<const cd*>(B);
    // X = 0: the first residual is B itself
    MW_CHECK_CUDA(cudaMemsetAsync(Xc, 0, sizeof(cd) * tot, st));
    std::vector<double> hn(2 * (size_t)batch), prev((size_t)batch, 0.0);
    std::vector<int32_t> hinfo(batch);
    double corr = INFINITY;
    int it = 0;
    const unsigned g1 = (unsigned)((tot + 255) / 256 < 8192 ? (tot + 255) / 256 : 8192);
    for (;; ++it) {
        if (it == 0)
            narrow_rhs_batched_kernel<<<g1, 256, 0, st>>>(Bc, ldb, b_stride, w.R32, n, nrhs, tot);
        else
            narrow_batched_kernel<<<g1, 256, 0, st>>>(w.R, w.R32, tot);
        count_launch();
        s = cgetrs_batched(n, nrhs, batch, Z32c, ldz32, z32_stride, ipiv, w.R32, st);
        if (s != MW_OK) return s;
        MW_CHECK_CUDA(cudaMemsetAsync(w.norms, 0, sizeof(double) * 2 * batch, st));
        {
            ProfileScope ps(PC_REFINE, st, 2.0 * (double)tot, 40.0 * (double)tot);
            dim3 g((unsigned)((per + 255) / 256 < 64 ? (per + 255) / 256 : 64), (unsigned)batch);
            accum_batched_kernel<<<g, 256, 0, st>>>(w.R32, Xc, per, w.norms, w.norms + batch);
            count_launch();
        }
        MW_CHECK_CUDA(cudaMemcpyAsync(hn.data(), w.norms, sizeof(double) * 2 * batch, cudaMemcpyDeviceToHost, st));
        int tce = 0;
        if (it == 0) {
            MW_CHECK_CUDA(cudaMemcpyAsync(hinfo.data(), info, sizeof(int32_t) * batch, cudaMemcpyDeviceToHost, st));
            MW_CHECK_CUDA(cudaMemcpyAsync(&tce, w.tc_err, sizeof(int), cudaMemcpyDeviceToHost, st));
        }
        MW_CHECK_CUDA(cudaStreamSynchronize(st));
        if (it == 0) {
            if (tce != 0) {
                set_error("batched factorisation: a bounded device wait timed out");
                return MW_ERR_TIMEOUT;
            }
            for (int b = 0; b < batch; ++b)
                if (hinfo[b] > 0) {
                    set_error("matrix %d of the batch: exact zero pivot at column %d", b, hinfo[b]);
                    return MW_ERR_SINGULAR;
                }
        }
        // as mw_zgesv_mixed: the relative correction, or once corrections
        // contract (q <= 1/2) the error estimated to remain, r q
        corr = 0.0;
        for (int b = 0; b < batch; ++b) {
            const double xm = hn[batch + b];
            const double r = xm > 0.0 ? hn[b] / xm : (hn[b] > 0.0 ? INFINITY : 0.0);
            double v = r;
            if (it > 0 && prev[b] > 0.0 && r <= 0.5 * prev[b]) v = fmin(r, r * (r / prev[b]));
            prev[b] = r;
            if (!(v <= corr)) corr = v;
        }
        if (corr <= tol || it >= max_iter) break;
        {
            ProfileScope ps(PC_REFINE, st, 8.0 * (double)n * n * nrhs * batch, 16.0 * (double)n * n * batch);
            resid_batched_kernel<<<dim3((n + 127) / 128, batch), 128, 0, st>>>(Zc, ldz, z_stride, Xc, n, per, Bc, ldb,
                                                                               b_stride, w.R, n, per, n, nrhs);
            count_launch();
        }
    }
    if (iterations) *iterations = it;
    if (last_correction) *last_correction = corr;
    if (!(corr <= tol)) {
        set_error("batched refinement did not reach tol %.3g in %d steps (last correction %.3g)", tol, it, corr);
        return MW_ERR_SINGULAR;
    }
    return MW_OK;
}
