// Complex128 LU of a block of columns by one thread-block cluster per matrix
// (lu_cluster.cu).
#pragma once

#include "common.cuh"

namespace mw {

struct ZluArgs {
    cd* A;  // column-major
    int64_t lda, a_stride;
    int n;       // order: rows [j0, n) take part
    int j0, jb;  // columns factored
    int32_t* ipiv;  // 1-based, whole matrix
    int64_t ipiv_stride;
    int32_t* info;  // info[0]: first exact zero pivot (1-based), untouched otherwise
    int64_t info_stride;
    cd* B;  // nrhs further columns of n rows (may be null with nrhs = 0)
    int64_t ldb, b_stride;
    int nrhs;
    int back;  // also B <- U^-1 B (whole matrix, nrhs <= 64)
    // single matrix, or null: n ints of scratch, and 2 jb ints that return
    // the block's row order -- order[i] the row that ends in position j0 + i,
    // order[jb + i] the position row j0 + i went to (-1: it stays within the
    // block)
    int32_t* rid;
    int32_t* order;
};

// The two streams and events of a look-ahead factorisation, one set per host
// thread and device (lu.cu).
struct ZluStreams {
    cudaStream_t trail, critical;
    cudaEvent_t ev_main, ev_handover;
    cudaEvent_t ev_trail[2];
};
mw_status zlu_streams(ZluStreams* out);

// Keeps the host at most DEPTH steps ahead of the one that the device works
// on, so that a cancellation flag polled before each step is seen meanwhile.  Off while the stream is being captured (nothing runs yet).
template <int DEPTH>
class Pace {
  public:
    mw_status start(cudaStream_t st) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        MW_CHECK_CUDA(cudaStreamIsCapturing(st, &cap));
        if (cap != cudaStreamCaptureStatusNone) return MW_OK;
        for (auto& e : ev_) MW_CHECK_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        on_ = true;
        return MW_OK;
    }
    // before step j is enqueued on st
    mw_status step(int64_t j, cudaStream_t st) {
        if (!on_) return MW_OK;
        cudaEvent_t e = ev_[j % DEPTH];
        if (j >= DEPTH) MW_CHECK_CUDA(cudaEventSynchronize(e));
        MW_CHECK_CUDA(cudaEventRecord(e, st));
        return MW_OK;
    }
    ~Pace() {
        for (auto e : ev_)
            if (e) cudaEventDestroy(e);
    }

  private:
    cudaEvent_t ev_[DEPTH] = {};
    bool on_ = false;
};

// Rows one cluster can hold.
int zlu_cluster_max_rows();
// CTAs of the cluster that takes m rows, at most max_ctas (> 0) if they hold
// them.
int zlu_cluster_ctas(int m, int max_ctas);
mw_status zlu_cluster(const ZluArgs& P, int batch, cudaStream_t st, int max_ctas = 0);
// Makes the exchange's wait run out after `limit` polls (selftest.cu).
mw_status zlu_exchange_wait_selftest(int32_t* err, int limit, cudaStream_t st);

// Columns of a block of the blocked factorisation.
constexpr int kZluBlock = 128;
// Whole factorisation of an order within zlu_cluster_max_rows() by blocks;
// rid: n + 4 kZluBlock ints.
mw_status zlu_blocked(int64_t n, cd* A, int64_t lda, int32_t* ipiv, int32_t* info, cd* B, int64_t ldb, int64_t nrhs,
                      int32_t* rid, const volatile int32_t* cancel, cudaStream_t st);
mw_status zlu_upper(int64_t n, const cd* LU, int64_t lda, cd* B, int64_t ldb, int64_t nrhs, cudaStream_t st);

// 1 / z with one reciprocal: z is first scaled by the power of two that
// brings its larger part into [1, 2) (exact), so |z|^2 neither overflows nor
// loses bits.  recip_special: zero, subnormal, infinite and NaN z, which take
// the plain division instead.
__device__ __forceinline__ int recip_exp(cd z) {
    return (int)((__double_as_longlong(fmax(fabs(z.re), fabs(z.im))) >> 52) & 0x7ff);
}
__device__ __forceinline__ bool recip_special(cd z) {
    const int ex = recip_exp(z);
    return ex < 2 || ex > 2044;
}
// (the reciprocal by Newton's iteration from the single-precision one: |z|^2
// is in [1, 8), two steps reach the last bits, and nothing branches)
__device__ __forceinline__ cd recip_fast(cd z) {
    const int ex = min(max(recip_exp(z), 2), 2044);
    const double s = __longlong_as_double((long long)(2046 - ex) << 52);  // 2^(1023 - ex)
    const double x = z.re * s, y = z.im * s;
    const double d = fma(x, x, y * y);
    float r0;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"((float)d));
    double r = (double)r0;
    r = fma(r, fma(-d, r, 1.0), r);
    r = fma(r, fma(-d, r, 1.0), r);
    const double t = s * r;
    return cd{x * t, -(y * t)};
}
__device__ __forceinline__ cd crecip(cd z) { return recip_special(z) ? cdiv(cd{1.0, 0.0}, z) : recip_fast(z); }

}  // namespace mw
