// mw_selftest_math: the kernels' own elementary functions on given arguments,
// for a test to hold against the correctly rounded values.
//
// mw_selftest_wait_timeout: makes one of the library's bounded device waits
// run out on purpose, with a short spin limit, so that a test can check
// that the wait ends, records MW_ERR_TIMEOUT and leaves the context usable.
// The waits are the production helpers themselves (waits.cuh, tc_common.cuh,
// lu_cluster.cu);
// only the limit is shortened and the awaited event never comes:
//   which = 0: the grid barrier of the complex128 LU panel, two CTAs waiting
//              for three arrivals;
//   which = 1: the mbarrier wait of the tensor-core kernels, one thread
//              waiting on a barrier that nobody arrives at;
//   which = 2: the pivot exchange of the complex128 cluster LU, two CTAs of a
//              cluster waiting for rows that neither sends.
#include "common.cuh"
#include "lu_cluster.cuh"
#include "pair_moments.cuh"
#include "tc_common.cuh"
#include "waits.cuh"

namespace mw {
namespace {

__global__ void grid_wait_selftest_kernel(PanelWs* ws, long long limit) {
    // gridDim.x CTAs can never make gridDim.x + 1 arrivals
    grid_sync_bounded(ws, gridDim.x + 1u, limit);
}

__global__ void mbar_wait_selftest_kernel(int* err, long long limit) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) mbar_wait(&bar, 0, err, limit);
    __syncthreads();
}

__global__ void math_selftest_kernel(int which, int64_t n, const double2* in, double2* out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double2 x = in[i];
    double a, b;
    if (which == 0) {
        a = rsqrt_pos(x.x);
        b = sqrt_pos(x.x, a);
    } else if (which == 1) {
        const cd z = crecip(cd{x.x, x.y});
        a = z.re;
        b = z.im;
    } else if (which == 2) {
        phase_step<kPhaseModeShort>(x.x, &a, &b);
    } else if (which == 3) {
        phase_step<kPhaseModeLong>(x.x, &a, &b);
    } else {
        phase_step<kPhaseModeAny>(x.x, &a, &b);
    }
    out[i] = make_double2(a, b);
}

}  // namespace
}  // namespace mw

extern "C" mw_status mw_selftest_math(int32_t which, int64_t n, const double* in, double* out, void* stream) {
    using namespace mw;
    MW_REQUIRE(which >= 0 && which <= 4, "which must lie in [0, 4], got %d", which);
    MW_REQUIRE(n >= 0 && n < (int64_t(1) << 31) && in && out, "bad arguments");
    if (n == 0) return MW_OK;
    math_selftest_kernel<<<(unsigned)((n + 127) / 128), 128, 0, as_stream(stream)>>>(
        which, n, reinterpret_cast<const double2*>(in), reinterpret_cast<double2*>(out));
    MW_CHECK_CUDA(cudaGetLastError());
    count_launch();
    return MW_OK;
}

extern "C" mw_status mw_selftest_wait_timeout(int32_t which, int64_t spin_limit, void* workspace, void* stream) {
    using namespace mw;
    MW_REQUIRE(which >= 0 && which <= 2, "which must be 0 (grid barrier), 1 (mbarrier) or 2 (exchange), got %d", which);
    MW_REQUIRE(spin_limit >= 256 && spin_limit <= (int64_t(1) << 24),
               "spin_limit must lie in [256, 2^24] (got %lld)", (long long)spin_limit);
    MW_REQUIRE(workspace != nullptr, "NULL workspace");
    cudaStream_t st = as_stream(stream);
    PanelWs* ws = static_cast<PanelWs*>(workspace);
    MW_CHECK_CUDA(cudaMemsetAsync(ws, 0, sizeof(PanelWs), st));
    if (which == 0)
        grid_wait_selftest_kernel<<<2, 32, 0, st>>>(ws, spin_limit);
    else if (which == 1)
        mbar_wait_selftest_kernel<<<1, 32, 0, st>>>(&ws->err, spin_limit);
    else if (mw_status s = zlu_exchange_wait_selftest(&ws->err, (int)spin_limit, st); s != MW_OK)
        return s;
    count_launch();
    MW_CHECK_CUDA(cudaGetLastError());
    int err = 0;
    MW_CHECK_CUDA(cudaMemcpyAsync(&err, &ws->err, sizeof(int), cudaMemcpyDeviceToHost, st));
    MW_CHECK_CUDA(cudaStreamSynchronize(st));
    if (err != 0) {
        static const char* const name[] = {"grid barrier", "mbarrier", "exchange"};
        set_error("bounded %s wait gave up after %lld polls (self-test)", name[which], (long long)spin_limit);
        return err;
    }
    return MW_OK;
}
