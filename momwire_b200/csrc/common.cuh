// Shared device/host helpers for the momwire_b200 kernels (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/momwire_b200.h"

namespace mw {

// ---------------------------------------------------------------- complex
struct cd {
    double re, im;
};
struct cf {
    float re, im;
};

__host__ __device__ __forceinline__ cd cmk(double r, double i) { return cd{r, i}; }
__host__ __device__ __forceinline__ cd operator+(cd a, cd b) { return cd{a.re + b.re, a.im + b.im}; }
__host__ __device__ __forceinline__ cd operator-(cd a, cd b) { return cd{a.re - b.re, a.im - b.im}; }
__host__ __device__ __forceinline__ cd operator*(cd a, cd b) {
    return cd{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
__host__ __device__ __forceinline__ cd operator*(double s, cd a) { return cd{s * a.re, s * a.im}; }
__host__ __device__ __forceinline__ cd cdiv(cd a, cd b) {
    // Smith's algorithm: avoids overflow/underflow of |b|^2.
    if (fabs(b.re) >= fabs(b.im)) {
        double r = b.im / b.re, den = b.re + b.im * r;
        return cd{(a.re + a.im * r) / den, (a.im - a.re * r) / den};
    } else {
        double r = b.re / b.im, den = b.re * r + b.im;
        return cd{(a.re * r + a.im) / den, (a.im * r - a.re) / den};
    }
}
__host__ __device__ __forceinline__ cf operator+(cf a, cf b) { return cf{a.re + b.re, a.im + b.im}; }
__host__ __device__ __forceinline__ cf operator-(cf a, cf b) { return cf{a.re - b.re, a.im - b.im}; }
__host__ __device__ __forceinline__ cf operator*(cf a, cf b) {
    return cf{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
__host__ __device__ __forceinline__ cf cdiv(cf a, cf b) {
    if (fabsf(b.re) >= fabsf(b.im)) {
        float r = b.im / b.re, den = b.re + b.im * r;
        return cf{(a.re + a.im * r) / den, (a.im - a.re * r) / den};
    } else {
        float r = b.re / b.im, den = b.re * r + b.im;
        return cf{(a.re * r + a.im) / den, (a.im * r - a.re) / den};
    }
}
__host__ __device__ __forceinline__ double cabs1(cd z) { return fabs(z.re) + fabs(z.im); }
__host__ __device__ __forceinline__ double cabs1(cf z) { return (double)fabsf(z.re) + (double)fabsf(z.im); }
#ifdef __CUDACC__
// a b and v - a b with their roundings spelled out: a complex product has two
// contracted forms of its imaginary part, and which one the compiler takes
// depends on the code around it.  FIRST rounds the product a.im b.re before
// the fused a.re b.im; otherwise the other way round.  Kernels that must give
// the same bits whatever their tiling use these.
template <bool FIRST>
__device__ __forceinline__ cf mul_rn(cf a, cf b) {
    const float re = __fmaf_rn(a.re, b.re, -__fmul_rn(a.im, b.im));
    const float im = FIRST ? __fmaf_rn(a.re, b.im, __fmul_rn(a.im, b.re))
                           : __fmaf_rn(a.im, b.re, __fmul_rn(a.re, b.im));
    return cf{re, im};
}
template <bool FIRST>
__device__ __forceinline__ cf submul_rn(cf v, cf a, cf b) {
    const cf p = mul_rn<FIRST>(a, b);
    return cf{__fsub_rn(v.re, p.re), __fsub_rn(v.im, p.im)};
}
#endif
template <class T> __host__ __device__ __forceinline__ T cone();
template <> __host__ __device__ __forceinline__ cd cone<cd>() { return cd{1.0, 0.0}; }
template <> __host__ __device__ __forceinline__ cf cone<cf>() { return cf{1.0f, 0.0f}; }

// Principal square root (branch cut on the negative real axis; Im >= 0
// except that -0 imaginary input maps to the lower half, like numpy).
__host__ __device__ __forceinline__ cd csqrt_p(cd z) {
    double x = z.re, y = z.im;
    if (x == 0.0 && y == 0.0) return cd{0.0, y};
    double r = hypot(x, y);
    if (x >= 0.0) {
        double t = sqrt(0.5 * (r + x));
        return cd{t, y / (2.0 * t)};
    } else {
        double t = sqrt(0.5 * (r - x));
        return cd{fabs(y) / (2.0 * t), copysign(t, y)};
    }
}

constexpr double kPi = 3.14159265358979323846;
constexpr double kInv4Pi = 0.079577471545947667884;  // 1/(4 pi)

// ------------------------------------------------------------ error state
void set_error(const char* fmt, ...);
mw_status cuda_status(cudaError_t e, const char* what);

#define MW_CHECK_CUDA(call)                                           \
    do {                                                              \
        cudaError_t _e = (call);                                      \
        if (_e != cudaSuccess) return ::mw::cuda_status(_e, #call);   \
    } while (0)

#define MW_REQUIRE(cond, ...)                                         \
    do {                                                              \
        if (!(cond)) {                                                \
            ::mw::set_error(__VA_ARGS__);                             \
            return MW_ERR_INVALID;                                    \
        }                                                             \
    } while (0)

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Host-side count of kernels this library has launched (mw_launch_count).
void count_launch(int64_t n = 1);

// Optional per-kernel-class timing (mw_profile_*): while enabled, a scope
// records a CUDA event pair around the launches it encloses on `stream` and
// carries the launch's algorithmic flop and byte counts.
enum ProfileClass {
    PC_TABLE = 0,
    PC_FILL = 1,
    PC_FILL_IMAGE = 2,
    PC_PANEL = 3,
    PC_LASWP = 4,
    PC_TRSM = 5,
    PC_ZGEMM = 6,
    PC_CGEMM_TC = 7,
    PC_REFINE = 8,
    PC_MISC = 9,
    PC_SOMM_GRID = 10,
    PC_SOMM_Q = 11,
    PC_FACTOR = 12,  // whole factorisations (wall, enclosing the classes above)
    PC_SOLVE = 13,   // whole triangular solves with many right-hand sides (wall)
    PC_L21 = 14,     // static-pivot panels: the rows below the diagonal block
    PC_COUNT = 15
};

struct ProfileScope {
    ProfileScope(int cls, cudaStream_t st, double flops = 0.0, double bytes = 0.0);
    ~ProfileScope();
    int cls_;
    cudaStream_t st_;
    double flops_, bytes_;
    void* rec_;
};

// Gauss-Legendre nodes/weights on [0,1] for n <= 32, computed on the host
// by Newton iteration on P_n (cached).  Returns pointers to host arrays.
void gauss_legendre01(int n, const double** t, const double** w);

// Whether p lies on a boundary of `bytes` (a power of two; null does).
inline bool aligned_to(const void* p, uintptr_t bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; }

// A complex entry at p, as one access where the caller's array is aligned to
// the pair (`wide`), else as two: the C interface takes arrays of double and
// float at their own alignment.
__device__ __forceinline__ double2 load_pair(const double* p, bool wide) {
    return wide ? *reinterpret_cast<const double2*>(p) : make_double2(p[0], p[1]);
}
__device__ __forceinline__ void store_pair(double* p, bool wide, double x, double y) {
    if (wide) {
        *reinterpret_cast<double2*>(p) = make_double2(x, y);
    } else {
        p[0] = x;
        p[1] = y;
    }
}
__device__ __forceinline__ void store_pair(float* p, bool wide, float x, float y) {
    if (wide) {
        *reinterpret_cast<float2*>(p) = make_float2(x, y);
    } else {
        p[0] = x;
        p[1] = y;
    }
}

// Upper-triangle tile pair of block b: tc(tc+1)/2 <= b < (tc+1)(tc+2)/2,
// tr = b - tc(tc+1)/2 <= tc.
__device__ __forceinline__ void tri_pair(int64_t b, int& tr, int& tc) {
    int64_t c = (int64_t)((sqrt(8.0 * (double)b + 1.0) - 1.0) * 0.5);
    while ((c + 1) * (c + 2) / 2 <= b) ++c;
    while (c * (c + 1) / 2 > b) --c;
    tc = (int)c;
    tr = (int)(b - c * (c + 1) / 2);
}

}  // namespace mw
