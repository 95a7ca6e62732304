// Arguments of the impedance fill's kernels (fill.cu, fill_rows.cu).
#pragma once

#include "common.cuh"

namespace mw {

struct GLParams {
    int nq;
    double t[8];    // nodes on [0,1]
    double w[8];    // weights on [0,1]
    double x20[20]; // 20-point nodes on [-1,1] (static panels)
    double w20[20];
};

struct FillArgs {
    mw_segments seg;
    mw_basis basis;
    const double* table;
    const int32_t* e_n;        // edges: segments per edge
    const int64_t* e_off;      // edges: table offsets
    mw_ground ground;
    double k, omega, eps0, mu0;
    double* Z;
    int64_t ldz;
    float* Z32;
    int64_t ldz32;
    // frequency batch (blockIdx.z): per-entry k / omega (NULL = the scalars
    // above) and the strides between consecutive tables and matrices
    const double* kb;
    const double* omegab;
    int64_t table_stride, z_stride, z32_stride;
    int nbatch;
    bool wide;  // table, Z and Z32 are aligned to their complex entries
};

// Z and its complex64 copy for one frequency, each sum in a fixed order
// (fill_rows.cu); ek: extended kernel, image: subtract the ground's image.
mw_status fill_rows(const FillArgs& A, const GLParams& gl, bool image, bool ek, double flops, cudaStream_t st);

}  // namespace mw
