// Block-Jacobi preconditioner of the condensed HDG system on sm_100a: the apply
// and the FP32 copy (the inverses: inverse_blocked.cuh).  Specification (the
// reference ships it only as a closed archive): kernel/mkBlockJacobi.m:1-16,
// M_i^-1 = inv(Hg_ii), the first block of row i.
#pragma once
#include <cuda_runtime.h>

namespace hfem {

// z = M^-1 b (block-diagonal apply; MT = float: the FP32 preconditioner of the mixed mode).
template <typename MT>
__global__ void bj_apply_kernel(int nrows, int bsz, const MT* __restrict__ Minv, const double* __restrict__ b,
                                double* __restrict__ z) {
    const long long total = (long long)nrows * bsz;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t / bsz), r = (int)(t % bsz);
        const MT* m = Minv + (size_t)i * bsz * bsz;
        const double* bi = b + (size_t)i * bsz;
        double s = 0.0;
        for (int c = 0; c < bsz; c++) s += (double)m[r + bsz * c] * bi[c];
        z[t] = s;
    }
}

// FP32 copy of the block-Jacobi inverses (the mixed mode's preconditioner).
__global__ void to_float_kernel(long long n, const double* __restrict__ a, float* __restrict__ b) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

}  // namespace hfem
