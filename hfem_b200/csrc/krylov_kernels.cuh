// Block-Jacobi preconditioner of the condensed HDG system on sm_100a: inverses
// of the diagonal blocks, the apply, and the FP32 copy.
//
// Specifications (the reference ships these only as closed archives):
//   kernel/mkBlockJacobi.m:1-16  M_i^-1 = inv(Hg_ii), the first block of row i
#pragma once
#include <cuda_runtime.h>

namespace hfem {

// Inverse of each row's diagonal block by Gauss-Jordan with partial pivoting.
// One CTA per block row; bsz <= 64.  info[i] = 1 + k on a zero pivot.
__global__ void bj_inverse_kernel(int nrows, int bsz, const int* __restrict__ rowstart, const double* __restrict__ Hg,
                                  double* __restrict__ Minv, int* __restrict__ info) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* a = reinterpret_cast<double*>(smem_raw);   // bsz x bsz
    double* col = a + bsz * bsz;
    int* piv = reinterpret_cast<int*>(col + bsz);
    __shared__ int s_p;
    const int tid = threadIdx.x;
    for (int i = blockIdx.x; i < nrows; i += gridDim.x) {
        __syncthreads();
        const double* blk = Hg + (size_t)rowstart[i] * bsz * bsz;
        for (int t = tid; t < bsz * bsz; t += blockDim.x) a[t] = blk[t];
        __syncthreads();
        int bad = 0;
        for (int k = 0; k < bsz; k++) {
            if (tid == 0) {
                int p = k;
                double best = fabs(a[k + bsz * k]);
                for (int r = k + 1; r < bsz; r++) {
                    const double v = fabs(a[r + bsz * k]);
                    if (v > best) { best = v; p = r; }
                }
                s_p = p;
                piv[k] = p;
            }
            __syncthreads();
            const int p = s_p;
            if (a[p + bsz * k] == 0.0) { bad = k + 1; break; }
            if (p != k)
                for (int c = tid; c < bsz; c += blockDim.x) {
                    const double t = a[k + bsz * c];
                    a[k + bsz * c] = a[p + bsz * c];
                    a[p + bsz * c] = t;
                }
            __syncthreads();
            const double dinv = 1.0 / a[k + bsz * k];
            for (int r = tid; r < bsz; r += blockDim.x) col[r] = (r == k) ? 0.0 : a[r + bsz * k];
            __syncthreads();
            for (int c = tid; c < bsz; c += blockDim.x) a[k + bsz * c] = (c == k ? 1.0 : a[k + bsz * c]) * dinv;
            __syncthreads();
            for (int t = tid; t < bsz * bsz; t += blockDim.x) {
                const int r = t % bsz, c = t / bsz;
                if (r != k) a[r + bsz * c] = (c == k ? 0.0 : a[r + bsz * c]) - col[r] * a[k + bsz * c];
            }
            __syncthreads();
        }
        if (bad) {
            if (tid == 0) info[i] = bad;
            continue;
        }
        for (int k = bsz - 1; k >= 0; k--) {
            const int p = piv[k];
            if (p != k)
                for (int r = tid; r < bsz; r += blockDim.x) {
                    const double t = a[r + bsz * k];
                    a[r + bsz * k] = a[r + bsz * p];
                    a[r + bsz * p] = t;
                }
            __syncthreads();
        }
        double* out = Minv + (size_t)i * bsz * bsz;
        for (int t = tid; t < bsz * bsz; t += blockDim.x) out[t] = a[t];
        if (tid == 0) info[i] = 0;
    }
}

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
