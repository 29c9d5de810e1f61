// Residual norms and the outcome of an assembly on sm_100a.
//
// One kernel reduces what the host reads after a pass into one record: the
// residual norm (computeResidualNorm, globalassembly.cpp:618-678), the first
// singular element and the expired-wait flag.  CTAs sum in a fixed order and the
// last CTA to finish (atomic ticket, nothing waits) adds the partials in CTA
// order, so the norm is reproducible.  (Partial sums followed by one thread
// adding 296 of them took 19 us, and three separate reads of the outcome 25 us,
// of a 310 us pass over 2,048 2D p=2 elements.)
#pragma once
#include <cuda_runtime.h>

namespace hfem {

constexpr int NORM_THREADS = 256;
constexpr int NORM_CTAS = 148;          // most CTAs of one norm (about one per SM)

struct PassStatus {
    double rnorm;
    int bad_elem;                       // first element whose LU failed, or -1
    int bad_pivot;                      // 1 + pivot step of that element
    int wait_err;                       // an expired wait in a kernel of the pass (0: none)
    int pad;
};

struct NormPart {
    double sum;
    int bad_elem, pad;
};

struct NormArgs {
    int ne;
    long long nr;                       // trace entries
    const double *ru2, *rr;
    const int* info;                    // NULL: residual-only pass
    const int* wait_err;
    NormPart* part;
    int* ticket;
    PassStatus* out;
};

__device__ __forceinline__ double norm_block_sum(double s, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < NORM_THREADS / 32; w++) t += red[w];
    return t;
}
__device__ __forceinline__ int norm_block_min(int v, int* red) {
    v = __reduce_min_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    int t = red[0];
#pragma unroll
    for (int w = 1; w < NORM_THREADS / 32; w++) t = min(t, red[w]);
    return t;
}

static __global__ void __launch_bounds__(NORM_THREADS) pass_status_kernel(NormArgs A) {
    __shared__ double red[NORM_THREADS / 32];
    __shared__ int ired[NORM_THREADS / 32];
    __shared__ int last;
    constexpr int NONE = 0x7fffffff;
    double s = 0.0;
    int bad = NONE;
    const long long stride = (long long)gridDim.x * NORM_THREADS, t0 = blockIdx.x * (long long)NORM_THREADS + threadIdx.x;
    for (long long i = t0; i < A.ne; i += stride) {
        s += A.ru2[i];
        if (A.info && A.info[i]) bad = min(bad, (int)i);
    }
#pragma unroll 4
    for (long long i = t0; i < A.nr; i += stride) s += A.rr[i] * A.rr[i];
    s = norm_block_sum(s, red);
    bad = norm_block_min(bad, ired);
    if (threadIdx.x == 0) {
        A.part[blockIdx.x] = NormPart{s, bad, 0};
        __threadfence();
        last = atomicAdd(A.ticket, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double t = 0.0;
    int b = NONE;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += NORM_THREADS) {
        t += __ldcg(&A.part[i].sum);
        b = min(b, __ldcg(&A.part[i].bad_elem));
    }
    t = norm_block_sum(t, red);
    b = norm_block_min(b, ired);
    if (threadIdx.x != 0) return;
    *A.ticket = 0;
    *A.out = PassStatus{sqrt(t), b == NONE ? -1 : b, b == NONE ? 0 : A.info[b], *A.wait_err, 0};
}

// Per problem p of a context with a problem map: the norm over its elements and
// faces.  NORM_SPLIT CTAs per problem share its index ranges lo[p] .. hi[p] of
// elements and faces (the whole mesh when the map is not sorted; entries of
// other problems are skipped).
constexpr int NORM_SPLIT = 8;

struct ProblemNormArgs {
    int bsz;
    const double *ru2, *rr;
    const int *eprob, *fprob;
    const int* range;                   // per problem: first and last + 1 element, first and last + 1 face
    double* part;                       // nprob x NORM_SPLIT
    int* ticket;                        // per problem, zero between launches
    double* out;
};

static __global__ void __launch_bounds__(NORM_THREADS) problem_norm_kernel(ProblemNormArgs A) {
    __shared__ double red[NORM_THREADS / 32];
    __shared__ int last;
    const int p = blockIdx.x / NORM_SPLIT, k = blockIdx.x % NORM_SPLIT;
    const int* rg = A.range + 4 * p;
    const int t0 = k * NORM_THREADS + threadIdx.x, stride = NORM_SPLIT * NORM_THREADS;
    double s = 0.0;
    for (int e = rg[0] + t0; e < rg[1]; e += stride)
        if (A.eprob[e] == p) s += A.ru2[e];
    const long long n1 = (long long)rg[3] * A.bsz;
#pragma unroll 4
    for (long long i = (long long)rg[2] * A.bsz + t0; i < n1; i += stride)
        if (A.fprob[i / A.bsz] == p) s += A.rr[i] * A.rr[i];
    s = norm_block_sum(s, red);
    if (threadIdx.x == 0) {
        A.part[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(&A.ticket[p], 1) == NORM_SPLIT - 1;
        if (last) {
            __threadfence();
            double t = 0.0;
            for (int q = 0; q < NORM_SPLIT; q++) t += __ldcg(&A.part[p * NORM_SPLIT + q]);
            A.out[p] = sqrt(t);
            A.ticket[p] = 0;
        }
    }
}

}  // namespace hfem
