// Kernel table of one element shape: what the host side launches, with sizes and
// attributes.  make_launch<Shape> is instantiated in one translation unit per
// shape (shape.cu), so that the shapes compile in parallel; the host side
// (hfem_capi.cu) only sees the declarations below.
#pragma once
#include <cuda_runtime.h>

#include "elem_kernels.cuh"
#include "schur_kernels.cuh"
#include "schur_tc.cuh"
#include "schur_fused.cuh"

namespace hfem {

// Element shapes with compiled kernels: (nd, npv, npf, ngv, ngf).
#define HFEM_SHAPES(X)          \
    X(2, 3, 2, 3, 2)            \
    X(2, 6, 3, 6, 3)            \
    X(2, 10, 4, 12, 4)          \
    X(2, 15, 5, 16, 5)          \
    X(3, 4, 3, 4, 3)            \
    X(3, 10, 6, 14, 6)          \
    X(3, 20, 10, 24, 12)

struct GemmLaunch {
    int bm, bn, threads;
    size_t smem;
    const void* fn;
    void (*run)(cudaStream_t, int, int, int, int, double, const double*, int, long long, const double*, int,
                long long, double, double*, int, long long);
};

template <class G, int MT, int WN, int NW, int BK, int ST>
void run_gemm(cudaStream_t st, int batch, int M, int N, int K, double alpha, const double* A, int lda, long long sA,
              const double* B, int ldb, long long sB, double beta, double* C, int ldc, long long sC) {
    const int tiles = ((M + G::BM - 1) / G::BM) * ((N + G::BN - 1) / G::BN);
    batched_dgemm_kernel<MT, WN, NW, BK, ST><<<(unsigned)(tiles * batch), G::THREADS, G::SMEM, st>>>(
        M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC);
}

template <class G> struct GemmParams;
template <int MT, int WN, int NW, int BK, int ST> struct GemmParams<GemmCfg<MT, WN, NW, BK, ST>> {
    static GemmLaunch make() {
        using G = GemmCfg<MT, WN, NW, BK, ST>;
        return GemmLaunch{G::BM, G::BN, G::THREADS, G::SMEM, (const void*)batched_dgemm_kernel<MT, WN, NW, BK, ST>,
                          run_gemm<G, MT, WN, NW, BK, ST>};
    }
};

struct Launch {
    int nd, npv, npf, ngv, ngf;
    size_t ws, ws_tf;           // workspace doubles per CTA slot of element_kernel, FP64 and 3xTF32 forms
    int elem_threads;           // threads per CTA of the element kernels
    size_t q_smem;
    int q_threads;
    void (*getq)(dim3, size_t, cudaStream_t, const QArgs&);
    void (*inverse)(dim3, cudaStream_t, int, double*, const double*, double*, int*);
    void (*element)(dim3, size_t, cudaStream_t, const ElemArgs&);
    // [tf][gen]: 3xTF32 contractions; Lax-Friedrichs / Roe tensor or Sutherland's law compiled in
    void (*element_v[2][2])(dim3, size_t, cudaStream_t, const ElemArgs&);
    size_t elem_smem;
    // residual-only pass [gen]
    void (*residual[2])(dim3, size_t, cudaStream_t, const ElemArgs&);
    const void* res_fn[2];
    size_t res_smem;
    int res_threads;
    const void* elem_fn;
    const void* elem_fn_v[2][2];
    int inv_threads, inv_per_cta;
    size_t inv_smem;
    const void *q_fn, *inv_fn;
    GemmLaunch g1, g2;
    void (*schur_tc)(dim3, size_t, cudaStream_t, const SchurTcArgs&);
    size_t tc_smem;
    int tc_tmem;                // tensor-memory columns of one tensor-core Schur CTA
    const void* tc_fn;
    void (*scatter_h)(dim3, cudaStream_t, const ScatterArgs&);
    void (*schur_fused)(cudaStream_t, const FusedArgs&);
    size_t fused_smem;
    const void* fused_fn;
};

template <class S>
Launch make_launch();

}  // namespace hfem
