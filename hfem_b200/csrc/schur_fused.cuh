// Static condensation, FP64, in one kernel (elementschur.cpp:6-329):
//   X = D^-1 (F + P H)  (n x nb, written out as DinvF),  H <- H - K X  and
//   Rh <- Rh - K (D^-1 Ru),
// on the FP64 tensor cores (mma.sync m8n8k4 f64).  One CTA per (element, strip
// of BN columns of F / DinvF / H): the strip of X never leaves shared memory
// between the two products.  A operands (D^-1, then K in row chunks) stream
// through a 2-stage cp.async ring in k tiles of 20; the B operand (the F strip,
// then the X strip) sits in shared memory whole.  Warp w owns m-tiles w, w+NW,
// ... of every job and all BN/8 n-tiles.  H's accumulators start from H.
// P H is the interior-face lift (lift.cuh), added as the F strip is loaded; the
// CTA of strip 0 also forms K (D^-1 Ru) from the K tiles in its ring (as kernels
// of their own these took 1.76 and 0.41 ms beside this one's 7.07 on 13,182
// tetrahedra p = 3).
// DinvF may be F itself: a CTA has its whole F strip in shared memory before it
// writes the X strip over it, and strips are disjoint.
#pragma once
#include <cuda_runtime.h>
#include "lift.cuh"
#include "schur_kernels.cuh"

namespace hfem {

template <int N, int NB, int BN, int NW>
struct FusedCfg {
    static constexpr int BK = 20;
    static constexpr int MT = (N + 7) / 8;                 // m-tiles per job (rows of D^-1, or a chunk of K)
    static constexpr int BM = 8 * MT;
    static constexpr int NTN = BN / 8;                     // n-tiles
    static constexpr int KT = (N + BK - 1) / BK;           // k tiles
    static constexpr int KP = KT * BK;                     // padded k extent (rows of the B strip)
    static constexpr int LDA = ((BM + 11) / 16) * 16 + 4;  // == 4 (mod 16)
    static constexpr int LDB = ((KP + 11) / 16) * 16 + 4;  // == 4 (mod 16)
    static constexpr int MPW = (MT + NW - 1) / NW;         // m-tiles per warp
    static constexpr int CHUNKS = (NB + BM - 1) / BM;      // row chunks of K / H
    static constexpr int STRIPS = (NB + BN - 1) / BN;
    static constexpr int THREADS = 32 * NW;
    static constexpr size_t SMEM = sizeof(double) * ((size_t)LDB * BN + 2 * (size_t)LDA * BK);
    static_assert(BM <= THREADS, "one thread per row of a chunk (Rh)");
    static_assert(BN % 8 == 0 && N % 2 == 0 && NB % 2 == 0, "tile and 16-byte copy granularity");
};

struct FusedArgs {
    int ne;
    const double *Dinv, *F, *K;
    double *H, *DinvF;          // DinvF may be F
    const double* DinvRu;
    double* Rh;
    LiftArgs lift;              // perm, bf and sizes; src and cols unused
};

template <int N, int NB, int BN, int NW>
__global__ void __launch_bounds__(32 * NW) schur_fused_kernel(FusedArgs A) {
    using C = FusedCfg<N, NB, BN, NW>;
    extern __shared__ __align__(16) double fsm[];
    double* Bs = fsm;                                  // LDB x BN: the F strip, then the X strip
    double* As = fsm + (size_t)C::LDB * BN;            // 2 stages of LDA x BK
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gr = lane >> 2, gc = lane & 3;
    const int e = blockIdx.x / C::STRIPS, c0 = (blockIdx.x % C::STRIPS) * BN;
    if (e >= A.ne) return;
    const double* De = A.Dinv + (size_t)e * N * N;
    const double* Fe = A.F + (size_t)e * N * NB;
    const double* Ke = A.K + (size_t)e * NB * N;
    double* He = A.H + (size_t)e * NB * NB;
    double* Xe = A.DinvF + (size_t)e * N * NB;

    // A tile loader: rows [m0, m0 + BM) of A (lda rows, m_end valid), k columns [k0, k0 + BK)
    auto load_a = [&](int st, const double* A, int lda, int m0, int m_end, int k0) {
        double* as = As + (size_t)st * C::LDA * C::BK;
        for (int t = tid; t < (C::BM / 2) * C::BK; t += C::THREADS) {
            const int m = 2 * (t % (C::BM / 2)), k = t / (C::BM / 2);
            const bool ok = m0 + m < m_end && k0 + k < N;
            cp_async16z(&as[m + C::LDA * k], A + (ok ? (m0 + m) + (size_t)lda * (k0 + k) : 0), ok);
        }
    };

    double acc[C::MPW][C::NTN][2];
    double yrow = 0.0;         // strip 0: row tid of K (D^-1 Ru), this chunk
    const bool rhs = c0 == 0;
    const double* dru = A.DinvRu + (size_t)e * N;
    // one product: acc (+)= alpha A[m0.., :] Bs, k tiles through the ring (the
    // first one already requested)
    auto run = [&](const double* A, int lda, int m0, int m_end, double alpha, bool gemv) {
        for (int kt = 0; kt < C::KT; kt++) {
            cp_async_wait<0>();
            __syncthreads();
            if (kt + 1 < C::KT) load_a((kt + 1) & 1, A, lda, m0, m_end, (kt + 1) * C::BK);
            cp_async_commit();
            const double* as = As + (size_t)(kt & 1) * C::LDA * C::BK;
            if (gemv && tid < C::BM) {
#pragma unroll 4
                for (int k = 0; k < C::BK; k++)
                    if (kt * C::BK + k < N) yrow = fma(as[tid + C::LDA * k], __ldg(&dru[kt * C::BK + k]), yrow);
            }
#pragma unroll
            for (int ks = 0; ks < C::BK; ks += 4) {
                double bf[C::NTN];
#pragma unroll
                for (int b = 0; b < C::NTN; b++) bf[b] = Bs[(kt * C::BK + ks + gc) + C::LDB * (8 * b + gr)];
#pragma unroll
                for (int a = 0; a < C::MPW; a++) {
                    const int mt = warp + NW * a;
                    if (mt < C::MT) {
                        const double af = alpha * as[(8 * mt + gr) + C::LDA * (ks + gc)];
#pragma unroll
                        for (int b = 0; b < C::NTN; b++) dmma8x8x4(acc[a][b][0], acc[a][b][1], af, bf[b]);
                    }
                }
            }
        }
        __syncthreads();   // every warp is done with the ring and with Bs
    };

    // ---- X = D^-1 (F + P H)_strip; the strip's rows >= N and columns past NB are
    // zero.  A thread keeps one row of F for all columns.
    load_a(0, De, N, 0, N, 0);
    cp_async_commit();
    {
        constexpr int CG = C::THREADS / N > 0 ? C::THREADS / N : 1;
        static_assert(N <= C::THREADS, "one thread per row of F");
        const int row = tid % N, cg = tid / N;
        if (cg < CG) {
            const LiftRow lr = lift_row(A.lift, e, row);
#pragma unroll 8
            for (int col = cg; col < BN; col += CG) {
                const bool ok = c0 + col < NB;
                Bs[row + C::LDB * col] =
                    ok ? lift_add_row(lr, He + (size_t)NB * (c0 + col), Fe[row + (size_t)N * (c0 + col)]) : 0.0;
            }
        }
        if constexpr (C::KP > N)
            for (int t = tid; t < (C::KP - N) * BN; t += C::THREADS)
                Bs[N + t % (C::KP - N) + C::LDB * (t / (C::KP - N))] = 0.0;
    }
#pragma unroll
    for (int a = 0; a < C::MPW; a++)
#pragma unroll
        for (int b = 0; b < C::NTN; b++) acc[a][b][0] = acc[a][b][1] = 0.0;
    run(De, N, 0, N, 1.0, false);
    // X to global and into Bs (the B operand of the second product)
#pragma unroll
    for (int a = 0; a < C::MPW; a++) {
        const int mt = warp + NW * a;
#pragma unroll
        for (int b = 0; b < C::NTN; b++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int row = 8 * mt + gr, col = 8 * b + 2 * gc + h;
                if (mt < C::MT && row < N) {
                    Bs[row + C::LDB * col] = acc[a][b][h];
                    if (c0 + col < NB) Xe[row + (size_t)N * (c0 + col)] = acc[a][b][h];
                }
            }
    }
    __syncthreads();

    // ---- H_strip -= K X, in row chunks of BM
    for (int ch = 0; ch < C::CHUNKS; ch++) {
        const int m0 = ch * C::BM;
        load_a(0, Ke, NB, m0, NB, 0);
        cp_async_commit();
#pragma unroll
        for (int a = 0; a < C::MPW; a++)
#pragma unroll
            for (int b = 0; b < C::NTN; b++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int mt = warp + NW * a;
                    const int row = m0 + 8 * mt + gr, col = c0 + 8 * b + 2 * gc + h;
                    acc[a][b][h] = (mt < C::MT && row < NB && col < NB) ? He[row + (size_t)NB * col] : 0.0;
                }
        yrow = 0.0;
        run(Ke, NB, m0, NB, -1.0, rhs);
        if (rhs && tid < C::BM && m0 + tid < NB) A.Rh[(size_t)e * NB + m0 + tid] -= yrow;
#pragma unroll
        for (int a = 0; a < C::MPW; a++) {
            const int mt = warp + NW * a;
#pragma unroll
            for (int b = 0; b < C::NTN; b++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int row = m0 + 8 * mt + gr, col = c0 + 8 * b + 2 * gc + h;
                    if (mt < C::MT && row < NB && col < NB) He[row + (size_t)NB * col] = acc[a][b][h];
                }
        }
    }
}

}  // namespace hfem
