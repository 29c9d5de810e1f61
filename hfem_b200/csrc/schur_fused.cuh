// Static condensation, FP64, in one kernel (elementschur.cpp:6-329):
//   X = D^-1 (F + P H)  (n x nb, written out as DinvF),  H <- H - K X  and
//   Rh <- Rh - K (D^-1 Ru),
// on the FP64 tensor cores (mma.sync m8n8k4 f64).  One CTA per (element, strip
// of BN columns of F / DinvF / H): the strip of F, then of -X, is the B operand in
// shared memory.  A warp owns row tiles (8 rows, all BN/8 column tiles) and reads
// its A fragments (D^-1, then K: no other warp needs them) straight from global
// memory, PD k-steps ahead, so the products run without staging, barriers or a
// scaling of A; the strips of an element share A in L2.
// P H is the interior-face lift (lift.cuh), added as the F strip is loaded; strip 0
// also forms K (D^-1 Ru) from its A fragments.
// DinvF may be F itself: a CTA has its whole F strip in shared memory before it
// writes the X strip over it, and strips are disjoint.
// Bound by the FP64 tensor pipe (3D p=3: 24.4k DMMAs per element, 16.4 ms for
// 48,000 at the measured 37 TFLOP/s).  13,182 tetrahedra p = 3: 8.27 -> 6.19 ms
// (25.6 TFLOP/s) against A tiles staged through a cp.async ring with a
// barrier per 20 columns and alpha A formed for every fragment.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>
#include "lift.cuh"
#include "schur_kernels.cuh"

namespace hfem {

template <int N, int NB, int BN, int NW>
struct FusedCfg {
    static constexpr int MT = (N + 7) / 8;                 // row tiles of X
    static constexpr int MTH = (NB + 7) / 8;               // row tiles of H
    static constexpr int NTN = BN / 8;                     // column tiles
    static constexpr int KS = (N + 3) / 4;                 // k-steps
    static constexpr int KP = 4 * KS;                      // padded k extent (rows of the B strip)
    static constexpr int LDB = ((KP + 11) / 16) * 16 + 4;  // == 4 (mod 16): conflict-free B fragments
    static constexpr int STRIPS = (NB + BN - 1) / BN;
    static constexpr int THREADS = 32 * NW;
    static constexpr size_t SMEM = sizeof(double) * ((size_t)LDB * BN + KP);
    static constexpr int XW = (MT + NW - 1) / NW;          // most row tiles of one warp, X and H
    static constexpr int HW = (MTH + NW - 1) / NW;
    // Row tiles of H at a time, k-steps that A is read ahead, and CTAs per SM.  Large
    // elements: two tiles share every B fragment, 128 registers.  Small ones are
    // bound by the latency of loading F, H and A of many short CTAs: one tile at a
    // time in 64 registers.  Measured (ms; 2, 6, 4 | 1, 4, 8): 13,182 3D p3 6.19 |
    // 11.7; 4,374 3D p2 0.536 | 0.493; 10,368 3D p1 0.304 | 0.218; 7,938 2D p4 0.419 |
    // 0.360; 4,050 2D p3 0.119 | 0.109; 2,048 2D p2 0.038 | 0.029.
    static constexpr bool LARGE = N >= 64;
    static constexpr int PASS = LARGE ? 2 : 1, PD = (LARGE ? 6 : 4) < KS ? (LARGE ? 6 : 4) : KS, CTAS = LARGE ? 4 : 8;
    static_assert(BN % 8 == 0, "whole column tiles");
};

struct FusedArgs {
    int ne;
    const double *Dinv, *F, *K;
    double *H, *DinvF;          // DinvF may be F
    const double* DinvRu;
    double* Rh;
    LiftArgs lift;              // perm, bf and sizes; src and cols unused
};

// acc[a] += A(rows of tile t[a], :) Bs for T row tiles of one warp: A column-major,
// rows past m_end repeat the last row (their results are not stored); RHS: also
// y[a] = this lane's share of A (row 8 t[a] + gr) . dru.
template <class C, int T, bool RHS>
__device__ __forceinline__ void fused_product(const double* __restrict__ A, int lda, int m_end, int n,
                                              const int (&t)[T], const double* Bs, const double* dru,
                                              double (&acc)[T][C::NTN][2], double (&y)[T]) {
    constexpr int PD = C::PD;
    const int lane = threadIdx.x & 31, gr = lane >> 2, gc = lane & 3;
    const double* ap[T];
#pragma unroll
    for (int a = 0; a < T; a++) {
        const int row = 8 * t[a] + gr;
        ap[a] = A + (row < m_end ? row : m_end - 1) + (size_t)lda * gc;
    }
    auto fetch = [&](int ks, double (&f)[T]) {
#pragma unroll
        for (int a = 0; a < T; a++)
            f[a] = (4 * C::KS == n || 4 * ks + gc < n) ? __ldg(ap[a] + (size_t)lda * 4 * ks) : 0.0;
    };
    double f[PD][T];
#pragma unroll
    for (int p = 0; p < PD; p++) fetch(p, f[p]);
    const double* bp = Bs + gc + C::LDB * gr;
#pragma unroll
    for (int ks = 0; ks < C::KS; ks++) {
        double af[T], bf[C::NTN];
#pragma unroll
        for (int a = 0; a < T; a++) af[a] = f[ks % PD][a];
        if (ks + PD < C::KS) fetch(ks + PD, f[ks % PD]);
#pragma unroll
        for (int b = 0; b < C::NTN; b++) bf[b] = bp[4 * ks + C::LDB * 8 * b];
#pragma unroll
        for (int b = 0; b < C::NTN; b++)
#pragma unroll
            for (int a = 0; a < T; a++) dmma8x8x4(acc[a][b][0], acc[a][b][1], af[a], bf[b]);
        if constexpr (RHS) {
            const double d = dru[4 * ks + gc];
#pragma unroll
            for (int a = 0; a < T; a++) y[a] = fma(af[a], d, y[a]);
        }
    }
}

template <int N, int NB, int BN, int NW>
__global__ void __launch_bounds__(32 * NW, (FusedCfg<N, NB, BN, NW>::CTAS)) schur_fused_kernel(FusedArgs A) {
    using C = FusedCfg<N, NB, BN, NW>;
    extern __shared__ __align__(16) double fsm[];
    double* Bs = fsm;                                  // LDB x BN: the F strip, then the -X strip
    double* dru = fsm + (size_t)C::LDB * BN;           // D^-1 Ru, zero padded
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gr = lane >> 2, gc = lane & 3;
    const int e = blockIdx.x / C::STRIPS, c0 = (blockIdx.x % C::STRIPS) * BN;
    if (e >= A.ne) return;
    const double* De = A.Dinv + (size_t)e * N * N;
    const double* Fe = A.F + (size_t)e * N * NB;
    const double* Ke = A.K + (size_t)e * NB * N;
    double* He = A.H + (size_t)e * NB * NB;
    double* Xe = A.DinvF + (size_t)e * N * NB;
    const bool rhs = c0 == 0;
    // the warps' shares rotate from CTA to CTA, so that the longer shares of the
    // CTAs of an SM do not meet on one scheduler
    const int w = (warp + (int)((blockIdx.x * 2654435761u) >> 16)) % NW;

    // the strip of F + P H; rows >= N and columns past NB are zero.  A thread keeps
    // one row of F for all columns.
    {
        constexpr int CG = C::THREADS / N;
        static_assert(CG > 0, "one thread per row of F");
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
        for (int t = tid; t < C::KP; t += C::THREADS) dru[t] = t < N ? A.DinvRu[(size_t)e * N + t] : 0.0;
    }
    __syncthreads();

    // ---- X = D^-1 (F + P H)_strip: row tiles w, w + NW, ...
    double x[C::XW][C::NTN][2];
    {
        int t[C::XW];
        double none[C::XW];
#pragma unroll
        for (int a = 0; a < C::XW; a++) {
            t[a] = w + NW * a;
#pragma unroll
            for (int b = 0; b < C::NTN; b++) x[a][b][0] = x[a][b][1] = 0.0;
        }
        // the last tile of a warp with fewer tiles than the others: nothing to do
        if (w + NW * (C::XW - 1) < C::MT) {
            fused_product<C, C::XW, false>(De, N, N, N, t, Bs, dru, x, none);
        } else if constexpr (C::XW > 1) {
            fused_product<C, C::XW - 1, false>(De, N, N, N, reinterpret_cast<const int(&)[C::XW - 1]>(t), Bs, dru,
                                               reinterpret_cast<double(&)[C::XW - 1][C::NTN][2]>(x),
                                               reinterpret_cast<double(&)[C::XW - 1]>(none));
        }
    }
    __syncthreads();
    // X to global memory, -X into Bs (the B operand of the second product)
#pragma unroll
    for (int a = 0; a < C::XW; a++) {
        const int mt = w + NW * a;
#pragma unroll
        for (int b = 0; b < C::NTN; b++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int row = 8 * mt + gr, col = 8 * b + 2 * gc + h;
                if (mt < C::MT && row < N) {
                    Bs[row + C::LDB * col] = -x[a][b][h];
                    if (c0 + col < NB) Xe[row + (size_t)N * (c0 + col)] = x[a][b][h];
                }
            }
    }
    __syncthreads();

    // ---- H_strip += K (-X): row tiles from the other end (w = NW - 1 first), so
    // that the warps with one tile of X more have one of H less; PASS at a time
    const int wh = NW - 1 - w;
    auto hpass = [&](auto tc, int a0) {
        constexpr int T = decltype(tc)::value;
        int t[T];
        double acc[T][C::NTN][2], y[T];
#pragma unroll
        for (int a = 0; a < T; a++) {
            t[a] = wh + NW * (a0 + a);
            y[a] = 0.0;
#pragma unroll
            for (int b = 0; b < C::NTN; b++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int row = 8 * t[a] + gr, col = c0 + 8 * b + 2 * gc + h;
                    acc[a][b][h] = (row < NB && col < NB) ? He[row + (size_t)NB * col] : 0.0;
                }
        }
        if (rhs) fused_product<C, T, true>(Ke, NB, NB, N, t, Bs, dru, acc, y);
        else fused_product<C, T, false>(Ke, NB, NB, N, t, Bs, dru, acc, y);
#pragma unroll
        for (int a = 0; a < T; a++) {
            const int row = 8 * t[a] + gr;
#pragma unroll
            for (int b = 0; b < C::NTN; b++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int col = c0 + 8 * b + 2 * gc + h;
                    if (row < NB && col < NB) He[row + (size_t)NB * col] = acc[a][b][h];
                }
            if (rhs) {
                y[a] += __shfl_xor_sync(0xffffffffu, y[a], 1);
                y[a] += __shfl_xor_sync(0xffffffffu, y[a], 2);
                if (gc == 0 && row < NB) A.Rh[(size_t)e * NB + row] -= y[a];
            }
        }
    };
    const int cnt = wh < C::MTH ? (C::MTH - wh + NW - 1) / NW : 0;      // this warp's row tiles of H
    int a0 = 0;
#pragma unroll 1
    for (; a0 + C::PASS <= cnt; a0 += C::PASS) hpass(std::integral_constant<int, C::PASS>{}, a0);
    if constexpr (C::PASS > 1)
        if (a0 < cnt) hpass(std::integral_constant<int, 1>{}, a0);
}

}  // namespace hfem
