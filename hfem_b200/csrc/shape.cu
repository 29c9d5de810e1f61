// The kernels of one element shape, given by HFEM_ND, HFEM_NPV, HFEM_NPF,
// HFEM_NGV and HFEM_NGF (one translation unit per shape; launch.cuh).
#include <cuda_runtime.h>

#include "launch.cuh"
#include "elem_kernel.cuh"
#include "inverse_blocked.cuh"
#include "residual.cuh"

namespace hfem {

// GEMM tile choices per shape (m-tiles, n-tiles per warp, warps): g1 for D^-1 F
// (n x nb, K = n), g2 for H - K D^-1 F (nb x nb, K = n); the fastest of the
// candidates below on a B200, timed on 20k-51k-element meshes of each shape.
// Small CTAs (1-3 warps, 2-stage) win: many resident CTAs hide the short
// (K <= 100) main loops' fill and drain.
template <class S> struct SchurCfg;
template <> struct SchurCfg<Shape<2, 3, 2, 3, 2>> { using g1 = GemmCfg<2, 3, 1>; using g2 = GemmCfg<3, 3, 1>; };
template <> struct SchurCfg<Shape<2, 6, 3, 6, 3>> { using g1 = GemmCfg<3, 5, 1>; using g2 = GemmCfg<5, 3, 2>; };
template <> struct SchurCfg<Shape<2, 10, 4, 12, 4>> { using g1 = GemmCfg<5, 3, 2>; using g2 = GemmCfg<6, 3, 2>; };
template <> struct SchurCfg<Shape<2, 15, 5, 16, 5>> { using g1 = GemmCfg<4, 4, 2>; using g2 = GemmCfg<4, 2, 4>; };
template <> struct SchurCfg<Shape<3, 4, 3, 4, 3>> { using g1 = GemmCfg<3, 4, 2>; using g2 = GemmCfg<4, 2, 4>; };
template <> struct SchurCfg<Shape<3, 10, 6, 14, 6>> { using g1 = GemmCfg<4, 4, 2>; using g2 = GemmCfg<4, 2, 4>; };
template <> struct SchurCfg<Shape<3, 20, 10, 24, 12>> { using g1 = GemmCfg<5, 3, 3>; using g2 = GemmCfg<5, 3, 2>; };

template <int N>
void launch_inverse(dim3 g, cudaStream_t st, int ne, double* D, const double* Ru, double* RuOut, int* info) {
    if constexpr (N <= 32)
        inverse_warp_kernel<N><<<g, 32 * WINV_WARPS, 0, st>>>(ne, D, Ru, RuOut, info);
    else
        inverse_blocked_kernel<N><<<g, InvBlk<N>::THREADS, InvBlk<N>::SMEM, st>>>(ne, D, Ru, RuOut, info);
}
// threads, dynamic shared memory, matrices per CTA and the kernel itself
template <int N>
void inverse_launch(Launch& L) {
    if constexpr (N <= 32) {
        L.inv_threads = 32 * WINV_WARPS;
        L.inv_smem = 0;
        L.inv_per_cta = WINV_WARPS;
        L.inv_fn = (const void*)inverse_warp_kernel<N>;
    } else {
        L.inv_threads = InvBlk<N>::THREADS;
        L.inv_smem = InvBlk<N>::SMEM;
        L.inv_per_cta = 1;
        L.inv_fn = (const void*)inverse_blocked_kernel<N>;
    }
}

template <class S, bool TF, bool GEN>
void launch_element(dim3 g, size_t sm, cudaStream_t st, const ElemArgs& a) {
    element_kernel<S, TF, GEN><<<g, S::NT, sm, st>>>(a);
}
template <class S, bool GEN>
void launch_residual(dim3 g, size_t sm, cudaStream_t st, const ElemArgs& a) {
    residual_kernel<S, GEN><<<g, RES_THREADS, sm, st>>>(a);
}
template <class S>
void launch_getq(dim3 g, size_t sm, cudaStream_t st, const QArgs& a) { getq_kernel<S><<<g, QT, sm, st>>>(a); }
template <class S>
void launch_scatter_h(dim3 g, cudaStream_t st, const ScatterArgs& a) {
    scatter_H_block_kernel<S::NPF, S::NCH, S::NFE><<<g, 256, 0, st>>>(a);
}
template <class S>
void launch_schur_tc(dim3 g, size_t sm, cudaStream_t st, const SchurTcArgs& a) {
    schur_tc_kernel<S::N, S::NB><<<g, TC_THREADS, sm, st>>>(a);
}

// strip width and warps of the fused FP64 condensation per shape: as few strips as
// 40 columns allow, all of one width (nb = 48 in strips of 24 against 40 + 8: 0.119
// against 0.187 ms on 4,050 elements; nb = 60 in 32 against 40 + 20: 0.42 against
// 0.55 ms on 7,938)
template <class S>
struct FusedPick {
    static constexpr int STRIPS = (S::NB + 39) / 40;
    static constexpr int BN = ((S::NB + STRIPS - 1) / STRIPS + 7) / 8 * 8;
    static constexpr int MT = (S::N + 7) / 8;
    static constexpr int NW = MT >= 4 ? 4 : MT;
    using Cfg = FusedCfg<S::N, S::NB, BN, NW>;
};
template <class S>
void launch_schur_fused(cudaStream_t st, const FusedArgs& a) {
    static_assert(S::NB <= LIFT_MAXNB, "lift_inplace_kernel stages one column of H per warp");
    using P = FusedPick<S>;
    schur_fused_kernel<S::N, S::NB, P::BN, P::NW>
        <<<(unsigned)(a.ne * P::Cfg::STRIPS), P::Cfg::THREADS, P::Cfg::SMEM, st>>>(a);
}

template <class S>
Launch make_launch() {
    Launch L;
    L.nd = S::ND; L.npv = S::NPV; L.npf = S::NPF; L.ngv = S::NGV; L.ngf = S::NGF;
    L.ws = EK<S>::WS;
    L.ws_tf = EK<S>::WS_TF;
    L.q_smem = sizeof(QSmem<S>);
    L.q_threads = QT;
    L.getq = launch_getq<S>;
    L.q_fn = (const void*)getq_kernel<S>;
    L.inverse = launch_inverse<S::N>;
    L.element = launch_element<S, false, false>;
    L.element_v[0][0] = launch_element<S, false, false>;
    L.element_v[0][1] = launch_element<S, false, true>;
    L.element_v[1][0] = launch_element<S, true, false>;
    L.element_v[1][1] = launch_element<S, true, true>;
    L.elem_threads = S::NT;
    L.residual[0] = launch_residual<S, false>;
    L.residual[1] = launch_residual<S, true>;
    L.res_fn[0] = (const void*)residual_kernel<S, false>;
    L.res_fn[1] = (const void*)residual_kernel<S, true>;
    L.res_smem = sizeof(ResSmem<S>);
    L.res_threads = RES_THREADS;
    L.elem_smem = sizeof(ElemSmem<S>);
    L.elem_fn = (const void*)element_kernel<S, false, false>;
    L.elem_fn_v[0][0] = (const void*)element_kernel<S, false, false>;
    L.elem_fn_v[0][1] = (const void*)element_kernel<S, false, true>;
    L.elem_fn_v[1][0] = (const void*)element_kernel<S, true, false>;
    L.elem_fn_v[1][1] = (const void*)element_kernel<S, true, true>;
    inverse_launch<S::N>(L);
    L.g1 = GemmParams<typename SchurCfg<S>::g1>::make();
    L.g2 = GemmParams<typename SchurCfg<S>::g2>::make();
    L.schur_tc = launch_schur_tc<S>;
    L.tc_smem = TcCfg<S::N, S::NB>::SMEM;
    L.tc_tmem = (int)TcCfg<S::N, S::NB>::TMEM_COLS;
    L.tc_fn = (const void*)schur_tc_kernel<S::N, S::NB>;
    L.scatter_h = launch_scatter_h<S>;
    L.schur_fused = launch_schur_fused<S>;
    L.fused_smem = FusedPick<S>::Cfg::SMEM;
    L.fused_fn = (const void*)schur_fused_kernel<S::N, S::NB, FusedPick<S>::BN, FusedPick<S>::NW>;
    return L;
}

template Launch make_launch<Shape<HFEM_ND, HFEM_NPV, HFEM_NPF, HFEM_NGV, HFEM_NGF>>();

}  // namespace hfem
