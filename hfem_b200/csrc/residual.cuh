// Residual-only element pass (computeResidualNorm, globalassembly.cpp:618-678) on
// sm_100a: Ru = Ru_vol + P Rh and Rh of every element, without the Jacobian blocks.
//
// The line search of a Newton iteration asks for the residual alone; the element
// kernel formed all four blocks for it (0.87 ms per pass over 1,296 tetrahedra
// p = 3, 7 of 47 ms of a DIRK step; this kernel: 0.058 ms).  Bound by FP64 latency in
// the point states and fluxes (FP64 pipe 11 % active; stalls on global loads, on
// fixed-latency results and at barriers, in this order): no block products, so 128
// threads; four CTAs per SM, as many as 128 registers a thread allow.
#pragma once
#include <cuda_runtime.h>
#include "elem_kernels.cuh"

namespace hfem {

constexpr int RES_THREADS = 128;

template <class S>
struct ResSmem {
    double x[S::NPV * S::ND];
    double jac[S::NGV], Xx[S::NGV * S::ND * S::ND];
    double jacf[S::NA], nl[S::NA * S::ND];
    double u[S::NPV * S::NC], uhe[S::NDF * S::NCH], shu[S::NPV * S::NCU];
    double ug[S::NGV * S::NC], ugf[S::NA * S::NC], uhg[S::NA * S::NCH];
    double wrk[S::NQ * S::NCU];
    double fn[S::NA * S::NCH];              // fhat times jacf
    double fb[S::NA * S::NCH];              // boundary flux times jacf (boundary faces)
    double rh[S::NB];
    double red[RES_THREADS / 32];
    int perm[S::NDF];
    int inc_n[S::NPV];
    int inc_f[S::NPV * S::MAXINC];
};

// GEN: the Lax-Friedrichs / Roe tensors and Sutherland's law compiled in
template <class S, bool GEN>
__global__ void __launch_bounds__(RES_THREADS, 4) residual_kernel(ElemArgs A) {
    constexpr int ND = S::ND, NPV = S::NPV, NPF = S::NPF, NGV = S::NGV, NGF = S::NGF, NFE = S::NFE;
    constexpr int NCU = S::NCU, NC = S::NC, NCH = S::NCH, NDF = S::NDF, ND1 = S::ND1, N = S::N, NB = S::NB;
    constexpr int NA = S::NA, NQ = S::NQ, NTH = RES_THREADS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ResSmem<S>& sm = *reinterpret_cast<ResSmem<S>*>(smem_raw);
    const Tables& T = A.T;
    const int tid = threadIdx.x;
    for (int t = tid; t < NDF; t += NTH) sm.perm[t] = T.perm[t];
    __syncthreads();
    for (int i = tid; i < NPV; i += NTH) {
        int c = 0;
        for (int f = 0; f < NDF; f++)
            if (sm.perm[f] == i && c < S::MAXINC) sm.inc_f[i * S::MAXINC + c++] = f;
        sm.inc_n[i] = c;
    }
    for (int e = A.e_begin + blockIdx.x; e < A.ne; e += gridDim.x) {
        __syncthreads();
        for (int t = tid; t < NPV * ND; t += NTH) sm.x[t] = A.dgnodes[(size_t)e * NPV * ND + t];
        for (int t = tid; t < NPV * NC; t += NTH) sm.u[t] = A.udg[(size_t)e * NPV * NC + t];
        for (int t = tid; t < NPV * NCU; t += NTH) sm.shu[t] = A.sh[(size_t)e * NPV * NC + t];
        for (int t = tid; t < NDF * NCH; t += NTH) {
            const int fdof = t / NCH, c = t % NCH;
            sm.uhe[fdof + NDF * c] = A.uh[(size_t)A.elcon[(size_t)e * NDF + fdof] * NCH + c];
        }
        __syncthreads();
        geometry<S>(T, sm.x, sm.jac, sm.Xx, sm.jacf, sm.nl);
        const double* P = A.pparam ? A.pparam + 8 * A.eprob[e] : A.param;
        const int tdep = A.pparam ? (int)P[6] : A.tdep;
        const double fc_u = A.pparam ? P[7] : A.fc_u;
        const int* bfe = A.bf ? A.bf + (size_t)e * NFE : nullptr;
        // states at the points
        for (int t = tid; t < NGV * NC; t += NTH) {
            const int g = t % NGV, c = t / NGV;
            double s = 0.0;
#pragma unroll 4
            for (int a = 0; a < NPV; a++) s = fma(__ldg(&T.shapvt[g + NGV * a]), sm.u[a + NPV * c], s);
            sm.ug[t] = s;
        }
        for (int t = tid; t < NA * (NC + NCH); t += NTH) {
            const int gg = t % NA, c = t / NA, fc = gg / NGF, q = gg % NGF;
            double s = 0.0;
            if (c < NC) {
#pragma unroll 4
                for (int m = 0; m < NPF; m++)
                    s = fma(__ldg(&T.shapft[q + NGF * m]), sm.u[sm.perm[fc * NPF + m] + NPV * c], s);
                sm.ugf[gg + NA * c] = s;
            } else {
#pragma unroll 4
                for (int m = 0; m < NPF; m++)
                    s = fma(__ldg(&T.shapft[q + NGF * m]), sm.uhe[fc * NPF + m + NDF * (c - NC)], s);
                sm.uhg[gg + NA * (c - NC)] = s;
            }
        }
        __syncthreads();
        // fluxes through each metric row of a volume point and the scaled normal of a face point
        const double gam = P[0], iRe = A.inviscid ? 0.0 : 1.0 / P[2], kappa = A.inviscid ? 0.0 : gam * iRe / P[3];
        constexpr int NVD = NGV * ND;
        for (int p = tid; p < NVD + NA; p += NTH) {
            const bool vol = p < NVD;
            const int g = vol ? p % NGV : p - NVD, r = p / NGV, fc = g / NGF;
            double w[NC], X[ND], f[NCU];
#pragma unroll
            for (int c = 0; c < NC; c++)
                w[c] = vol ? sm.ug[g + NGV * c] : ((c < NCU) ? sm.uhg[g + NA * c] : sm.ugf[g + NA * c]);
#pragma unroll
            for (int d = 0; d < ND; d++) X[d] = vol ? sm.Xx[g + NGV * (d + ND * r)] : sm.nl[g + NA * d] * sm.jacf[g];
            double mu = 1.0;
            if constexpr (GEN) {
                if (A.visc_model != 0 && !A.inviscid) {
                    Dual<1> wd[NCU];
#pragma unroll
                    for (int c = 0; c < NCU; c++) wd[c] = dc<1>(w[c]);
                    mu = ns_sutherland<ND, 1>(P, wd).v;
                }
            }
            NsDir<ND> s;
            ns_dir<ND>(gam, iRe, kappa, mu, w, X, s);
            ns_dir_value<ND>(s, [&](int j, double v) { f[j] = v; });
            if (vol) {
#pragma unroll
                for (int j = 0; j < NCU; j++) sm.wrk[g + NGV * (r + 1 + ND1 * j)] = f[j];
                if (r == 0) {
                    const double jg = sm.jac[g];
#pragma unroll
                    for (int j = 0; j < NCU; j++) {
                        double src = 0.0;
                        if (tdep) {
                            double tt = 0.0;
#pragma unroll 4
                            for (int a = 0; a < NPV; a++) tt = fma(__ldg(&T.shapvt[g + NGV * a]), sm.shu[a + NPV * j], tt);
                            src = tt - w[j] * fc_u;
                        }
                        sm.wrk[g + NGV * ND1 * j] = src * jg;
                    }
                }
                continue;
            }
            const double jf = sm.jacf[g];
            if (!GEN || A.conv_stab == 0) {
                const double tau = P[5];
#pragma unroll
                for (int j = 0; j < NCU; j++) sm.fn[g + NA * j] = fma(tau * jf, sm.ugf[g + NA * j] - w[j], f[j]);
            } else {
                Dual<1> uhd[NCU], dv[NCU], st[NCU];
                double nlq[ND];
#pragma unroll
                for (int d = 0; d < ND; d++) nlq[d] = sm.nl[g + NA * d];
#pragma unroll
                for (int m = 0; m < NCU; m++) {
                    uhd[m] = dc<1>(w[m]);
                    dv[m] = dc<1>(sm.ugf[g + NA * m] - w[m]);
                }
                ns_stab_apply<ND, 1>(A.conv_stab, P, nlq, uhd, dv, st);
#pragma unroll
                for (int j = 0; j < NCU; j++) sm.fn[g + NA * j] = fma(st[j].v, jf, f[j]);
            }
            // boundary faces: the trace equations take the boundary flux (faceint 1075-1246)
            if (bfe && bfe[fc] < 0) {
                Dual<1> wd[NC], uhd[NCH], fb[NCH];
                double nlq[ND];
#pragma unroll
                for (int d = 0; d < ND; d++) nlq[d] = sm.nl[g + NA * d];
#pragma unroll
                for (int c = 0; c < NC; c++) wd[c] = dc<1>(sm.ugf[g + NA * c]);
#pragma unroll
                for (int c = 0; c < NCH; c++) uhd[c] = dc<1>(w[c]);
                const int ib = -bfe[fc] - 1;
                if (!ns_fbou_dual<ND, 1, GEN>(A.bcm[ib], P, A.bcs + (size_t)ib * NCH, nlq, wd, uhd, fb, !A.inviscid,
                                              A.conv_stab, A.visc_model))
                    for (int j = 0; j < NCH; j++) fb[j] = dc<1>(0.0);
#pragma unroll
                for (int j = 0; j < NCH; j++) sm.fb[g + NA * j] = fb[j].v * jf;
            }
        }
        __syncthreads();
        // Rh: fhat on every face for the element equations, the boundary flux for the
        // trace equations of boundary faces
        for (int t = tid; t < NB; t += NTH) {
            const int j = t % NCH, fdof = t / NCH, fc = fdof / NPF, ip = fdof % NPF;
            double s = 0.0, b = 0.0;
            const bool bnd = bfe && bfe[fc] < 0;
#pragma unroll 4
            for (int q = 0; q < NGF; q++) {
                const double w = __ldg(&T.shapfg[ip + NPF * q]);
                s = fma(w, sm.fn[q + NGF * fc + NA * j], s);
                if (bnd) b = fma(w, sm.fb[q + NGF * fc + NA * j], b);
            }
            sm.rh[t] = -s;
            A.Ro[(size_t)e * NB + t] = bnd ? -b : -s;
        }
        __syncthreads();
        double ru2 = 0.0;
        for (int t = tid; t < N; t += NTH) {
            const int i = t % NPV, j = t / NPV;
            double sp[ND1];
#pragma unroll
            for (int r = 0; r < ND1; r++) sp[r] = 0.0;
#pragma unroll 4
            for (int g = 0; g < NGV; g++)
#pragma unroll
                for (int r = 0; r < ND1; r++)
                    sp[r] = fma(__ldg(&T.shapvg[i + NPV * (g + NGV * r)]), sm.wrk[g + NGV * r + NQ * j], sp[r]);
            double s = 0.0;
#pragma unroll
            for (int r = 0; r < ND1; r++) s += sp[r];
            for (int c = 0; c < sm.inc_n[i]; c++) s += sm.rh[j + NCH * sm.inc_f[i * S::MAXINC + c]];
            A.Ru[(size_t)e * N + t] = s;
            ru2 += s * s;
        }
        const double tot = block_sum(ru2, sm.red);
        if (tid == 0) A.ru2[e] = tot;
    }
}

}  // namespace hfem
