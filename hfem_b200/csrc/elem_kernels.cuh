// Shared pieces of the HDG element kernels for sm_100a: element shapes and
// arguments, geometry and q-equation matrices, the Cholesky helpers, the
// face-block scatter, q recovery and the solution update.
// The element assembly itself is element_kernel (elem_kernel.cuh).
//
// Structure of the element blocks (restating elementassembly.cpp faceint
// 717-1321): every face contribution to the element equations is the
// trace-equation entry lifted to the element node that carries the face dof,
//   D = D_vol + P K,   F = F_vol + P H,   Ru = Ru_vol + P Rh,
// where P (npv x ndf) is the incidence perm[fdof] = node.
#pragma once
#include <cuda_runtime.h>
#include "ns_flux.cuh"
#include "schur_kernels.cuh"

namespace hfem {

template <int ND_, int NPV_, int NPF_, int NGV_, int NGF_>
struct Shape {
    static constexpr int ND = ND_, NPV = NPV_, NPF = NPF_, NGV = NGV_, NGF = NGF_;
    static constexpr int NFE = ND + 1, NCU = ND + 2, NC = NCU * (ND + 1), NCH = NCU;
    static constexpr int NDF = NPF * NFE, ND1 = ND + 1, N = NPV * NCU, NB = NCH * NDF, BSZ = NCH * NPF;
    static constexpr int NA = NGF * NFE;          // face points of one element
    static constexpr int NQ = NGV * ND1;          // (volume point, derivative) pairs
    static constexpr int MAXINC = ND;             // faces meeting at a node
    // threads per CTA of the element kernel, at 512 threads per SM: the phases of a
    // small element have too little work for 8 warps, so more and smaller CTAs per SM
    // overlap their barriers and latencies.  Measured (ms, 64 / 128 / 256 threads):
    // 2D p1, 7,200 elements 0.130 / 0.173 / 0.311; 2D p2, 2,048: 0.081 / 0.108 / 0.133;
    // 3D p1, 10,368: 0.56 / 0.60 / 0.86; 2D p3, 4,050 (Roe, Sutherland): 0.45 / 0.35 /
    // 0.44; 2D p4, 7,938: 0.88 / 0.76 / 1.00; 3D p2, 4,374: 1.41 / 0.96 / 1.11; 3D p3,
    // 4,374: 7.3 / 4.2 / 3.1.  (Caps of 640 to 1,024 threads per SM: slower, spills.)
    static constexpr int NT = N <= 24 ? 64 : (N <= 60 ? 128 : 256);
};

struct Tables {                 // master element tables, reference layouts
    const double *shapvt, *shapvg, *svsv, *shapft, *shapfg, *sfsf;
    const int* perm;            // nfe x npf
};

struct ElemArgs {
    Tables T;
    const double* dgnodes;      // ne x nd x npv
    const int* elcon;           // ne x ndf
    const double *udg, *uh, *sh;
    double param[6];
    int tdep;
    double fc_u, fc_q;
    int ne;
    double *D, *F, *K, *H, *Ru, *Rh, *Ro, *ru2;
    double* ws;                 // gridDim.x workspace slots of EK<S>::WS (3xTF32: WS_TF) doubles (element_kernel)
    // several problems in one mesh (NULL = the uniform values above): element ->
    // problem, and per problem [gamma, eps, Re, Pr, Mach, tau, tdep, fc_u]
    const int* eprob;
    const double* pparam;
    // boundary faces (NULL bf = none): bf[e * nfe + face] < 0 is boundary -(ib + 1),
    // condition bcm[ib] (fbou.cpp types 1, 2, 5, 6, 7) with state bcs[ib * nch + c]
    const int* bf;
    const int* bcm;
    const double* bcs;
    int inviscid;               // 1: Euler flux (app.appname 0)
    int* err = nullptr;         // set to 2 when a bulk-copy wait expires (NULL: not recorded)
    int conv_stab = 0;          // app.convStabMethod: 0 constant tau, 1 Lax-Friedrichs, 2 Roe
    int visc_model = 0;         // app.viscosityModel: 0 constant, 1 Sutherland's law
    int e_begin = 0;            // element range [e_begin, ne) of this launch
};


// --------------------------------------------------------------- helpers
__device__ __forceinline__ double block_sum(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) s += red[i];
    return s;                   // valid on thread 0
}

// Geometry at volume and face points (elementassembly.cpp:11-237).
template <class S>
__device__ void geometry(const Tables& T, const double* x, double* jac, double* Xx, double* jacf, double* nl) {
    constexpr int ND = S::ND, NPV = S::NPV, NGV = S::NGV, NGF = S::NGF, NPF = S::NPF, NA = S::NA;
    for (int g = threadIdx.x; g < NGV + NA; g += blockDim.x) {
        if (g < NGV) {
            double J[ND][ND];
#pragma unroll
            for (int d = 0; d < ND; d++)
#pragma unroll
                for (int i = 0; i < ND; i++) {
                    double s = 0.0;
                    for (int a = 0; a < NPV; a++) s += T.shapvt[g + NGV * (a + NPV * (i + 1))] * x[a + NPV * d];
                    J[d][i] = s;
                }
            double adj[ND][ND], det;
            if constexpr (ND == 2) {
                det = J[0][0] * J[1][1] - J[0][1] * J[1][0];
                adj[0][0] = J[1][1]; adj[0][1] = -J[0][1];
                adj[1][0] = -J[1][0]; adj[1][1] = J[0][0];
            } else {
                adj[0][0] = J[1][1] * J[2][2] - J[1][2] * J[2][1];
                adj[0][1] = J[0][2] * J[2][1] - J[0][1] * J[2][2];
                adj[0][2] = J[0][1] * J[1][2] - J[0][2] * J[1][1];
                adj[1][0] = J[1][2] * J[2][0] - J[1][0] * J[2][2];
                adj[1][1] = J[0][0] * J[2][2] - J[0][2] * J[2][0];
                adj[1][2] = J[0][2] * J[1][0] - J[0][0] * J[1][2];
                adj[2][0] = J[1][0] * J[2][1] - J[1][1] * J[2][0];
                adj[2][1] = J[0][1] * J[2][0] - J[0][0] * J[2][1];
                adj[2][2] = J[0][0] * J[1][1] - J[0][1] * J[1][0];
                det = J[0][0] * adj[0][0] + J[0][1] * adj[1][0] + J[0][2] * adj[2][0];
            }
            jac[g] = det;
#pragma unroll
            for (int d = 0; d < ND; d++)
#pragma unroll
                for (int i = 0; i < ND; i++) Xx[g + NGV * (d + ND * i)] = adj[i][d];
        } else {
            const int gg = g - NGV, fc = gg / NGF, q = gg % NGF;
            double Tt[ND][ND - 1];
#pragma unroll
            for (int d = 0; d < ND; d++)
#pragma unroll
                for (int r = 0; r < ND - 1; r++) {
                    double s = 0.0;
                    for (int m = 0; m < NPF; m++)
                        s += T.shapft[q + NGF * (m + NPF * (r + 1))] * x[T.perm[fc * NPF + m] + NPV * d];
                    Tt[d][r] = s;
                }
            double nv[ND];
            if constexpr (ND == 2) {
                nv[0] = Tt[1][0];
                nv[1] = -Tt[0][0];
            } else {
                nv[0] = Tt[1][0] * Tt[2][1] - Tt[2][0] * Tt[1][1];
                nv[1] = Tt[2][0] * Tt[0][1] - Tt[0][0] * Tt[2][1];
                nv[2] = Tt[0][0] * Tt[1][1] - Tt[1][0] * Tt[0][1];
            }
            double j = 0.0;
#pragma unroll
            for (int d = 0; d < ND; d++) j += nv[d] * nv[d];
            j = sqrt(j);
            jacf[gg] = j;
#pragma unroll
            for (int d = 0; d < ND; d++) nl[gg + NA * d] = nv[d] / j;
        }
    }
}

// q-equation matrices (elementassembly.cpp:1323-1412): M (npv^2), C (npv^2 nd), E (npv ndf nd).
template <class S>
__device__ void qmatrices(const Tables& T, double fc_q, const double* jac, const double* Xx, const double* jacf,
                          const double* nl, double* M, double* C, double* E) {
    constexpr int ND = S::ND, NPV = S::NPV, NGV = S::NGV, NGF = S::NGF, NPF = S::NPF, NA = S::NA, NDF = S::NDF;
    constexpr int NPV2 = NPV * NPV, NPF2 = NPF * NPF;
    for (int t = threadIdx.x; t < NPV2 * (ND + 1); t += blockDim.x) {
        const int r = t % NPV2, d = t / NPV2;
        if (d == 0) {
            double s = 0.0;
            for (int g = 0; g < NGV; g++) s += T.svsv[r + NPV2 * g] * jac[g];
            M[r] = fc_q * s;
        } else {
            double c = 0.0;
            for (int i = 0; i < ND; i++)
                for (int g = 0; g < NGV; g++)
                    c += T.svsv[r + NPV2 * (g + NGV * (i + 1))] * Xx[g + NGV * ((d - 1) + ND * i)];
            C[r + NPV2 * (d - 1)] = c;
        }
    }
    for (int t = threadIdx.x; t < NPV * NDF * ND; t += blockDim.x) E[t] = 0.0;
    __syncthreads();
    for (int t = threadIdx.x; t < ND * NDF * NPF; t += blockDim.x) {
        const int k = t % NPF, j = (t / NPF) % NPF, fc = (t / NPF2) % S::NFE, d = t / (NPF2 * S::NFE);
        double s = 0.0;
        for (int g = 0; g < NGF; g++)
            s += T.sfsf[(k + NPF * j) + NPF2 * g] * nl[g + NGF * fc + NA * d] * jacf[g + NGF * fc];
        E[T.perm[fc * NPF + k] + NPV * ((fc * NPF + j) + NDF * d)] = s;
    }
}

// The same matrices for the element kernel's FP64 form, from the factors held in
// shared memory instead of the product tables (307 KB of svsv for the
// tetrahedron p = 3, re-read from L2 for every element): with
//   P_0(b, g) = fc_q shapvg(b, g) jac(g),  P_d(b, g) = sum_i shapvg(b, (g, i)) Xx(g; d, i)
// M and C_d are the products P_d phi', npv (nd + 1) rows by npv columns, on the
// FP64 tensor cores; E's entries are shapfg shapfc sums with shapfg and shapfc
// from shared memory.  av(b, q) = shapvg, af(k, g) = shapfg, sfc = shapfc.
template <class S, int NTHR, class AV, class AF>
__device__ __forceinline__ void qmatrices_factored(const Tables& T, double fc_q, const double* jac, const double* Xx,
                                                   const double* jacf, const double* nl, AV av, AF af,
                                                   const double* sfc, const int* perm, double* M, double* C, double* E) {
    constexpr int ND = S::ND, NPV = S::NPV, NGV = S::NGV, NGF = S::NGF, NPF = S::NPF, NA = S::NA, NDF = S::NDF;
    constexpr int NR = NPV * (ND + 1), MT = (NR + 7) / 8, KS = (NGV + 3) / 4, NTN = (NPV + 7) / 8;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gr = lane >> 2, gc = lane & 3;
    for (int t = threadIdx.x; t < NPV * NDF * ND; t += NTHR) E[t] = 0.0;
    double bf[KS][NTN];
#pragma unroll
    for (int ks = 0; ks < KS; ks++)
#pragma unroll
        for (int b = 0; b < NTN; b++) {
            const int g = 4 * ks + gc, a = 8 * b + gr;
            bf[ks][b] = (g < NGV && a < NPV) ? __ldg(&T.shapvt[g + NGV * a]) : 0.0;
        }
    for (int mt = warp; mt < MT; mt += NTHR / 32) {
        const int r = 8 * mt + gr, b = r % NPV, d = r / NPV;
        double acc[NTN][2];
#pragma unroll
        for (int n = 0; n < NTN; n++) acc[n][0] = acc[n][1] = 0.0;
#pragma unroll
        for (int ks = 0; ks < KS; ks++) {
            const int g = 4 * ks + gc;
            double a = 0.0;
            if (g < NGV && r < NR) {
                if (d == 0) {
                    a = av(b, g) * (fc_q * jac[g]);
                } else {
#pragma unroll
                    for (int i = 0; i < ND; i++) a += av(b, g + NGV * (i + 1)) * Xx[g + NGV * ((d - 1) + ND * i)];
                }
            }
#pragma unroll
            for (int n = 0; n < NTN; n++) dmma8x8x4(acc[n][0], acc[n][1], a, bf[ks][n]);
        }
        if (r < NR)
#pragma unroll
            for (int n = 0; n < NTN; n++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int a = 8 * n + 2 * gc + h;
                    if (a < NPV) (d == 0 ? M : C + NPV * NPV * (d - 1))[b + NPV * a] = acc[n][h];
                }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < ND * NDF * NPF; t += NTHR) {
        const int k = t % NPF, j = (t / NPF) % NPF, fc = (t / (NPF * NPF)) % S::NFE, d = t / (NPF * NPF * S::NFE);
        double s = 0.0;
#pragma unroll 4
        for (int g = 0; g < NGF; g++)
            s += af(k, g) * sfc[g + NGF * j] * (nl[g + NGF * fc + NA * d] * jacf[g + NGF * fc]);
        E[perm[fc * NPF + k] + NPV * ((fc * NPF + j) + NDF * d)] = s;
    }
}

// Lower Cholesky of M (npv x npv) in place by one warp, right-looking: lane i
// holds row i in registers, so a column costs one reciprocal square root and one
// shuffle per entry of its row instead of a dot product over the columns before
// it; rdg receives the reciprocals of the diagonal.
template <int NPV>
__device__ __forceinline__ void cholesky_warp_rows(double* a, double* rdg) {
    static_assert(NPV <= 32, "one row per lane");
    const int lane = threadIdx.x & 31, row = lane < NPV ? lane : NPV - 1;
    double r[NPV];
#pragma unroll
    for (int k = 0; k < NPV; k++) r[k] = a[row + NPV * k];
#pragma unroll
    for (int j = 0; j < NPV; j++) {
        const double inv = rsqrt(__shfl_sync(0xffffffffu, r[j], j));
        if (lane == j) rdg[j] = inv;
        r[j] *= inv;
#pragma unroll
        for (int k = j + 1; k < NPV; k++) r[k] = fma(-r[j], __shfl_sync(0xffffffffu, r[j], k), r[k]);
    }
    if (lane < NPV)
#pragma unroll
        for (int k = 0; k < NPV; k++)
            if (k <= lane) a[lane + NPV * k] = r[k];
}

// Lower Cholesky of M (npv x npv) in place, one warp; rdg (if given) receives
// the reciprocals of the diagonal.
template <int NPV>
__device__ void cholesky_warp(double* a, double* rdg = nullptr) {
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    for (int j = 0; j < NPV; j++) {
        if (lane == 0) {
            double s = a[j + NPV * j];
            for (int k = 0; k < j; k++) s -= a[j + NPV * k] * a[j + NPV * k];
            a[j + NPV * j] = sqrt(s);
            if (rdg) rdg[j] = 1.0 / a[j + NPV * j];
        }
        __syncwarp();
        const double djj = a[j + NPV * j];
        for (int i = j + 1 + lane; i < NPV; i += 32) {
            double t = a[i + NPV * j];
            for (int k = 0; k < j; k++) t -= a[i + NPV * k] * a[j + NPV * k];
            a[i + NPV * j] = t / djj;
        }
        __syncwarp();
    }
}

// --------------------------------------------------------------- scatter
// Owner-gather into the face-block system (globalassembly.cpp:40-89): every
// Hg entry sums its (at most two) element contributions in ascending element
// order, exactly the order of the reference's serial element loop.
struct ScatterArgs {
    int nblk, nf, npf, nch, nfe, nb;
    const int* blk_src;        // nblk x 2 x 3: (element, a, b) or -1
    const int* face_src;       // nf x 2 x 2: (element, a) or -1
    const int* elcon;          // ne x ndf
    const int* rowface;        // nblk: row face i of block k
    const int* colface;        // nblk: column face j of block k
    const double *H, *Rh, *Ro;
    double *Hg, *Rg, *Rr;
};

// Rg (condensed Rh, when A.Rg) and Rr (Rh before condensation) by the threads of the grid.
static __device__ __forceinline__ void scatter_R(const ScatterArgs& A) {
    const int bsz = A.npf * A.nch, ndf = A.npf * A.nfe;
    const int total = A.nf * bsz;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const int i = t / bsz, w = t % bsz, m1 = w / A.nch, n1 = w % A.nch;
        double s = 0.0, so = 0.0;
        for (int c = 0; c < 2; c++) {
            const int e = A.face_src[(i * 2 + c) * 2 + 0];
            if (e < 0) break;
            const int a = A.face_src[(i * 2 + c) * 2 + 1];
            const int ind = A.elcon[(size_t)e * ndf + a * A.npf + m1] - i * A.npf;
            const size_t idx = (size_t)e * A.nb + a * bsz + ind * A.nch + n1;
            if (A.Rg) s += A.Rh[idx];
            if (A.Ro) so += A.Ro[idx];
        }
        if (A.Rg) A.Rg[t] = s;
        if (A.Rr) A.Rr[t] = so;
    }
}

static __global__ void scatter_R_kernel(ScatterArgs A) { scatter_R(A); }

// Scatter of the condensed blocks into Hg (mapElement2LinearSystem,
// globalassembly.cpp:40-89) as an owner-gather, one warp per Hg block, face shape known
// at compile time: the warp first resolves, for each (at most two) contributing
// element, the offsets of the block's rows and columns inside that element's H
// (elcon gives the permutation of the face nodes).  A lane keeps its rows' offsets in
// registers and walks the columns (32 / BSZ at a time for small blocks), eight of
// them in flight; off-diagonal blocks, with one element, take a loop without the
// second one.  The vectors Rg and Rr are scattered by the same launch.  Bound by HBM,
// H read and Hg written once (us, with one element a time and 8-byte gathers behind
// a table look-up each): 13,182 3D p3 1,735 -> 1,577 (5.0 TB/s), 4,374 3D p2 304 ->
// 207, 7,938 2D p4 138 -> 109, 4,050 2D p3 52 -> 35.
template <int NPF, int NCH, int NFE>
static __global__ void __launch_bounds__(256) scatter_H_block_kernel(ScatterArgs A) {
    constexpr int BSZ = NPF * NCH, NDF = NPF * NFE, NB = NDF * NCH;
    constexpr int WARPS = 8;
    constexpr int G = BSZ <= 16 ? 32 / BSZ : 1, R = (BSZ + 31) / 32;
    __shared__ int s_col[WARPS][2][BSZ];
    __shared__ int s_row[WARPS][2][NPF];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = G > 1 ? lane / BSZ : 0, r0 = G > 1 ? lane % BSZ : lane;
    const bool on = g < G;
    scatter_R(A);
    for (int k = blockIdx.x * WARPS + w; k < A.nblk; k += gridDim.x * WARPS) {
        const int i = A.rowface[k], j = A.colface[k];
        const int* src = A.blk_src + (size_t)k * 6;
        const int e0 = src[0], e1 = src[3], n = e0 < 0 ? 0 : (e1 < 0 ? 1 : 2);
        for (int t = lane; t < n * NPF; t += 32) {
            const int c = t / NPF, m = t % NPF, e = src[3 * c], a = src[3 * c + 1];
            s_row[w][c][m] = a * BSZ + (A.elcon[(size_t)e * NDF + a * NPF + m] - i * NPF) * NCH;
        }
        for (int t = lane; t < n * BSZ; t += 32) {
            const int c = t / BSZ, q = t % BSZ, m = q / NCH, e = src[3 * c], b = src[3 * c + 2];
            s_col[w][c][q] = NB * (b * BSZ + (A.elcon[(size_t)e * NDF + b * NPF + m] - j * NPF) * NCH + q % NCH);
        }
        __syncwarp();
        double* out = A.Hg + (size_t)k * BSZ * BSZ;
        const double* h0 = A.H + (size_t)(n > 0 ? e0 : 0) * NB * NB;
        const double* h1 = A.H + (size_t)(n > 1 ? e1 : 0) * NB * NB;
        int o0[R], o1[R];
#pragma unroll
        for (int t = 0; t < R; t++) {
            const int r = r0 + 32 * t, m = r < BSZ ? r / NCH : 0, q = r < BSZ ? r % NCH : 0;
            o0[t] = n > 0 ? s_row[w][0][m] + q : 0;
            o1[t] = n > 1 ? s_row[w][1][m] + q : 0;
        }
        if (n == 1) {
#pragma unroll 8
            for (int c = g; c < BSZ; c += G) {
                const int cc = s_col[w][0][c];
#pragma unroll
                for (int t = 0; t < R; t++)
                    if (on && r0 + 32 * t < BSZ) out[c * BSZ + r0 + 32 * t] = __ldg(&h0[o0[t] + cc]);
            }
        } else {
#pragma unroll 8
            for (int c = g; c < BSZ; c += G) {
#pragma unroll
                for (int t = 0; t < R; t++) {
                    if (!on || r0 + 32 * t >= BSZ) continue;
                    double s = 0.0;
                    if (n > 0) s += __ldg(&h0[o0[t] + s_col[w][0][c]]);
                    if (n > 1) s += __ldg(&h1[o1[t] + s_col[w][1][c]]);
                    out[c * BSZ + r0 + 32 * t] = s;
                }
            }
        }
        __syncwarp();
    }
}

// ------------------------------------------------------ q recovery / update
struct QArgs {
    Tables T;
    const double* dgnodes;
    const int* elcon;
    double* udg;                // u read, q written
    const double *uh, *sh;
    double fc_q;
    int ne;
    // optional update before the q solve: u += alpha (DinvRu - DinvF duh_e)
    const double *DinvRu, *DinvF, *duh;
    double alpha;
    const int* eprob;           // per-problem step lengths (NULL: alpha for all)
    const double* palpha;
};

constexpr int QT = 128;         // threads per CTA of the q recovery

template <class S>
struct QSmem {
    double x[S::NPV * S::ND];
    double jac[S::NGV], Xx[S::NGV * S::ND * S::ND];
    double jacf[S::NA], nl[S::NA * S::ND];
    double M[S::NPV * S::NPV], rdg[S::NPV];
    double u[S::NPV * S::NCU], ug[S::NGV * S::NCU];
    double uhe[S::NDF * S::NCH], uhq[S::NA * S::NCH];
    double de[S::NB], part[QT > S::N ? QT / S::N * S::N : S::N];
    double q[S::NPV * S::NCU * S::ND];
    int perm[S::NDF];
    int inc_n[S::NPV];
    int inc_f[S::NPV * S::MAXINC];
};

// Cholesky solves L L' x = b for one column held in registers, in the axpy
// (column) form: after x_j is final every later entry takes its update, so each
// step has up to npv - 1 independent FMAs; rdg holds 1 / L(j, j).
template <int NPV>
__device__ __forceinline__ void chol_solve_col_axpy(const double* lm, const double* rdg, double* col) {
    const volatile double* l = lm;
    double x[NPV];
#pragma unroll
    for (int i = 0; i < NPV; i++) x[i] = col[i];
#pragma unroll
    for (int j = 0; j < NPV; j++) {
        x[j] *= rdg[j];
#pragma unroll
        for (int i = j + 1; i < NPV; i++) x[i] = fma(-l[i + NPV * j], x[j], x[i]);
    }
#pragma unroll
    for (int j = NPV - 1; j >= 0; j--) {
        x[j] *= rdg[j];
#pragma unroll
        for (int i = 0; i < j; i++) x[i] = fma(-l[j + NPV * i], x[j], x[i]);
    }
#pragma unroll
    for (int i = 0; i < NPV; i++) col[i] = x[i];
}

// getQ (elementassembly.cpp:1414-1479), optionally preceded by getU
// (solutionupdate.cpp:6-68).  The right-hand side C u - E uhat is summed from u and
// uhat at the quadrature points (C and E themselves, 72 products for each of 1,200
// entries of the tetrahedron p = 3, are not formed), the source's part of q is added
// after the solve, D^-1 F duh is read by all threads, several columns each, and the
// factorisation runs under the sums.  Bound by HBM in the update (D^-1 F once).
// 1,296 tetrahedra p = 3: getQ 205 -> 70 us, with the update 242 -> 123 us.
template <class S>
static __global__ void __launch_bounds__(QT) getq_kernel(QArgs A) {
    constexpr int ND = S::ND, NPV = S::NPV, NPF = S::NPF, NGV = S::NGV, NGF = S::NGF, NA = S::NA;
    constexpr int NCU = S::NCU, NC = S::NC, NCH = S::NCH, NDF = S::NDF, N = S::N, NB = S::NB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    QSmem<S>& sm = *reinterpret_cast<QSmem<S>*>(smem_raw);
    const Tables& T = A.T;
    const int tid = threadIdx.x;
    for (int t = tid; t < NDF; t += QT) sm.perm[t] = T.perm[t];
    __syncthreads();
    for (int i = tid; i < NPV; i += QT) {
        int c = 0;
        for (int f = 0; f < NDF; f++)
            if (sm.perm[f] == i && c < S::MAXINC) sm.inc_f[i * S::MAXINC + c++] = f;
        sm.inc_n[i] = c;
    }
    for (int e = blockIdx.x; e < A.ne; e += gridDim.x) {
        __syncthreads();
        double* ue = A.udg + (size_t)e * NPV * NC;
        for (int t = tid; t < NPV * ND; t += QT) sm.x[t] = A.dgnodes[(size_t)e * NPV * ND + t];
        for (int t = tid; t < NDF * NCH; t += QT) {
            const int fn = t / NCH, c = t % NCH;
            const int gd = A.elcon[(size_t)e * NDF + fn];
            sm.uhe[fn + NDF * c] = A.uh[(size_t)gd * NCH + c];
            if (A.DinvF) sm.de[fn * NCH + c] = A.duh[(size_t)gd * NCH + c];
        }
        __syncthreads();
        if (A.DinvF) {
            // u += alpha (D^-1 Ru - D^-1 F duh): thread (row, group), groups of columns
            constexpr int G = QT / N > 0 ? QT / N : 1;
            const double alpha = A.palpha ? A.palpha[A.eprob[e]] : A.alpha;
            const double* df = A.DinvF + (size_t)e * N * NB;
            for (int t = tid; t < N * G; t += QT) {
                const int row = t % N, g = t / N;
                double s[4] = {0.0, 0.0, 0.0, 0.0};
                int c = g;
#pragma unroll 4
                for (; c + 3 * G < NB; c += 4 * G)
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        s[k] = fma(__ldg(&df[row + (size_t)N * (c + k * G)]), sm.de[c + k * G], s[k]);
                for (; c < NB; c += G) s[0] = fma(__ldg(&df[row + (size_t)N * c]), sm.de[c], s[0]);
                sm.part[t] = (s[0] + s[1]) + (s[2] + s[3]);
            }
            __syncthreads();
            for (int t = tid; t < N; t += QT) {
                double s = 0.0;
#pragma unroll
                for (int g = 0; g < G; g++) s += sm.part[t + N * g];
                double v = ue[t];
                v += -alpha * s;
                v += alpha * A.DinvRu[(size_t)e * N + t];
                ue[t] = v;
                sm.u[t] = v;
            }
        } else {
            for (int t = tid; t < N; t += QT) sm.u[t] = ue[t];
        }
        geometry<S>(T, sm.x, sm.jac, sm.Xx, sm.jacf, sm.nl);
        __syncthreads();
        // M, and u and uhat at the points
        for (int t = tid; t < NPV * NPV; t += QT) {
            const int i = t % NPV, a = t / NPV;
            double s = 0.0;
#pragma unroll 4
            for (int g = 0; g < NGV; g++)
                s = fma(__ldg(&T.shapvg[i + NPV * g]) * sm.jac[g], __ldg(&T.shapvt[g + NGV * a]), s);
            sm.M[t] = A.fc_q * s;
        }
        for (int t = tid; t < NGV * NCU; t += QT) {
            const int g = t % NGV, c = t / NGV;
            double s = 0.0;
#pragma unroll 4
            for (int a = 0; a < NPV; a++) s = fma(__ldg(&T.shapvt[g + NGV * a]), sm.u[a + NPV * c], s);
            sm.ug[t] = s;
        }
        for (int t = tid; t < NA * NCH; t += QT) {
            const int gg = t % NA, c = t / NA, fc = gg / NGF, q = gg % NGF;
            double s = 0.0;
#pragma unroll 4
            for (int m = 0; m < NPF; m++) s = fma(__ldg(&T.shapft[q + NGF * m]), sm.uhe[fc * NPF + m + NDF * c], s);
            sm.uhq[t] = s * sm.jacf[gg];
        }
        __syncthreads();
        // the last warp factors M while the others form the right-hand sides
        if (tid >= QT - 32) {
            cholesky_warp_rows<NPV>(sm.M, sm.rdg);
        } else {
            for (int t = tid; t < NPV * NCU * ND; t += QT - 32) {
                const int i = t % NPV, c = (t / NPV) % NCU, d = t / (NPV * NCU);
                double sp[ND];
#pragma unroll
                for (int r = 0; r < ND; r++) sp[r] = 0.0;
#pragma unroll 4
                for (int g = 0; g < NGV; g++) {
                    const double v = sm.ug[g + NGV * c];
#pragma unroll
                    for (int r = 0; r < ND; r++)
                        sp[r] = fma(__ldg(&T.shapvg[i + NPV * (g + NGV * (r + 1))]) * sm.Xx[g + NGV * (d + ND * r)], v,
                                    sp[r]);
                }
                double s = 0.0;
#pragma unroll
                for (int r = 0; r < ND; r++) s += sp[r];
                for (int k = 0; k < sm.inc_n[i]; k++) {
                    const int f = sm.inc_f[i * S::MAXINC + k], fc = f / NPF, ip = f % NPF;
                    double b = 0.0;
#pragma unroll 4
                    for (int q = 0; q < NGF; q++) {
                        const int gg = q + NGF * fc;
                        b = fma(__ldg(&T.shapfg[ip + NPF * q]) * sm.nl[gg + NA * d], sm.uhq[gg + NA * c], b);
                    }
                    s -= b;
                }
                sm.q[t] = s;
            }
        }
        __syncthreads();
        for (int t = tid; t < NCU * ND; t += QT) chol_solve_col_axpy<NPV>(sm.M, sm.rdg, &sm.q[NPV * t]);
        __syncthreads();
        const double* she = A.sh + (size_t)e * NPV * NC;
        for (int t = tid; t < NPV * NCU * ND; t += QT) {
            const int i = t % NPV, c = (t / NPV) % NCU, d = t / (NPV * NCU);
            const int at = i + NPV * (NCU * (1 + d) + c);
            ue[at] = sm.q[t] + she[at];
        }
    }
}

static __global__ void axpy_kernel(long long n, double alpha, const double* x, double* y) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] += alpha * x[i];
}

// y += alpha[prob[i / per]] x  (per-problem step lengths on the trace unknowns)
static __global__ void axpy_prob_kernel(long long n, int per, const int* __restrict__ prob, const double* __restrict__ alpha,
                                 const double* x, double* y) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] += alpha[prob[i / per]] * x[i];
}

}  // namespace hfem
