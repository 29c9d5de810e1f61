// One restart cycle of the segmented GMRES in a single cooperative kernel, for
// systems whose Arnoldi steps are bound by launch and memory latency (sm_100a).
//
// One CTA per SM owns a contiguous range of block rows and its slice of every
// basis vector (in shared memory when it fits, else in L2).  An Arnoldi step is
//   product  w = M^-1 Hg V_j on the CTA's rows, a warp per row; meanwhile
//            warp 0 sums |V_j| and, in the CTA that owns the problem's first piece, runs
//            step j-1's Givens rotation and stopping test
//   BAR 1    h1 = V^T w from all pieces' partial sums; w -= V h1; V^T w again
//   BAR 2    h2 likewise; V_{j+1} = w - V h2 to global memory, its norm's partial
//   BAR 3
// the same classical Gram-Schmidt applied twice, and the same lazily scaled basis,
// as the kernels of krylov_seg.cuh.  Every CTA sums the partials it needs itself,
// in piece order, so no second reduction stage and no broadcast is waited for, and
// all CTAs see the same values.  The stopping tests of step j-1 are read after
// BAR 1 of step j, so a cycle ends without the host.
//
// Measured (B200): 36,864 unknowns of 2D p = 2, 62 steps, 1.15 ms against 2.9 ms
// with the four launches per step of krylov_seg.cuh; eight problems of 104k unknowns
// together, 74 steps, 2.2 against 4.2 ms.
//
// EXT (block size 50): the product stays a launch of its own, one CTA per row (rows
// of 140 KB streamed by the cycle's CTAs took 105 us a step against 74), and the
// kernel is one step's orthogonalisation, the unscaled w read from V_{j+1}: 129,600 unknowns of
// 3D p = 3, 32 us a step against 41 us with the three launches of krylov_seg.cuh.
//
// Barriers spin on a counter in global memory; the launch is cooperative, so all
// CTAs are resident, and every spin is bounded: on expiry the kernel sets err and
// returns.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>
#include "krylov_seg.cuh"

namespace hfem {

constexpr int CYC_THREADS = 768;
constexpr int CYC_WARPS = CYC_THREADS / 32;
constexpr int CYC_MAXP = 8;             // pieces (problems) one CTA's rows may span
constexpr int CYC_MAXR = 100;           // largest restart
constexpr int CYC_MAXL = 2304;          // most entries of one CTA's slice
constexpr int CYC_R = CYC_MAXL / CYC_THREADS;

struct CycleArgs {
    const int *rowstart, *colidx;
    const double* Hg;
    const void* Minv;                   // NULL: no preconditioner
    double* V;
    long long n;
    const int* cp0;                     // per CTA (gridDim.x + 1): first piece
    const int* prow;                    // per piece (npieces + 1): first row
    const int* pseg;                    // segment of each piece
    const int* seg_p0;                  // per segment: first piece
    int npieces;
    double *part1, *part2, *partn;      // partial sums: (restart + 1) x npieces twice, npieces
    double *h1, *h2;                    // this step's projections, entry (i, seg) at i * P + seg
    unsigned* bar;                      // 3 counters, zero before a cycle
    int* err;
    int j0, j1;                         // steps of this launch (EXT: one; else 0, restart)
    int lmax;                           // entries of the largest slice
    int vcache;                         // the slices of V fit in shared memory
};

// Dynamic shared memory in doubles: w, per-piece column factors and coefficients,
// the warps' row buffers, and the slices of V
constexpr int CYC_YS = 64;              // one warp's row buffer: 32 / (BSZ / 2) groups of BSZ entries
inline size_t cyc_smem_doubles(int lmax, int restart, bool vcache) {
    return (size_t)lmax + 2 * CYC_MAXP * (size_t)(restart + 2) + (size_t)CYC_WARPS * CYC_YS +
           (vcache ? (size_t)lmax * (restart + 1) : 0);
}

// Barrier `which` (0, 1, 2 in turn) of the CTAs.  Each has its own counter, zero
// when the first CTA arrives; past barrier b every CTA has left barrier b - 1, so
// CTA 0 zeroes that counter for its next use.
__device__ __forceinline__ bool cyc_barrier(unsigned* bar, int which, int* err) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&bar[which], 1u);
        unsigned v = 0;
        int good = 0;
        for (int it = 0; it < (1 << 21); it++) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&bar[which]) : "memory");
            if (v >= gridDim.x) {
                good = 1;
                break;
            }
        }
        if (!good) atomicExch(err, 3);
        else if (blockIdx.x == 0) bar[(which + 2) % 3] = 0;
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// z = M^-1 (Hg x) on block row i by one warp, out(r, z_r); x is read through L2
// (other SMs wrote it in this kernel).  ys: the warp's buffer of CYC_YS doubles.
template <int BSZ, typename MT, class Out>
__device__ __forceinline__ void cyc_row(int i, const int* __restrict__ rowstart, const int* __restrict__ colidx,
                                        const double* __restrict__ Hg, const MT* __restrict__ Minv, const double* x,
                                        double* ys, Out out) {
    const int lane = threadIdx.x & 31;
    const int k0 = __ldg(&rowstart[i]), ncol = (__ldg(&rowstart[i + 1]) - k0) * BSZ;
    constexpr bool PAIRS = BSZ % 2 == 0;
    constexpr int L2 = PAIRS ? BSZ / 2 : BSZ, G = 32 / L2, MC = (BSZ + G - 1) / G;
    const int g = lane / L2, q = lane - g * L2;
    static_assert(G * BSZ <= CYC_YS, "row buffer");
    const bool on = g < G;
    const double* A = Hg + (size_t)k0 * BSZ * BSZ;
    double2 m[MC];
    if constexpr (PAIRS) {
        double a0 = 0.0, a1 = 0.0;
        if (on) {
#pragma unroll 6
            for (int cc = g; cc < ncol; cc += G) {
                const int kb = cc / BSZ, c = cc - kb * BSZ;
                const double xv = __ldcg(&x[(size_t)__ldg(&colidx[k0 + kb]) * BSZ + c]);
                const double2 av = ldg_pair(A + (size_t)cc * BSZ + 2 * q);
                a0 = fma(av.x, xv, a0);
                a1 = fma(av.y, xv, a1);
            }
            if (Minv)
#pragma unroll
                for (int t = 0; t < MC; t++) {
                    const int c = g + G * t;
                    m[t] = c < BSZ ? ldg_pair(Minv + (size_t)i * BSZ * BSZ + (size_t)c * BSZ + 2 * q)
                                   : make_double2(0.0, 0.0);
                }
            ys[g * BSZ + 2 * q] = a0;
            ys[g * BSZ + 2 * q + 1] = a1;
        }
    } else {
        double a0 = 0.0;
        if (on) {
#pragma unroll 8
            for (int cc = g; cc < ncol; cc += G) {
                const int kb = cc / BSZ, c = cc - kb * BSZ;
                const double xv = __ldcg(&x[(size_t)__ldg(&colidx[k0 + kb]) * BSZ + c]);
                a0 = fma(__ldg(&A[(size_t)cc * BSZ + q]), xv, a0);
            }
            if (Minv)
#pragma unroll
                for (int t = 0; t < MC; t++) {
                    const int c = g + G * t;
                    m[t].x = c < BSZ ? (double)__ldg(&Minv[(size_t)i * BSZ * BSZ + (size_t)c * BSZ + q]) : 0.0;
                }
            ys[g * BSZ + q] = a0;
        }
    }
    __syncwarp();
    double y = 0.0;
    if (lane < BSZ)
#pragma unroll
        for (int gg = 0; gg < G; gg++) y += ys[gg * BSZ + lane];
    __syncwarp();
    if (!Minv) {
        if (lane < BSZ) out(lane, y);
        return;
    }
    if (lane < BSZ) ys[lane] = y;
    __syncwarp();
    double b0 = 0.0, b1 = 0.0;
    if (on)
#pragma unroll
        for (int t = 0; t < MC; t++) {
            const int c = g + G * t;
            const double yc = c < BSZ ? ys[c] : 0.0;
            b0 = fma(m[t].x, yc, b0);
            if constexpr (PAIRS) b1 = fma(m[t].y, yc, b1);
        }
    __syncwarp();
    if (on) {
        if constexpr (PAIRS) {
            ys[g * BSZ + 2 * q] = b0;
            ys[g * BSZ + 2 * q + 1] = b1;
        } else {
            ys[g * BSZ + q] = b0;
        }
    }
    __syncwarp();
    double z = 0.0;
    if (lane < BSZ)
#pragma unroll
        for (int gg = 0; gg < G; gg++) z += ys[gg * BSZ + lane];
    __syncwarp();
    if (lane < BSZ) out(lane, z);
}

template <int BSZ, typename MT, bool EXT = false>
__global__ void __launch_bounds__(CYC_THREADS, 1) gmres_cycle_kernel(CycleArgs A, GmState S) {
    extern __shared__ __align__(16) double cyc_sm[];
    __shared__ int run[CYC_MAXP], pseg[CYC_MAXP], pofs[CYC_MAXP + 1], s_any;
    __shared__ double s_nn[CYC_MAXP], red[CYC_WARPS];
    const int R = S.restart, P = S.P, R2 = R + 2;
    double* ws = cyc_sm;
    double* scs = ws + A.lmax;                       // factors of the basis columns, per own piece
    double* cf = scs + CYC_MAXP * R2;                // coefficients, per own piece
    double* ysall = cf + CYC_MAXP * R2;
    double* vsm = ysall + CYC_WARPS * CYC_YS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double* ys = ysall + warp * CYC_YS;
    const MT* Minv = static_cast<const MT*>(A.Minv);
    const int pc0 = A.cp0[blockIdx.x], npc = A.cp0[blockIdx.x + 1] - pc0;
    const int row0 = A.prow[pc0], nrow = A.prow[pc0 + npc] - row0, len = nrow * BSZ;
    double* Vg = A.V + (size_t)row0 * BSZ;           // this CTA's slice of column 0
    // column i of the slice: shared memory or global
    double* vb = A.vcache ? vsm : Vg;
    const size_t ldv = A.vcache ? (size_t)A.lmax : (size_t)A.n;
    if (tid <= npc) pofs[tid] = (A.prow[pc0 + tid] - row0) * BSZ;
    if (tid < npc) {
        pseg[tid] = A.pseg[pc0 + tid];
        run[tid] = S.act[pseg[tid]];
        for (int i = 0; i <= A.j0; i++) scs[tid * R2 + i] = S.sc[(size_t)i * P + pseg[tid]];
    }
    if (tid == 0) s_any = 0;
    __syncthreads();
    if constexpr (EXT) {
        for (int p = tid; p < P; p += CYC_THREADS)
            if (S.act[p]) s_any = 1;
        __syncthreads();
        if (!s_any) return;
    }
    if (A.vcache)
        for (int t = tid; t < len; t += CYC_THREADS) vsm[t] = Vg[t];
    __syncthreads();
    auto owner = [&](int c) { return A.seg_p0[pseg[c]] == pc0 + c; };

    // sum over the pieces of own piece c's segment of `cnt` rows of partials, into
    // fin(column, sum) by lane 0 of the warp that has the column
    auto gather = [&](int c, const double* part, int cnt, auto fin) {
        const int p0 = A.seg_p0[pseg[c]], p1 = A.seg_p0[pseg[c] + 1];
        for (int base = warp; base < cnt; base += 4 * CYC_WARPS) {
            double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
            for (int q = p0 + lane; q < p1; q += 32)
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (base + CYC_WARPS * u < cnt) t[u] += __ldcg(&part[(size_t)(base + CYC_WARPS * u) * A.npieces + q]);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (base + CYC_WARPS * u >= cnt) continue;
                t[u] = seg_warp_sum(t[u]);
                if (lane == 0) fin(base + CYC_WARPS * u, t[u]);
            }
        }
    };
    // <V_i, w> for i < k over own piece c: a warp per column (NC columns at a time
    // when there are more columns than warps), or SP warps per column when there are
    // few, their sums added through shared memory
    auto columns = [&](int c, int k, double* part, auto ncc) {
        constexpr int NC = decltype(ncc)::value;
        const int o0 = pofs[c], o1 = pofs[c + 1];
        for (int base = warp; base < k; base += NC * CYC_WARPS) {
            double t[NC];
#pragma unroll
            for (int u = 0; u < NC; u++) t[u] = 0.0;
            const double* vp = vb + (size_t)base * ldv;
#pragma unroll(NC == 1 ? 16 : 8)
            for (int i = o0 + lane; i < o1; i += 32) {
                const double x = ws[i];
#pragma unroll
                for (int u = 0; u < NC; u++)
                    if (base + CYC_WARPS * u < k) t[u] = fma(vp[(size_t)CYC_WARPS * u * ldv + i], x, t[u]);
            }
#pragma unroll
            for (int u = 0; u < NC; u++) {
                if (base + CYC_WARPS * u >= k) continue;
                t[u] = seg_warp_sum(t[u]);
                if (lane == 0) part[(size_t)(base + CYC_WARPS * u) * A.npieces + pc0 + c] = t[u];
            }
        }
    };
    auto dots = [&](int c, int k, double* part) {
        const int SP = k <= CYC_WARPS / 8 ? 8 : (k <= CYC_WARPS / 4 ? 4 : (k <= CYC_WARPS / 2 ? 2 : 1));
        if (SP == 1) {
            if (k <= CYC_WARPS) columns(c, k, part, std::integral_constant<int, 1>{});
            else columns(c, k, part, std::integral_constant<int, 2>{});
            return;
        }
        const int o0 = pofs[c], o1 = pofs[c + 1], i = warp / SP;
        double t = 0.0;
        if (i < k) {
            const double* vp = vb + (size_t)i * ldv;
#pragma unroll 8
            for (int q = o0 + 32 * (warp % SP) + lane; q < o1; q += 32 * SP) t = fma(vp[q], ws[q], t);
        }
        t = seg_warp_sum(t);
        __syncthreads();
        if (lane == 0) red[warp] = t;
        __syncthreads();
        if (tid < k) {
            double s = 0.0;
            for (int q = 0; q < SP; q++) s += red[tid * SP + q];
            part[(size_t)tid * A.npieces + pc0 + c] = s;
        }
    };
    // v[r] = scale(c) ws - sum_{i<k} cf_i V_i at this thread's entries
    auto update = [&](int k, bool scaled, double (&v)[CYC_R]) {
#pragma unroll
        for (int r = 0; r < CYC_R; r++) {
            const int i = tid + CYC_THREADS * r;
            v[r] = 0.0;
            if (i >= len) continue;
            int c = 0;
            while (i >= pofs[c + 1]) c++;
            if (!run[c]) continue;
            const double* cc = cf + c * R2;
            const double* vp = vb + i;
            double a[4] = {0.0, 0.0, 0.0, 0.0};
            int q = 0;
#pragma unroll 4
            for (; q + 4 <= k; q += 4)
#pragma unroll
                for (int u = 0; u < 4; u++) a[u] = fma(cc[q + u], vp[(size_t)(q + u) * ldv], a[u]);
            for (; q < k; q++) a[0] = fma(cc[q], vp[(size_t)q * ldv], a[0]);
            const double w = scaled ? scs[c * R2 + k - 1] * ws[i] : ws[i];
            v[r] = w - ((a[0] + a[1]) + (a[2] + a[3]));
        }
    };
    // |V_j| of the own pieces' problems and step j - 1's bookkeeping (warp 0)
    auto finish = [&](int j) {
        for (int c = 0; c < npc; c++) {
            if (!run[c]) continue;
            const int p0 = A.seg_p0[pseg[c]], p1 = A.seg_p0[pseg[c] + 1];
            double t = 0.0;
            for (int q = p0 + lane; q < p1; q += 32) t += __ldcg(&A.partn[q]);
            const double nn = sqrt(seg_warp_sum(t));
            if (lane == 0) s_nn[c] = nn;
            if (owner(c)) gm_givens_warp(S, pseg[c], j - 1, A.h1, A.h2, nn);
        }
        __syncwarp();
    };

    for (int j = A.j0; j < A.j1; j++) {
        // ---- product on the rows of running problems
        if constexpr (EXT) {
            for (int i = tid; i < len; i += CYC_THREADS) ws[i] = Vg[(size_t)(j + 1) * A.n + i];
        } else {
        if (warp == 0 && j > 0) finish(j);
        const double* x = A.V + (size_t)j * A.n;
        // warp 0 takes a row last: it has the norms to sum
        for (int r = CYC_WARPS - 1 - warp; r < nrow; r += CYC_WARPS) {
            int c = 0;
            while (r * BSZ >= pofs[c + 1]) c++;
            if (!run[c]) continue;
            cyc_row<BSZ, MT>(row0 + r, A.rowstart, A.colidx, A.Hg, Minv, x, ys,
                             [&](int q, double z) { ws[r * BSZ + q] = z; });
        }
        }
        __syncthreads();
        if (!EXT && j > 0 && tid < npc && run[tid]) scs[tid * R2 + j] = s_nn[tid] == 0.0 ? 1.0 : 1.0 / s_nn[tid];
        for (int c = 0; c < npc; c++)
            if (run[c]) dots(c, j + 1, A.part1);
        if (!cyc_barrier(A.bar, 0, A.err)) return;
        // ---- step j - 1's stopping tests
        if constexpr (!EXT) {
            if (tid == 0) s_any = 0;
            __syncthreads();
            for (int p = tid; p < P; p += CYC_THREADS)
                if (__ldcg(&S.act[p])) s_any = 1;
            if (tid < npc) run[tid] = __ldcg(&S.act[pseg[tid]]);
            __syncthreads();
            if (!s_any) return;
        }
        // ---- first projection: h1_i = sc_i sc_j <V_i, z>
        for (int c = 0; c < npc; c++)
            if (run[c])
                gather(c, A.part1, j + 1, [&](int i, double t) {
                    const double s = scs[c * R2 + i], h = s * scs[c * R2 + j] * t;
                    cf[c * R2 + i] = s * h;
                    if (owner(c)) A.h1[(size_t)i * P + pseg[c]] = h;
                });
        __syncthreads();
        double v[CYC_R];
        update(j + 1, true, v);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < CYC_R; r++)
            if (tid + CYC_THREADS * r < len) ws[tid + CYC_THREADS * r] = v[r];
        __syncthreads();
        for (int c = 0; c < npc; c++)
            if (run[c]) dots(c, j + 1, A.part2);
        if (!cyc_barrier(A.bar, 1, A.err)) return;
        // ---- second projection
        for (int c = 0; c < npc; c++)
            if (run[c])
                gather(c, A.part2, j + 1, [&](int i, double t) {
                    const double s = scs[c * R2 + i], h = s * t;
                    cf[c * R2 + i] = s * h;
                    if (owner(c)) A.h2[(size_t)i * P + pseg[c]] = h;
                });
        __syncthreads();
        update(j + 1, false, v);
        double* vn = Vg + (size_t)(j + 1) * A.n;
#pragma unroll
        for (int r = 0; r < CYC_R; r++) {
            const int i = tid + CYC_THREADS * r;
            if (i >= len) continue;
            vn[i] = v[r];
            if (A.vcache) vsm[(size_t)(j + 1) * A.lmax + i] = v[r];
        }
        for (int c = 0; c < npc; c++) {
            double s = 0.0;
#pragma unroll
            for (int r = 0; r < CYC_R; r++) {
                const int i = tid + CYC_THREADS * r;
                if (i >= pofs[c] && i < pofs[c + 1]) s = fma(v[r], v[r], s);
            }
            s = seg_warp_sum(s);
            __syncthreads();
            if (lane == 0) red[warp] = s;
            __syncthreads();
            if (warp == 0) {
                double t = lane < CYC_WARPS ? red[lane] : 0.0;
                t = seg_warp_sum(t);
                if (lane == 0) A.partn[pc0 + c] = t;
            }
        }
        if (!cyc_barrier(A.bar, 2, A.err)) return;
    }
    if (warp == 0) finish(A.j1);
}

}  // namespace hfem
