// Krylov kernels for several independent systems packed into one vector
// (sm_100a): each problem's trace unknowns form one contiguous segment, and
// every reduction is per segment, so one launch advances the GMRES of every
// problem while each keeps its own Arnoldi basis, Hessenberg matrix and
// convergence test (the per-problem algorithm of kernel/gmres_bilu0.m:17-105).
// A single system is one segment.
//
// A segment is cut into pieces of at most SEG_PIECE entries, one CTA each
// (the host picks the piece length so that there is about one CTA per SM).
// Reductions are deterministic: a CTA reduces its piece in a fixed tree, and
// the last CTA of a segment to finish (counted with an atomic ticket, the
// threadfence-reduction pattern; nothing waits) sums the segment's piece
// partials in piece order and resets the ticket.
//
// One Arnoldi step is the matrix product and three kernels, classical
// Gram-Schmidt applied twice:
//   seg_project_kernel<R, false>   h1 = V^T w
//   seg_project_kernel<R, true>    w -= V h1,  h2 = V^T w   (one pass: the
//                                  piece of V is read again from cache)
//   seg_finish_step_kernel<R>      w -= V h2, |w|, then in the segment's last
//                                  CTA the Givens rotation and stopping test
// The basis columns are kept as they leave the last kernel, without a pass
// that divides them by their norm: column i's factor 1 / |w_i| (GmState::sc)
// is applied to the projections, the coefficients and the matrix product's
// result instead.
#pragma once
#include <cuda_runtime.h>

namespace hfem {

constexpr int SEG_PIECE = 2048;
constexpr int SEG_THREADS = 256;
constexpr int SEG_WARPS = SEG_THREADS / 32;

struct SegPieces {
    int npieces;
    const long long* pstart;   // npieces + 1 entry offsets
    const int* pseg;           // segment of each piece
    const int* seg_p0;         // first piece of each segment (nseg + 1)
    int* ticket;               // per segment, zero between launches
    double* part;              // partial sums, row i of npieces entries per projection
    const unsigned char* act;  // per segment: 0 = skip
};

// GMRES bookkeeping on the device, so that the host enqueues Arnoldi steps
// without reading every Hessenberg column back.  Per problem p: H ((restart + 1)
// x restart, column-major), Givens cosines and sines (restart), g (restart + 1),
// the rhs norm nrmb, state (2 running, 1 converged, 0 iteration limit, -1
// breakdown), iterations, the cycle's step count jc, and act (the segment mask
// every segment kernel reads).  sc[i * P + p] is basis column i's factor.
struct GmState {
    int P, restart, maxit;
    double tol;
    double *H, *cs, *sn, *g, *nrmb, *sc;
    int *state, *its, *jc;
    unsigned char* act;
    double* hist;               // problem 0's relative residual per iteration (hist_len entries) or NULL
    int hist_len;
};

__device__ __forceinline__ double seg_warp_sum(double s) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// sum over the CTA, valid in every thread of warp 0
__device__ __forceinline__ double seg_block_sum(double s, double* red) {
    s = seg_warp_sum(s);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x < 32) {
        t = threadIdx.x < SEG_WARPS ? red[threadIdx.x] : 0.0;
#pragma unroll
        for (int o = SEG_WARPS / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    return t;
}

// true in every thread of the segment's last CTA to arrive; the caller's
// partial sums were written (and fenced by their writers) before the call
__device__ __forceinline__ bool seg_last(const SegPieces& P, int seg) {
    __shared__ int last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const int need = P.seg_p0[seg + 1] - P.seg_p0[seg];
        last = atomicAdd(&P.ticket[seg], 1) == need - 1;
        if (last) P.ticket[seg] = 0;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// v[r] -= sum_{i<k} c_i V_i[i0 + threadIdx.x + SEG_THREADS r], c_i = coef[i * nseg + seg].
// Four partial sums per entry: a single chain of k dependent FMAs would cost
// more than the loads (FP64 latency about 45 cycles).
template <int R>
__device__ __forceinline__ void seg_sub_basis(double (&v)[R], const double* __restrict__ V, long long n, long long i0,
                                              int len, int k, int nseg, int seg, const double* __restrict__ coef,
                                              double* cs) {
    constexpr int CH = 64;
    for (int c0 = 0; c0 < k; c0 += CH) {
        const int m = min(CH, k - c0);
        __syncthreads();
        if (threadIdx.x < m) cs[threadIdx.x] = coef[(size_t)(c0 + threadIdx.x) * nseg + seg];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int idx = threadIdx.x + SEG_THREADS * r;
            if (idx >= len) continue;
            const double* vp = V + (size_t)c0 * n + i0 + idx;
            double a[4] = {0.0, 0.0, 0.0, 0.0};
            int i = 0;
#pragma unroll 8
            for (; i + 4 <= m; i += 4)
#pragma unroll
                for (int q = 0; q < 4; q++) a[q] = fma(cs[i + q], __ldg(vp + (size_t)(i + q) * n), a[q]);
            for (; i < m; i++) a[0] = fma(cs[i], __ldg(vp + (size_t)i * n), a[0]);
            v[r] -= (a[0] + a[1]) + (a[2] + a[3]);
        }
    }
}

// Projections of the new vector on the basis, column i of stride n:
//   UPDATE: w -= sum_{i<k} coef_i V_i first (w is written back)
//   out[i * P + seg] = h_i = <v_i, w>,  outc[i * P + seg] = the coefficient
//   sc_i h_i of the stored column V_i = v_i / sc_i
// A warp takes columns warp, warp + 8, ..., four at a time, over the CTA's
// piece of w in shared memory, so a column costs one warp reduction and no CTA
// barrier (up to four columns: all warps share them).  Bound by latency for
// small systems (2D p=2, 36,864 unknowns, k <= 50: a step's orthogonalisation
// took 92 us when a CTA reduced one column after the other), by the basis
// traffic, 3 passes a step, for large ones.
template <int R, bool UPDATE>
__global__ void __launch_bounds__(SEG_THREADS) seg_project_kernel(SegPieces P, long long n, int k, int nseg,
                                                                  const double* __restrict__ V, double* w,
                                                                  const double* __restrict__ coef,
                                                                  const double* __restrict__ sc,
                                                                  double* __restrict__ out,
                                                                  double* __restrict__ outc) {
    __shared__ double ws[R * SEG_THREADS];
    __shared__ double cs[64];
    const int piece = blockIdx.x;
    const int seg = P.pseg[piece];
    if (P.act && !P.act[seg]) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long i0 = P.pstart[piece];
    const int len = (int)(P.pstart[piece + 1] - i0);
    {
        double v[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int idx = threadIdx.x + SEG_THREADS * r;
            v[r] = idx < len ? w[i0 + idx] : 0.0;
        }
        if constexpr (UPDATE) seg_sub_basis<R>(v, V, n, i0, len, k, nseg, seg, coef, cs);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int idx = threadIdx.x + SEG_THREADS * r;
            ws[idx] = v[r];
            if (UPDATE && idx < len) w[i0 + idx] = v[r];
        }
    }
    __syncthreads();
    if (k <= 4) {
        double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int idx = threadIdx.x + SEG_THREADS * r;
            if (idx >= len) continue;
            const double x = ws[idx];
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (q < k) a[q] = fma(__ldg(V + (size_t)q * n + i0 + idx), x, a[q]);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            a[q] = seg_warp_sum(a[q]);
            if (lane == 0) cs[q * SEG_WARPS + warp] = a[q];
        }
        __syncthreads();
        if (threadIdx.x < k) {
            double t = 0.0;
#pragma unroll
            for (int q = 0; q < SEG_WARPS; q++) t += cs[threadIdx.x * SEG_WARPS + q];
            P.part[(size_t)threadIdx.x * P.npieces + piece] = t;
            __threadfence();
        }
    } else {
        for (int base = warp; base < k; base += 4 * SEG_WARPS) {
            double a[4] = {0.0, 0.0, 0.0, 0.0};
            const double* vp = V + (size_t)base * n + i0;
            const size_t st = (size_t)SEG_WARPS * n;
#pragma unroll 8
            for (int idx = lane; idx < len; idx += 32) {
                const double x = ws[idx];
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (base + SEG_WARPS * q < k) a[q] = fma(__ldg(vp + q * st + idx), x, a[q]);
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                a[q] = seg_warp_sum(a[q]);
                const int i = base + SEG_WARPS * q;
                if (lane == 0 && i < k) P.part[(size_t)i * P.npieces + piece] = a[q];
            }
        }
        if (lane == 0) __threadfence();
    }
    if (!seg_last(P, seg)) return;
    const int p0 = P.seg_p0[seg], p1 = P.seg_p0[seg + 1];
    for (int base = warp; base < k; base += 4 * SEG_WARPS) {
        double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
        for (int q = p0 + lane; q < p1; q += 32)
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (base + SEG_WARPS * u < k) t[u] += __ldcg(&P.part[(size_t)(base + SEG_WARPS * u) * P.npieces + q]);
#pragma unroll
        for (int u = 0; u < 4; u++) t[u] = seg_warp_sum(t[u]);
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = base + SEG_WARPS * u;
            if (lane != u || i >= k) continue;
            const double s = sc[(size_t)i * nseg + seg], h = t[u] * s;
            out[(size_t)i * nseg + seg] = h;
            outc[(size_t)i * nseg + seg] = h * s;
        }
    }
}

// |v| over the segment in every lane of warp 0 of its last CTA; false in the others
__device__ __forceinline__ bool seg_norm(const SegPieces& P, int piece, int seg, double s, double* red, double& nrm) {
    s = seg_block_sum(s, red);
    if (threadIdx.x == 0) P.part[piece] = s;
    if (!seg_last(P, seg)) return false;
    double t = 0.0;
    for (int q = P.seg_p0[seg] + threadIdx.x; q < P.seg_p0[seg + 1]; q += SEG_THREADS) t += __ldcg(&P.part[q]);
    nrm = sqrt(seg_block_sum(t, red));
    return threadIdx.x < 32;
}

// Arnoldi step j of problem p by one warp: the new Hessenberg column (both
// projections and the new norm nn), the previous rotations applied, the new
// rotation, the residual estimate and the stopping test
// (kernel/gmres_bilu0.m:17-105).  The rotations form a chain in `carry`; what
// does not depend on it is formed lane-parallel first.
__device__ __forceinline__ void gm_givens_warp(const GmState& S, int p, int j, const double* __restrict__ h1,
                                               const double* __restrict__ h2, double nn) {
    const int R = S.restart, P = S.P, lane = threadIdx.x & 31;
    double* hc = S.H + (size_t)(R + 1) * R * p + (size_t)(R + 1) * j;
    double* cp = S.cs + (size_t)R * p;
    double* sp = S.sn + (size_t)R * p;
    auto h = [&](int i) { return __ldcg(&h1[(size_t)i * P + p]) + __ldcg(&h2[(size_t)i * P + p]); };
    double carry = h(0);
    for (int i0 = 0; i0 < j; i0 += 32) {
        const int i = i0 + lane;
        double c = 0.0, s = 0.0, sb = 0.0, cb = 0.0, mine = 0.0;
        if (i < j) {
            const double b = h(i + 1);
            c = cp[i];
            s = sp[i];
            sb = s * b;
            cb = c * b;
        }
        const int m = min(32, j - i0);
#pragma unroll 4
        for (int t = 0; t < m; t++) {
            const double ct = __shfl_sync(0xffffffffu, c, t), st = __shfl_sync(0xffffffffu, s, t);
            const double sbt = __shfl_sync(0xffffffffu, sb, t), cbt = __shfl_sync(0xffffffffu, cb, t);
            if (lane == t) mine = fma(ct, carry, sbt);
            carry = fma(-st, carry, cbt);
        }
        if (i < j) hc[i] = mine;
    }
    if (lane != 0) return;
    const double rr = sqrt(carry * carry + nn * nn);
    const double c = carry / rr, s = nn / rr;
    cp[j] = c;
    sp[j] = s;
    hc[j] = rr;
    hc[j + 1] = 0.0;
    double* gp = S.g + (size_t)(R + 1) * p;
    const double g = gp[j];
    gp[j + 1] = -s * g;
    gp[j] = c * g;
    S.sc[(size_t)(j + 1) * P + p] = nn == 0.0 ? 1.0 : 1.0 / nn;
    const int it = ++S.its[p];
    S.jc[p] = j + 1;
    const double res = fabs(-s * g);
    if (p == 0 && S.hist && it - 1 < S.hist_len) S.hist[it - 1] = res / S.nrmb[0];
    int stop = 2;
    if (res / S.nrmb[p] <= S.tol) stop = 1;
    else if (it >= S.maxit) stop = 0;
    else if (nn == 0.0) stop = -1;
    if (stop != 2) {
        S.state[p] = stop;
        S.act[p] = 0;
    }
}

// w -= sum_{i<=j} coef_i V_i (the second projection), |w|, and the step's bookkeeping
template <int R>
__global__ void __launch_bounds__(SEG_THREADS) seg_finish_step_kernel(SegPieces P, GmState S, long long n, int j,
                                                                      const double* __restrict__ V, double* w,
                                                                      const double* __restrict__ coef,
                                                                      const double* __restrict__ h1,
                                                                      const double* __restrict__ h2) {
    __shared__ double red[SEG_WARPS];
    __shared__ double cs[64];
    const int piece = blockIdx.x;
    const int seg = P.pseg[piece];
    if (P.act && !P.act[seg]) return;
    const long long i0 = P.pstart[piece];
    const int len = (int)(P.pstart[piece + 1] - i0);
    double v[R], s = 0.0;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int idx = threadIdx.x + SEG_THREADS * r;
        v[r] = idx < len ? w[i0 + idx] : 0.0;
    }
    seg_sub_basis<R>(v, V, n, i0, len, j + 1, S.P, seg, coef, cs);
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int idx = threadIdx.x + SEG_THREADS * r;
        if (idx < len) w[i0 + idx] = v[r];
        s += v[r] * v[r];
    }
    double nn;
    if (seg_norm(P, piece, seg, s, red, nn)) gm_givens_warp(S, seg, j, h1, h2, nn);
}

// Start of a restart cycle: V_0 = b (first: x = 0) or b - V_0 (V_0 holds
// M^-1 A x), beta = |V_0| per problem, and the problems that go on.
template <int R>
__global__ void __launch_bounds__(SEG_THREADS) seg_start_kernel(SegPieces P, GmState S, bool first,
                                                                const double* __restrict__ b, double* v0) {
    __shared__ double red[SEG_WARPS];
    const int piece = blockIdx.x;
    const int seg = P.pseg[piece];
    if (!first && !S.act[seg]) return;
    const long long i0 = P.pstart[piece];
    const int len = (int)(P.pstart[piece + 1] - i0);
    double s = 0.0;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int idx = threadIdx.x + SEG_THREADS * r;
        if (idx >= len) continue;
        const double v = first ? b[i0 + idx] : b[i0 + idx] - v0[i0 + idx];
        v0[i0 + idx] = v;
        s += v * v;
    }
    double beta;
    if (!seg_norm(P, piece, seg, s, red, beta) || threadIdx.x != 0) return;
    if (first) {
        S.nrmb[seg] = beta == 0.0 ? 1.0 : beta;
        S.its[seg] = 0;
    }
    S.jc[seg] = 0;
    const bool done = beta / S.nrmb[seg] <= S.tol;
    S.state[seg] = done ? 1 : 2;
    S.act[seg] = done ? 0 : 1;
    S.g[(size_t)(S.restart + 1) * seg] = beta;
    S.sc[seg] = beta == 0.0 ? 1.0 : 1.0 / beta;
}

// End of a cycle: y = H^-1 g by back substitution, one warp per problem, the
// basis columns' factors included; kseg = its step count (0: none), and act =
// the problems still running.  s holds the right-hand side being reduced: in
// shared memory when it fits, else in y itself.
constexpr int GM_SOLVE_MAX = 1024;
__global__ void __launch_bounds__(32) gm_solve_kernel(GmState S, double* __restrict__ y, int* __restrict__ kseg) {
    __shared__ double buf[GM_SOLVE_MAX];
    const int p = blockIdx.x, lane = threadIdx.x;
    const int R = S.restart, J = S.jc[p];
    if (lane == 0) {
        S.act[p] = S.state[p] == 2;
        kseg[p] = J;
        S.jc[p] = 0;
    }
    const double* hp = S.H + (size_t)(R + 1) * R * p;
    const double* gp = S.g + (size_t)(R + 1) * p;
    double* yp = y + (size_t)R * p;
    double* s = J <= GM_SOLVE_MAX ? buf : yp;
    for (int i = lane; i < J; i += 32) s[i] = gp[i];
    __syncwarp();
    for (int i = J - 1; i >= 0; i--) {
        const double* col = hp + (size_t)(R + 1) * i;
        const double yi = s[i] / col[i];
        for (int q = lane; q < i; q += 32) s[q] -= col[q] * yi;
        __syncwarp();
        if (lane == 0) s[i] = yi;
    }
    __syncwarp();
    for (int i = lane; i < J; i += 32) yp[i] = s[i] * S.sc[(size_t)i * S.P + p];
}

// x += sum_{j<kseg[seg]} V_j y[seg * ldy + j]   (columns of stride n)
template <int R>
__global__ void __launch_bounds__(SEG_THREADS) seg_combine_kernel(SegPieces P, long long n, const int* __restrict__ kseg,
                                                                  int ldy, const double* __restrict__ V,
                                                                  const double* __restrict__ y,
                                                                  double* __restrict__ x) {
    __shared__ double cs[64];
    const int piece = blockIdx.x;
    const int seg = P.pseg[piece];
    const int k = kseg[seg];
    if (k == 0) return;
    const long long i0 = P.pstart[piece];
    const int len = (int)(P.pstart[piece + 1] - i0);
    double v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = 0.0;
    seg_sub_basis<R>(v, V, n, i0, len, k, 1, 0, y + (size_t)seg * ldy, cs);
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int idx = threadIdx.x + SEG_THREADS * r;
        if (idx < len) x[i0 + idx] -= v[r];
    }
}

// z = xsc M^-1 (Hg x) with one warp per block row (xsc: a factor per segment,
// NULL: 1), for block sizes below 20.  A row's blocks are contiguous in Hg, so the row
// is one column-major BSZ x (nblk * BSZ) matrix; the warp's lanes form G groups of
// columns, and the groups' partial sums are added in group order.  Even block sizes: a
// lane reads two rows of a column as one 16-byte load, BSZ / 2 lanes per column (2D p=2:
// 0.91 -> 0.66 ms per 62 products).  Rows of inactive segments (act[rseg[i]] == 0; rseg
// NULL: one segment) are skipped.
template <int BSZ, typename MT>
__global__ void __launch_bounds__(256) bsr_matvec_warp_kernel(int nrows, const int* __restrict__ rowstart,
                                                              const int* __restrict__ colidx,
                                                              const double* __restrict__ Hg,
                                                              const MT* __restrict__ Minv,
                                                              const double* __restrict__ x,
                                                              const double* __restrict__ xsc, double* __restrict__ z,
                                                              const int* __restrict__ rseg,
                                                              const unsigned char* __restrict__ act) {
    static_assert(BSZ <= 32, "a lane per row");
    constexpr bool PAIRS = BSZ % 2 == 0;
    constexpr int LC = PAIRS ? BSZ / 2 : BSZ, G = 32 / LC;      // lanes per column, columns at a time
    __shared__ double ys[8][G][32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int g = lane / LC, q = lane - g * LC;
    const int nwarps = gridDim.x * 8;
    for (int i = blockIdx.x * 8 + wib; i < nrows; i += nwarps) {
        if (act && !act[rseg ? rseg[i] : 0]) continue;
        const int k0 = rowstart[i], k1 = rowstart[i + 1];
        const int ncol = (k1 - k0) * BSZ;
        const double* A = Hg + (size_t)k0 * BSZ * BSZ;
        if (g < G) {
            double a0 = 0.0, a1 = 0.0;
#pragma unroll 4
            for (int cc = g; cc < ncol; cc += G) {
                const int kb = cc / BSZ, c = cc - kb * BSZ;
                const double xv = __ldg(&x[(size_t)colidx[k0 + kb] * BSZ + c]);
                if constexpr (PAIRS) {
                    const double2 av = __ldg(reinterpret_cast<const double2*>(A + (size_t)cc * BSZ) + q);
                    a0 += av.x * xv;
                    a1 += av.y * xv;
                } else {
                    a0 += __ldg(&A[(size_t)cc * BSZ + q]) * xv;
                }
            }
            if constexpr (PAIRS) {
                ys[wib][g][2 * q] = a0;
                ys[wib][g][2 * q + 1] = a1;
            } else {
                ys[wib][g][q] = a0;
            }
        }
        __syncwarp();
        double y = 0.0;
        if (lane < BSZ)
#pragma unroll
            for (int gg = 0; gg < G; gg++) y += ys[wib][gg][lane];
        if (xsc) y *= xsc[rseg ? rseg[i] : 0];
        __syncwarp();
        if (!Minv) {
            if (lane < BSZ) z[(size_t)i * BSZ + lane] = y;
            continue;
        }
        if (lane < BSZ) ys[wib][0][lane] = y;
        __syncwarp();
        const MT* m = Minv + (size_t)i * BSZ * BSZ;
        if (lane < BSZ) {
            double s = 0.0;
#pragma unroll 4
            for (int c = 0; c < BSZ; c++) s += (double)__ldg(&m[(size_t)c * BSZ + lane]) * ys[wib][0][c];
            z[(size_t)i * BSZ + lane] = s;
        }
        __syncwarp();
    }
}

// The same product with one CTA per block row, for even block sizes from 20 on.
// The row is one column-major BSZ x (nblk * BSZ) array; thread t owns the row
// pair t % (BSZ / 2) of columns g, g + G, ..., g = t / (BSZ / 2), so that every
// load of A is 16 bytes and all threads of the CTA stream the row together; the
// G partial sums are added in group order.  M^-1's entries are requested before
// the barrier that ends the product.  Bound by HBM (Hg once): 2,592 rows of block
// size 50, 363 MB, 198 us with a warp per row (1.8 TB/s), 66 us here (5.5 TB/s).
template <int BSZ>
struct RowMv {
    static constexpr int L2 = BSZ / 2;
    static constexpr int G = BSZ >= 30 ? 8 : 12;
    static constexpr int USED = L2 * G;
    static constexpr int THREADS = (USED + 31) / 32 * 32;
    static constexpr int MC = (BSZ + G - 1) / G;      // columns of M^-1 per thread
};
__device__ __forceinline__ double2 ldg_pair(const double* p) { return __ldg(reinterpret_cast<const double2*>(p)); }
__device__ __forceinline__ double2 ldg_pair(const float* p) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    return make_double2((double)v.x, (double)v.y);
}

template <int BSZ, typename MT>
__global__ void __launch_bounds__(RowMv<BSZ>::THREADS) bsr_matvec_row_kernel(int nrows, const int* __restrict__ rowstart,
                                                                             const int* __restrict__ colidx,
                                                                             const double* __restrict__ Hg,
                                                                             const MT* __restrict__ Minv,
                                                                             const double* __restrict__ x,
                                                                             const double* __restrict__ xsc,
                                                                             double* __restrict__ z,
                                                                             const int* __restrict__ rseg,
                                                                             const unsigned char* __restrict__ act) {
    using C = RowMv<BSZ>;
    static_assert(BSZ % 2 == 0, "16-byte loads of row pairs");
    __shared__ double ys[C::G][BSZ + 2];
    __shared__ double y[BSZ];
    const int tid = threadIdx.x, g = tid / C::L2, q = tid - g * C::L2;
    const int i = blockIdx.x;
    if (act && !act[rseg ? rseg[i] : 0]) return;
    const int k0 = rowstart[i], ncol = (rowstart[i + 1] - k0) * BSZ;
    const bool on = tid < C::USED;
    double a0 = 0.0, a1 = 0.0;
    if (on) {
        const double* A = Hg + (size_t)k0 * BSZ * BSZ + 2 * q;
#pragma unroll 8
        for (int cc = g; cc < ncol; cc += C::G) {
            const int kb = cc / BSZ, c = cc - kb * BSZ;
            const double xv = __ldg(&x[(size_t)__ldg(&colidx[k0 + kb]) * BSZ + c]);
            const double2 av = ldg_pair(A + (size_t)cc * BSZ);
            a0 = fma(av.x, xv, a0);
            a1 = fma(av.y, xv, a1);
        }
        ys[g][2 * q] = a0;
        ys[g][2 * q + 1] = a1;
    }
    double2 m[C::MC];
    if (Minv && on) {
        const MT* M = Minv + (size_t)i * BSZ * BSZ + 2 * q;
#pragma unroll
        for (int t = 0; t < C::MC; t++) {
            const int c = g + C::G * t;
            m[t] = c < BSZ ? ldg_pair(M + (size_t)c * BSZ) : make_double2(0.0, 0.0);
        }
    }
    __syncthreads();
    if (tid < BSZ) {
        double s = 0.0;
#pragma unroll
        for (int gg = 0; gg < C::G; gg++) s += ys[gg][tid];
        if (xsc) s *= xsc[rseg ? rseg[i] : 0];
        if (Minv) y[tid] = s;
        else z[(size_t)i * BSZ + tid] = s;
    }
    if (!Minv) return;
    __syncthreads();
    if (on) {
        double b0 = 0.0, b1 = 0.0;
#pragma unroll
        for (int t = 0; t < C::MC; t++) {
            const int c = g + C::G * t;
            const double yc = c < BSZ ? y[c] : 0.0;
            b0 = fma(m[t].x, yc, b0);
            b1 = fma(m[t].y, yc, b1);
        }
        ys[g][2 * q] = b0;
        ys[g][2 * q + 1] = b1;
    }
    __syncthreads();
    if (tid < BSZ) {
        double s = 0.0;
#pragma unroll
        for (int gg = 0; gg < C::G; gg++) s += ys[gg][tid];
        z[(size_t)i * BSZ + tid] = s;
    }
}

}  // namespace hfem
