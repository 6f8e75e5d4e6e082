// batched.cu -- many independent BiCGSTAB solves in one persistent launch.
//
// The systems are laid side by side as one block-diagonal SELL-32 matrix (a
// slice never straddles two systems). One cooperative kernel runs the whole
// solve: every phase sweeps the rows of the systems still iterating, with
// grid-wide barriers between phases, and every reduction is per system
// (warp/slice partial sums, then one block per system summing its partials in
// a fixed order: deterministic, no atomics on floating point). Per system:
//   * BiCGSTAB (the recurrences of bicgstab.cpp's Eigen solver) on A D^-1,
//     in FP32 with FP64 dot products when mixed, else in FP64;
//   * each inner solve stops when its residual has dropped by itol (or on a
//     breakdown, or after max_inner iterations); then an FP64 refinement step
//     x += D^-1 d, r = b - A x (FP64 matrix) decides: converged
//     (||r|| <= tol ||b||), failed (max_pass / maxit reached) or a new inner
//     solve on r.
// Systems finish independently: every block lists the systems in the state a
// phase works on (in shared memory, from the states), and each warp walks a
// contiguous run of their slices, so finished systems cost nothing.
// Launch shape (block size, lanes per row of the SpMV sweeps) is autotuned on
// the batch itself and kept with the plan.
#include <cooperative_groups.h>

#include <chrono>
#include <cmath>
#include <cstring>

#include "batched.h"
#include "reduce.cuh"

namespace cg = cooperative_groups;

namespace pb {

namespace {

constexpr int MAX_BLOCK = 512;

enum { S_INNER = 0, S_REFINE = 1, S_DONE = 2, S_FAILED = 3 };

struct BState {
    double rho, alpha, omega, beta, bb, tol2, rr64, rr0;
    long long iter;
    int state, fresh, pass, inner, status, stop;
};

template <typename T>
struct BP {
    int nprob, nslices;
    const int* slice_prob;
    const int* prob_slice0;
    const int* prob_n;
    const int* sl_off;
    const int* col;
    const double* A64;
    const T* A;  // column-scaled inner matrix A D^-1
    const double* b64;
    const double* dinv;
    double* x64;
    T *r, *r0, *p, *v, *s, *t, *d;
    double* cdot;  // 3 per chunk of the SpMV sweeps (nslices * lpr chunks)
    double* sdot;  // 2 per slice (update sweep)
    BState* st;
    int* ctl;  // [2 * buffer]: systems still active, systems waiting for refinement
    double tol2, itol2;
    int max_inner, max_pass, max_steps;
    long long maxit;
};

// Data written inside the launch by other blocks is read through L2 (ld.cg).
__device__ __forceinline__ int stateOf(const BState* st, int p) { return __ldcg(&st[p].state); }
__device__ __forceinline__ double ld(const double* a, int i) { return __ldcg(a + i); }
__device__ __forceinline__ float ld(const float* a, int i) { return __ldcg(a + i); }

// block-wide sums of a and b (valid in thread 0); sh holds 2 * MAX_BLOCK / 32 doubles
__device__ __forceinline__ void blockSum2(double& a, double& b, double* sh) {
    a = warpSum(a);
    b = warpSum(b);
    const int w = threadIdx.x >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        sh[w] = a;
        sh[MAX_BLOCK / 32 + w] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ta = 0.0, tb = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
            ta += sh[i];
            tb += sh[MAX_BLOCK / 32 + i];
        }
        a = ta;
        b = tb;
    }
}

// Sum over this row's SELL slots of val * xf(col), LPR adjacent lanes per row;
// the total is returned in every lane of the group.
template <int LPR, typename V, typename F>
__device__ __forceinline__ double rowDot(const int* sl_off, const int* col, const V* val, int row, int sub, F xf) {
    const int s = row >> 5;
    const int s0 = sl_off[s];
    const int width = (sl_off[s + 1] - s0) >> 5;
    const int bo = s0 + (row & 31);
    double sum = 0.0;
    for (int j = sub; j < width; j += LPR) {
        const int q = bo + 32 * j;
        sum += (double)val[q] * xf(col[q]);
    }
    if constexpr (LPR > 1) {
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    return sum;
}

// Systems in state `want`, listed in every block's shared memory: ids[k] and
// the prefix pre[k] of their slice counts (pre[m] = total). Each block builds
// the same list from the states, so no extra grid barrier is needed.
template <typename T>
__device__ int buildList(const BP<T>& P, int want, int* pre, int* ids, int* tmp, int& m_out) {
    const int nt = blockDim.x, t = threadIdx.x;
    const int per = (P.nprob + nt - 1) / nt;
    const int k0 = min(t * per, P.nprob), k1 = min(k0 + per, P.nprob);
    int cnt = 0, sl = 0;
    for (int k = k0; k < k1; ++k)
        if (stateOf(P.st, k) == want) {
            ++cnt;
            sl += P.prob_slice0[k + 1] - P.prob_slice0[k];
        }
    __syncthreads();
    tmp[t] = cnt;
    tmp[nt + t] = sl;
    __syncthreads();
    if (t == 0) {
        int c = 0, q = 0;
        for (int i = 0; i < nt; ++i) {
            const int a = tmp[i], b = tmp[nt + i];
            tmp[i] = c;
            tmp[nt + i] = q;
            c += a;
            q += b;
        }
        tmp[2 * nt] = c;
        tmp[2 * nt + 1] = q;
    }
    __syncthreads();
    int c = tmp[t], q = tmp[nt + t];
    for (int k = k0; k < k1; ++k)
        if (stateOf(P.st, k) == want) {
            ids[c] = k;
            pre[c] = q;
            ++c;
            q += P.prob_slice0[k + 1] - P.prob_slice0[k];
        }
    const int m = tmp[2 * nt], total = tmp[2 * nt + 1];
    if (t == 0) pre[m] = total;
    __syncthreads();
    m_out = m;
    return total;
}
// list entry holding virtual slice v (pre[k] <= v < pre[k+1])
__device__ __forceinline__ int findEntry(const int* pre, int m, int v) {
    int lo = 0, hi = m;  // pre[lo] <= v < pre[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pre[mid] <= v) lo = mid;
        else hi = mid;
    }
    return lo;
}

// A warp's contiguous run of list units (slices, or chunks of LPR per slice):
// tracks the system of the current unit so that per-system data is loaded once
// per run segment instead of once per unit.
struct Run {
    int v, vend;  // units [v, vend)
    int k, kend;  // list entry and the unit where it ends
    int pr, slice0, rows_end;
};
template <typename T>
__device__ __forceinline__ void runEnter(const BP<T>& P, const int* pre, const int* ids, int upu, Run& R) {
    R.pr = ids[R.k];
    R.kend = pre[R.k + 1] * upu;
    R.slice0 = P.prob_slice0[R.pr] - pre[R.k];
    R.rows_end = 32 * P.prob_slice0[R.pr] + P.prob_n[R.pr];
}
// upu: units per slice; returns false when the warp has no units
template <typename T>
__device__ __forceinline__ bool runStart(const BP<T>& P, const int* pre, const int* ids, int m, int total_units,
                                         int upu, int gwarp, int nwarps, Run& R) {
    const int per = (total_units + nwarps - 1) / nwarps;
    R.v = gwarp * per;
    R.vend = min(R.v + per, total_units);
    if (R.v >= R.vend) return false;
    R.k = findEntry(pre, m, R.v / upu);
    runEnter(P, pre, ids, upu, R);
    return true;
}
// advance to the system of unit R.v; true when the system changed
template <typename T>
__device__ __forceinline__ bool runSeek(const BP<T>& P, const int* pre, const int* ids, int upu, Run& R) {
    if (R.v < R.kend) return false;
    while (R.v >= pre[R.k + 1] * upu) ++R.k;
    runEnter(P, pre, ids, upu, R);
    return true;
}

// Row sums of US consecutive units (chunks of one system) starting at R.v:
// the slots of all units are walked together so that their loads overlap.
template <typename T, int LPR, int US, typename V, typename F>
__device__ __forceinline__ void spmvUnits(const BP<T>& P, const V* val, const Run& R, int nh, int lane, int* row,
                                          int* chunk, double* sum, F xf) {
    constexpr int RPC = 32 / LPR;
    const int sub = lane % LPR;
    int bo[US], w[US];
    int wmax = 0;
#pragma unroll
    for (int u = 0; u < US; ++u) {
        const int vu = R.v + (u < nh ? u : 0);
        const int slice = R.slice0 + vu / LPR;
        chunk[u] = slice * LPR + vu % LPR;
        row[u] = 32 * slice + (vu % LPR) * RPC + lane / LPR;
        const int s0 = P.sl_off[slice];
        w[u] = u < nh ? (P.sl_off[slice + 1] - s0) >> 5 : 0;
        bo[u] = s0 + (row[u] & 31);
        sum[u] = 0.0;
        wmax = max(wmax, w[u]);
    }
    for (int j = sub; j < wmax; j += LPR) {
#pragma unroll
        for (int u = 0; u < US; ++u)
            if (j < w[u]) {
                const int q = bo[u] + 32 * j;
                sum[u] += (double)val[q] * xf(P.col[q]);
            }
    }
    if constexpr (LPR > 1) {
#pragma unroll
        for (int u = 0; u < US; ++u)
#pragma unroll
            for (int o = LPR / 2; o > 0; o >>= 1) sum[u] += __shfl_xor_sync(0xffffffffu, sum[u], o);
    }
}

// At most 64 registers per thread (2 blocks of 512 per SM): the sweeps are
// latency-bound, so loads in flight (UR / US units per warp step) and
// occupancy matter more than registers.
template <typename T, int LPR>
__global__ void __launch_bounds__(MAX_BLOCK, 2) batch_kernel(const BP<T> P) {
    __shared__ double sh[2 * MAX_BLOCK / 32];
    extern __shared__ int lists[];  // pre (nprob + 1) | ids (nprob) | scan scratch (2 * blockDim + 2)
    int* pre = lists;
    int* ids = lists + P.nprob + 1;
    int* tmp = lists + 2 * P.nprob + 1;
    cg::grid_group grid = cg::this_grid();
    const int lane = threadIdx.x & 31;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    constexpr int RPC = 32 / LPR;  // rows per chunk (one warp)
    constexpr int UR = 2;          // slices per warp step in the row sweeps
    constexpr int US = LPR == 1 ? 2 : 1;  // units per warp step in the SpMV sweeps
    Run R;

    for (int step = 0; step < P.max_steps; ++step) {
        const int cur = step & 1, nxt = cur ^ 1;
        const int n_active = __ldcg(&P.ctl[2 * cur]);
        const int n_refine = __ldcg(&P.ctl[2 * cur + 1]);
        if (n_active == 0) break;  // the same value in every thread: read after a grid barrier
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            P.ctl[2 * nxt] = 0;
            P.ctl[2 * nxt + 1] = 0;
        }
        int m;
        if (n_refine > 0) {
            const int total = buildList(P, S_REFINE, pre, ids, tmp, m);
            // R1: x += D^-1 d, d = 0 (systems waiting for refinement)
            if (runStart(P, pre, ids, m, total, 1, gwarp, nwarps, R)) {
                for (; R.v < R.vend; ++R.v) {
                    runSeek(P, pre, ids, 1, R);
                    const int r = 32 * (R.slice0 + R.v) + lane;
                    if (r >= R.rows_end) continue;
                    P.x64[r] = ld(P.x64, r) + P.dinv[r] * (double)ld(P.d, r);
                    P.d[r] = (T)0;
                }
            }
            grid.sync();
            // R2: r = b - A x in FP64; the inner residual starts from (T) r
            if (runStart(P, pre, ids, m, total * LPR, LPR, gwarp, nwarps, R)) {
                for (; R.v < R.vend; ++R.v) {
                    runSeek(P, pre, ids, LPR, R);
                    const int slice = R.slice0 + R.v / LPR;
                    const int chunk = slice * LPR + R.v % LPR;
                    const int row = 32 * slice + (R.v % LPR) * RPC + lane / LPR, sub = lane % LPR;
                    const bool valid = row < R.rows_end;
                    // every lane runs the same shuffles; padding rows hold zero values
                    const double ax = rowDot<LPR>(P.sl_off, P.col, P.A64, row, sub,
                                                  [&](int c) { return ld(P.x64, c); });
                    double t0 = 0.0, t1 = 0.0;
                    if (valid && sub == 0) {
                        const double r64 = P.b64[row] - ax;
                        const T rt = (T)r64;
                        P.r[row] = rt;
                        t0 = r64 * r64;
                        t1 = (double)rt * (double)rt;
                    }
                    t0 = warpSum(t0);
                    t1 = warpSum(t1);
                    if (lane == 0) {
                        P.cdot[3 * chunk] = t0;
                        P.cdot[3 * chunk + 1] = t1;
                    }
                }
            }
            grid.sync();
            // RED(R): converged, failed, or a new inner solve
            for (int pr = blockIdx.x; pr < P.nprob; pr += gridDim.x) {
                if (stateOf(P.st, pr) != S_REFINE) continue;
                const int c0 = P.prob_slice0[pr] * LPR, c1 = P.prob_slice0[pr + 1] * LPR;
                double a = 0.0, b = 0.0;
                for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
                    a += ld(P.cdot, 3 * c);
                    b += ld(P.cdot, 3 * c + 1);
                }
                blockSum2(a, b, sh);
                if (threadIdx.x == 0) {
                    BState& S = P.st[pr];
                    S.rr64 = a;
                    if (!isfinite(a)) {
                        S.status = PRISM_NONFINITE;
                        S.state = S_FAILED;
                    } else if (a <= P.tol2 * S.bb) {
                        S.state = S_DONE;
                    } else if (S.stop || S.pass >= P.max_pass || S.iter >= P.maxit) {
                        S.status = PRISM_NOT_CONVERGED;
                        S.state = S_FAILED;
                    } else {
                        S.pass += 1;
                        S.inner = 0;
                        S.rho = b;
                        S.rr0 = b;
                        S.alpha = 1.0;
                        S.omega = 1.0;
                        S.beta = 0.0;
                        S.tol2 = P.itol2 * b;
                        S.fresh = 1;
                        S.state = S_INNER;
                    }
                }
                __syncthreads();
            }
            grid.sync();
        }
        const int total = buildList(P, S_INNER, pre, ids, tmp, m);
        if (n_refine > 0) {
            // R3: fresh inner solves: r0 = r, p = v = 0
            if (runStart(P, pre, ids, m, total, 1, gwarp, nwarps, R)) {
                bool fresh = __ldcg(&P.st[R.pr].fresh);
                for (; R.v < R.vend; ++R.v) {
                    if (runSeek(P, pre, ids, 1, R)) fresh = __ldcg(&P.st[R.pr].fresh);
                    const int r = 32 * (R.slice0 + R.v) + lane;
                    if (!fresh || r >= R.rows_end) continue;
                    P.r0[r] = ld(P.r, r);
                    P.p[r] = (T)0;
                    P.v[r] = (T)0;
                }
            }
            grid.sync();
        }

        // ---- one BiCGSTAB iteration of every system in an inner solve
        // A: p = r + beta (p - omega v)          (UR slices per warp step: loads first, then stores)
        if (runStart(P, pre, ids, m, total, 1, gwarp, nwarps, R)) {
            double beta = __ldcg(&P.st[R.pr].beta), omega = __ldcg(&P.st[R.pr].omega);
            while (R.v < R.vend) {
                if (runSeek(P, pre, ids, 1, R)) {
                    beta = __ldcg(&P.st[R.pr].beta);
                    omega = __ldcg(&P.st[R.pr].omega);
                }
                const int nh = min(UR, min(R.kend, R.vend) - R.v);
                int rr[UR];
                T a0[UR], a1[UR], a2[UR];
#pragma unroll
                for (int u = 0; u < UR; ++u) {
                    rr[u] = 32 * (R.slice0 + R.v + u) + lane;
                    if (u < nh && rr[u] < R.rows_end) {
                        a0[u] = ld(P.r, rr[u]);
                        a1[u] = ld(P.p, rr[u]);
                        a2[u] = ld(P.v, rr[u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < UR; ++u)
                    if (u < nh && rr[u] < R.rows_end)
                        P.p[rr[u]] = (T)((double)a0[u] + beta * ((double)a1[u] - omega * (double)a2[u]));
                R.v += nh;
            }
        }
        grid.sync();
        // B: v = A' p ; r0.v
        if (runStart(P, pre, ids, m, total * LPR, LPR, gwarp, nwarps, R)) {
            while (R.v < R.vend) {
                runSeek(P, pre, ids, LPR, R);
                const int nh = min(US, min(R.kend, R.vend) - R.v);
                int row[US], chunk[US];
                double sum[US];
                const int sub = lane % LPR;
                spmvUnits<T, LPR, US>(P, P.A, R, nh, lane, row, chunk, sum, [&](int c) { return (double)ld(P.p, c); });
#pragma unroll
                for (int u = 0; u < US; ++u) {
                    double t0 = 0.0;
                    if (u < nh && row[u] < R.rows_end && sub == 0) {
                        const T vt = (T)sum[u];
                        P.v[row[u]] = vt;
                        t0 = (double)ld(P.r0, row[u]) * (double)vt;
                    }
                    t0 = warpSum(t0);
                    if (lane == 0 && u < nh) P.cdot[3 * chunk[u]] = t0;
                }
                R.v += nh;
            }
        }
        grid.sync();
        // RED(B): alpha = rho / (r0.v)
        for (int pr = blockIdx.x; pr < P.nprob; pr += gridDim.x) {
            if (stateOf(P.st, pr) != S_INNER) continue;
            const int c0 = P.prob_slice0[pr] * LPR, c1 = P.prob_slice0[pr + 1] * LPR;
            double a = 0.0, b = 0.0;
            for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) a += ld(P.cdot, 3 * c);
            blockSum2(a, b, sh);
            if (threadIdx.x == 0) {
                BState& S = P.st[pr];
                const double alpha = S.rho / a;
                if (a == 0.0 || !isfinite(alpha)) {
                    S.state = S_REFINE;  // breakdown: refine and restart
                } else {
                    S.alpha = alpha;
                }
            }
            __syncthreads();
        }
        grid.sync();
        // D: s = r - alpha v   (systems that broke down in RED(B) are skipped from here on)
        if (runStart(P, pre, ids, m, total, 1, gwarp, nwarps, R)) {
            bool on = stateOf(P.st, R.pr) == S_INNER;
            double alpha = __ldcg(&P.st[R.pr].alpha);
            while (R.v < R.vend) {
                if (runSeek(P, pre, ids, 1, R)) {
                    on = stateOf(P.st, R.pr) == S_INNER;
                    alpha = __ldcg(&P.st[R.pr].alpha);
                }
                const int nh = min(UR, min(R.kend, R.vend) - R.v);
                if (on) {
                    int rr[UR];
                    T a0[UR], a1[UR];
#pragma unroll
                    for (int u = 0; u < UR; ++u) {
                        rr[u] = 32 * (R.slice0 + R.v + u) + lane;
                        if (u < nh && rr[u] < R.rows_end) {
                            a0[u] = ld(P.r, rr[u]);
                            a1[u] = ld(P.v, rr[u]);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < UR; ++u)
                        if (u < nh && rr[u] < R.rows_end) P.s[rr[u]] = (T)((double)a0[u] - alpha * (double)a1[u]);
                }
                R.v += nh;
            }
        }
        grid.sync();
        // E: t = A' s ; t.s, t.t
        if (runStart(P, pre, ids, m, total * LPR, LPR, gwarp, nwarps, R)) {
            bool on = stateOf(P.st, R.pr) == S_INNER;
            while (R.v < R.vend) {
                if (runSeek(P, pre, ids, LPR, R)) on = stateOf(P.st, R.pr) == S_INNER;
                const int nh = min(US, min(R.kend, R.vend) - R.v);
                if (on) {  // the same system in the whole warp
                    int row[US], chunk[US];
                    double sum[US];
                    const int sub = lane % LPR;
                    spmvUnits<T, LPR, US>(P, P.A, R, nh, lane, row, chunk, sum,
                                          [&](int c) { return (double)ld(P.s, c); });
#pragma unroll
                    for (int u = 0; u < US; ++u) {
                        double t0 = 0.0, t1 = 0.0;
                        if (u < nh && row[u] < R.rows_end && sub == 0) {
                            const T tt = (T)sum[u];
                            P.t[row[u]] = tt;
                            t0 = (double)tt * (double)ld(P.s, row[u]);
                            t1 = (double)tt * (double)tt;
                        }
                        t0 = warpSum(t0);
                        t1 = warpSum(t1);
                        if (lane == 0 && u < nh) {
                            P.cdot[3 * chunk[u]] = t0;
                            P.cdot[3 * chunk[u] + 1] = t1;
                        }
                    }
                }
                R.v += nh;
            }
        }
        grid.sync();
        // RED(E): omega = (t.s) / (t.t)
        for (int pr = blockIdx.x; pr < P.nprob; pr += gridDim.x) {
            if (stateOf(P.st, pr) != S_INNER) continue;
            const int c0 = P.prob_slice0[pr] * LPR, c1 = P.prob_slice0[pr + 1] * LPR;
            double a = 0.0, b = 0.0;
            for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
                a += ld(P.cdot, 3 * c);
                b += ld(P.cdot, 3 * c + 1);
            }
            blockSum2(a, b, sh);
            if (threadIdx.x == 0) P.st[pr].omega = b > 0.0 ? a / b : 0.0;
            __syncthreads();
        }
        grid.sync();
        // G: d += alpha p + omega s ; r = s - omega t ; r0.r, r.r per slice
        if (runStart(P, pre, ids, m, total, 1, gwarp, nwarps, R)) {
            bool on = stateOf(P.st, R.pr) == S_INNER;
            double alpha = __ldcg(&P.st[R.pr].alpha), omega = __ldcg(&P.st[R.pr].omega);
            while (R.v < R.vend) {
                if (runSeek(P, pre, ids, 1, R)) {
                    on = stateOf(P.st, R.pr) == S_INNER;
                    alpha = __ldcg(&P.st[R.pr].alpha);
                    omega = __ldcg(&P.st[R.pr].omega);
                }
                const int nh = min(UR, min(R.kend, R.vend) - R.v);
                if (on) {  // the same system in the whole warp
                    int rr[UR];
                    T a0[UR], a1[UR], a2[UR], a3[UR], a4[UR];
                    bool ok[UR];
#pragma unroll
                    for (int u = 0; u < UR; ++u) {
                        rr[u] = 32 * (R.slice0 + R.v + u) + lane;
                        ok[u] = u < nh && rr[u] < R.rows_end;
                        if (ok[u]) {
                            a0[u] = ld(P.s, rr[u]);
                            a1[u] = ld(P.d, rr[u]);
                            a2[u] = ld(P.p, rr[u]);
                            a3[u] = ld(P.t, rr[u]);
                            a4[u] = ld(P.r0, rr[u]);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < UR; ++u) {
                        double t0 = 0.0, t1 = 0.0;
                        if (ok[u]) {
                            const double si = (double)a0[u];
                            P.d[rr[u]] = (T)((double)a1[u] + alpha * (double)a2[u] + omega * si);
                            const T rt = (T)(si - omega * (double)a3[u]);
                            P.r[rr[u]] = rt;
                            t0 = (double)a4[u] * (double)rt;
                            t1 = (double)rt * (double)rt;
                        }
                        t0 = warpSum(t0);
                        t1 = warpSum(t1);
                        if (lane == 0 && u < nh) {
                            P.sdot[2 * (R.slice0 + R.v + u)] = t0;
                            P.sdot[2 * (R.slice0 + R.v + u) + 1] = t1;
                        }
                    }
                }
                R.v += nh;
            }
        }
        grid.sync();
        // RED(G): next beta, inner convergence; every system is counted for the next step
        for (int pr = blockIdx.x; pr < P.nprob; pr += gridDim.x) {
            const int stt = stateOf(P.st, pr);
            if (stt == S_INNER) {
                const int c0 = P.prob_slice0[pr], c1 = P.prob_slice0[pr + 1];
                double a = 0.0, b = 0.0;
                for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
                    a += ld(P.sdot, 2 * c);
                    b += ld(P.sdot, 2 * c + 1);
                }
                blockSum2(a, b, sh);
                if (threadIdx.x == 0) {
                    BState& S = P.st[pr];
                    S.fresh = 0;
                    S.iter += 1;
                    S.inner += 1;
                    if (!isfinite(a) || !isfinite(b)) {
                        S.state = S_REFINE;
                    } else if (b <= S.tol2 || S.inner >= P.max_inner || S.omega == 0.0 ||
                               fabs(a) < EPSILON * EPSILON * S.rr0) {
                        S.state = S_REFINE;
                    } else if (S.iter >= P.maxit) {
                        S.stop = 1;
                        S.state = S_REFINE;
                    } else {
                        S.beta = (a / S.rho) * (S.alpha / S.omega);
                        S.rho = a;
                    }
                }
                __syncthreads();
            }
            if (threadIdx.x == 0) {
                const int now = P.st[pr].state;
                if (now == S_INNER || now == S_REFINE) atomicAdd(&P.ctl[2 * nxt], 1);
                if (now == S_REFINE) atomicAdd(&P.ctl[2 * nxt + 1], 1);
            }
        }
        grid.sync();
    }
}

// ---------------------------------------------------------------- setup kernels
constexpr int BS = 256;
inline int grid(int64_t n) { return std::max(1, ceil_div(n, BS)); }

__global__ void shift_kernel(int64_t n, const int* in, int add, int* out) {
    for (int64_t i = blockIdx.x * (int64_t)BS + threadIdx.x; i < n; i += (int64_t)gridDim.x * BS) out[i] = in[i] + add;
}
__global__ void fill_int_kernel(int n, int value, int* out) {
    int i = blockIdx.x * BS + threadIdx.x;
    if (i < n) out[i] = value;
}
// D^-1 of every row (1 on padding rows)
// one system's buffers and its place in the concatenated ones
struct CopyEntry {
    const double* vals;
    const double* b;
    double* x;
    long long nnz, nnz_off, row_off;
    int n;
};
// gather (dir 0: systems -> concatenated values, b, x) or scatter (dir 1: x back);
// blockIdx.y is the system, blockIdx.x strides within it
__global__ void batch_copy_kernel(const CopyEntry* tab, int dir, double* A64, double* b64, double* x64) {
    const CopyEntry e = tab[blockIdx.y];
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
    if (dir == 0) {
        for (long long i = t; i < e.nnz; i += stride) A64[e.nnz_off + i] = e.vals[i];
        for (long long i = t; i < e.n; i += stride) {
            b64[e.row_off + i] = e.b[i];
            x64[e.row_off + i] = e.x[i];
        }
    } else {
        for (long long i = t; i < e.n; i += stride) e.x[i] = x64[e.row_off + i];
    }
}

__global__ void batch_dinv_kernel(int nrows, const int* diag, const double* A64, double* dinv) {
    int r = blockIdx.x * BS + threadIdx.x;
    if (r >= nrows) return;
    const int q = diag[r];
    const double dd = q >= 0 ? A64[q] : 0.0;
    dinv[r] = dd != 0.0 ? 1.0 / dd : 1.0;
}
// inner matrix A D^-1 (column scaling)
template <typename T>
__global__ void batch_scale_kernel(int64_t nnz, const int* col, const double* A64, const double* dinv, T* A) {
    for (int64_t k = blockIdx.x * (int64_t)BS + threadIdx.x; k < nnz; k += (int64_t)gridDim.x * BS)
        A[k] = (T)(A64[k] * dinv[col[k]]);
}
// per system: ||b||^2 and the initial state
__global__ void batch_init_kernel(int nprob, const int* prob_slice0, const int* prob_n, const double* b,
                                  BState* st) {
    __shared__ double sh[2 * MAX_BLOCK / 32];
    for (int pr = blockIdx.x; pr < nprob; pr += gridDim.x) {
        const int r0 = 32 * prob_slice0[pr], n = prob_n[pr];
        double a = 0.0, z = 0.0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) a += b[r0 + i] * b[r0 + i];
        blockSum2(a, z, sh);
        if (threadIdx.x == 0) {
            BState S{};
            S.bb = a;
            S.rho = S.alpha = S.omega = 1.0;
            S.state = a == 0.0 ? S_DONE : S_REFINE;  // b = 0: x = 0 (zeroed below)
            S.status = PRISM_OK;
            st[pr] = S;
        }
        __syncthreads();
    }
}
__global__ void batch_count_kernel(int nprob, const BState* st, int* ctl) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    int a = 0;
    for (int p = 0; p < nprob; ++p) a += st[p].state == S_REFINE ? 1 : 0;
    ctl[0] = a;
    ctl[1] = a;
    ctl[2] = 0;
    ctl[3] = 0;
}
__global__ void zero_b0_kernel(int nprob, const int* prob_slice0, const int* prob_n, const BState* st, double* x) {
    for (int pr = blockIdx.x; pr < nprob; pr += gridDim.x) {
        if (st[pr].state != S_DONE) continue;
        const int r0 = 32 * prob_slice0[pr];
        for (int i = threadIdx.x; i < prob_n[pr]; i += blockDim.x) x[r0 + i] = 0.0;
    }
}

int smCountBatch() {
    static const int c = [] {
        int d = 0, v = 0;
        cudaGetDevice(&d);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d);
        return v > 0 ? v : NUM_SMS;
    }();
    return c;
}

template <typename T>
void* kernelFor(int lpr) {
    if (lpr == 1) return (void*)batch_kernel<T, 1>;
    if (lpr == 2) return (void*)batch_kernel<T, 2>;
    return (void*)batch_kernel<T, 4>;
}

// All blocks co-resident (cooperative launch): one per slot the occupancy allows.
template <typename T>
void launchBatch(const BP<T>& P, int block, int lpr, cudaStream_t s) {
    void* fn = kernelFor<T>(lpr);
    const size_t smem = sizeof(int) * (2 * (size_t)P.nprob + 1 + 2 * (size_t)block + 2);
    if (smem > 48 * 1024) PB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    PB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, block, smem));
    if (per_sm < 1) fail(PRISM_INTERNAL, "batched solver: kernel does not fit on an SM");
    const int blocks = per_sm * smCountBatch();
    BP<T> args = P;
    void* kargs[] = {&args};
    PB_CUDA(cudaLaunchCooperativeKernel(fn, blocks, block, kargs, smem, s));
    countLaunch();
}

template <typename T>
struct InnerBufs {
    T* A;
    T *r, *r0, *p, *v, *s, *t, *d;
};
InnerBufs<float> innerBufs(BatchPlan& pl, float) {
    return {pl.A32f.p, pl.r32.p, pl.r032.p, pl.p32.p, pl.v32.p, pl.s32.p, pl.t32.p, pl.d32.p};
}
InnerBufs<double> innerBufs(BatchPlan& pl, double) {
    return {pl.A32d.p, pl.r64b.p, pl.r064.p, pl.p64.p, pl.v64.p, pl.s64.p, pl.t64.p, pl.d64.p};
}

template <typename T>
std::vector<BatchOut> runBatch(const std::vector<BatchSystem>& sys, BatchPlan& pl, double tol, double itol,
                               int max_inner, int max_pass, long long maxit, cudaStream_t s) {
    const int nrows = pl.nslices * 32;
    auto ensure = [&](auto& buf, size_t n) {
        if (buf.n != n) {
            buf.alloc(n);
            buf.zero(s);
        }
    };
    if constexpr (sizeof(T) == 4) {
        ensure(pl.A32f, pl.nnz);
        for (auto* b : {&pl.r32, &pl.r032, &pl.p32, &pl.v32, &pl.s32, &pl.t32, &pl.d32}) ensure(*b, nrows);
    } else {
        ensure(pl.A32d, pl.nnz);
        for (auto* b : {&pl.r64b, &pl.r064, &pl.p64, &pl.v64, &pl.s64, &pl.t64, &pl.d64}) ensure(*b, nrows);
    }
    InnerBufs<T> ib = innerBufs(pl, T{});
    // the systems' buffers, for the gather and scatter kernels (one grid row per system)
    if (sys.size() > 65535) fail(PRISM_BAD_ARG, "batched solve: at most 65535 systems per call");
    std::vector<CopyEntry> tab(sys.size());
    for (size_t i = 0; i < sys.size(); ++i) {
        const BatchSystem& q = sys[i];
        tab[i] = {q.vals, q.b, q.x, (long long)q.nnz_padded, (long long)pl.nnz_off[i], 32LL * pl.slice0[i], q.n};
    }
    std::vector<uintptr_t> key = {sizeof(T), (uintptr_t)max_inner, (uintptr_t)max_pass, (uintptr_t)maxit};
    for (double v : {tol, itol}) {
        uint64_t bits;
        std::memcpy(&bits, &v, sizeof bits);
        key.push_back((uintptr_t)bits);
    }
    for (const auto& e : tab)
        for (uintptr_t v : {(uintptr_t)e.vals, (uintptr_t)e.b, (uintptr_t)e.x}) key.push_back(v);
    const size_t tab_bytes = tab.size() * sizeof(CopyEntry);
    // graph_key = this prefix (6 entries) + the systems' pointers + the launch shape (2 entries)
    const bool same_systems = pl.graph_key.size() == key.size() + 2 &&
                              std::equal(key.begin() + 6, key.end(), pl.graph_key.begin() + 6);
    if (!same_systems) {
        if (pl.copy_tab.n < tab_bytes) pl.copy_tab.alloc(tab_bytes);
        pl.copy_tab.upload(reinterpret_cast<const unsigned char*>(tab.data()), tab_bytes, s);
    }
    const CopyEntry* dtab = reinterpret_cast<const CopyEntry*>(pl.copy_tab.p);
    const dim3 copy_grid(64, (unsigned)sys.size());
    auto gather = [&] {
        batch_copy_kernel<<<copy_grid, BS, 0, s>>>(dtab, 0, pl.A64.p, pl.b64.p, pl.x64.p); countLaunch();
        batch_dinv_kernel<<<grid(nrows), BS, 0, s>>>(nrows, pl.diag.p, pl.A64.p, pl.dinv.p); countLaunch();
        const int sg = (int)std::min<int64_t>(grid(pl.nnz), NUM_SMS * 32);
        batch_scale_kernel<T><<<sg, BS, 0, s>>>(pl.nnz, pl.col.p, pl.A64.p, pl.dinv.p, ib.A); countLaunch();
        PB_LAUNCH("batched setup");
    };

    BP<T> P{};
    P.nprob = pl.nprob;
    P.nslices = pl.nslices;
    P.slice_prob = pl.slice_prob.p;
    P.prob_slice0 = pl.prob_slice0.p;
    P.prob_n = pl.prob_n.p;
    P.sl_off = pl.sl_off.p;
    P.col = pl.col.p;
    P.A64 = pl.A64.p;
    P.A = ib.A;
    P.b64 = pl.b64.p;
    P.dinv = pl.dinv.p;
    P.x64 = pl.x64.p;
    P.r = ib.r;
    P.r0 = ib.r0;
    P.p = ib.p;
    P.v = ib.v;
    P.s = ib.s;
    P.t = ib.t;
    P.d = ib.d;
    P.cdot = pl.cdot.p;
    P.sdot = pl.cdot.p + 3 * (int64_t)pl.nslices * 4;
    P.st = reinterpret_cast<BState*>(pl.state.p);
    P.ctl = pl.ctl.p;
    P.tol2 = tol * tol;
    P.itol2 = itol * itol;
    P.max_inner = max_inner;
    P.max_pass = max_pass;
    P.maxit = maxit;

    auto init = [&] {
        PB_CUDA(cudaMemsetAsync(ib.d, 0, nrows * sizeof(T), s));
        batch_init_kernel<<<std::min(pl.nprob, NUM_SMS * 4), BS, 0, s>>>(pl.nprob, pl.prob_slice0.p, pl.prob_n.p,
                                                                         pl.b64.p, P.st); countLaunch();
        zero_b0_kernel<<<std::min(pl.nprob, NUM_SMS * 4), BS, 0, s>>>(pl.nprob, pl.prob_slice0.p, pl.prob_n.p, P.st,
                                                                      pl.x64.p); countLaunch();
        batch_count_kernel<<<1, 32, 0, s>>>(pl.nprob, P.st, P.ctl); countLaunch();
        PB_LAUNCH("batched init");
    };
    // autotune the launch shape on this batch: a few steps of every candidate from the same start
    BatchTuning& tune = pl.tune[sizeof(T) == 4 ? 1 : 0];
    if (tune.block == 0) {
        gather();
        DevBuf<double> xsave(nrows);
        PB_CUDA(cudaMemcpyAsync(xsave.p, pl.x64.p, nrows * sizeof(double), cudaMemcpyDeviceToDevice, s));
        cudaEvent_t e0, e1;
        PB_CUDA(cudaEventCreate(&e0));
        PB_CUDA(cudaEventCreate(&e1));
        for (int block : {128, 256, 512}) {
            for (int lpr : {1, 2, 4}) {
                init();
                BP<T> Q = P;
                Q.max_steps = 8;
                PB_CUDA(cudaEventRecord(e0, s));
                launchBatch(Q, block, lpr, s);
                PB_CUDA(cudaEventRecord(e1, s));
                PB_CUDA(cudaEventSynchronize(e1));
                float ms = 0.f;
                PB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
                if (tune.block == 0 || ms < tune.ms) {
                    tune.block = block;
                    tune.lpr = lpr;
                    tune.ms = ms;
                }
                PB_CUDA(cudaMemcpyAsync(pl.x64.p, xsave.p, nrows * sizeof(double), cudaMemcpyDeviceToDevice, s));
            }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        if (verbose())
            std::fprintf(stderr, "[prism] batched solver tuned: block %d, %d lanes per row (%.3f ms for 8 steps)\n",
                         tune.block, tune.lpr, tune.ms);
    }
    // every step is one iteration (plus at most one refinement) of every active system
    P.max_steps = (int)std::min<long long>(maxit + (long long)max_pass + 2, (long long)1 << 30);
    key.push_back((uintptr_t)tune.block);
    key.push_back((uintptr_t)tune.lpr);
    // the call: gather, set-up, the persistent solve and the scatter of the solutions
    auto call = [&] {
        gather();
        init();
        launchBatch(P, tune.block, tune.lpr, s);
        PB_LAUNCH("batched solve");
        batch_copy_kernel<<<copy_grid, BS, 0, s>>>(dtab, 1, pl.A64.p, pl.b64.p, pl.x64.p); countLaunch();
    };
    const auto t0 = std::chrono::steady_clock::now();
    if (pl.graph.g && key == pl.graph_key) {
        PB_CUDA(cudaGraphLaunch(pl.graph.g, s));
        graphLaunchCounter().fetch_add(1, std::memory_order_relaxed);
    } else {
        pl.graph.reset();
        pl.graph_key.clear();
        // a capture that the runtime refuses leaves nothing executed: run the call directly
        cudaGraph_t g = nullptr;
        bool captured = false;
        if (cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed) == cudaSuccess) {
            try {
                call();
                captured = cudaStreamEndCapture(s, &g) == cudaSuccess && g != nullptr;
            } catch (...) {
                cudaStreamEndCapture(s, &g);
            }
            if (captured && cudaGraphInstantiate(&pl.graph.g, g, 0) != cudaSuccess) {
                pl.graph.g = nullptr;
                captured = false;
            }
            if (g) cudaGraphDestroy(g);
        }
        cudaGetLastError();
        if (captured) {
            pl.graph_key = key;
            PB_CUDA(cudaGraphLaunch(pl.graph.g, s));
            graphLaunchCounter().fetch_add(1, std::memory_order_relaxed);
        } else {
            call();
        }
    }
    if (verbose()) {
        PB_CUDA(cudaStreamSynchronize(s));
        std::fprintf(stderr, "[prism] batched solve of %d systems (%d rows): %.3f ms in one graph launch\n", pl.nprob,
                     nrows, std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count());
    }
    std::vector<BState> hs(pl.nprob);
    PB_CUDA(cudaMemcpyAsync(hs.data(), P.st, pl.nprob * sizeof(BState), cudaMemcpyDeviceToHost, s));
    PB_CUDA(cudaStreamSynchronize(s));
    std::vector<BatchOut> out(pl.nprob);
    for (int i = 0; i < pl.nprob; ++i) {
        out[i].iterations = hs[i].iter;
        out[i].passes = hs[i].pass;
        out[i].rel_residual = hs[i].bb > 0 ? std::sqrt(hs[i].rr64 / hs[i].bb) : 0.0;
        out[i].status = hs[i].state == S_DONE ? PRISM_OK
                                              : (hs[i].status != PRISM_OK ? hs[i].status : PRISM_NOT_CONVERGED);
    }
    return out;
}


// ---------------------------------------------------------------- flexible CG over the batch
// Symmetric systems: one flexible CG (krylov.cu) over the block-diagonal matrix, every system
// with its own scalars, preconditioned by one smoothed-aggregation hierarchy of the whole
// (aggregates never straddle systems: nothing couples them). It takes 20-30 iterations where
// Jacobi-BiCGSTAB takes 100-300: 24 systems of 16^3 to 48^3 rows in 4.3 instead of 23.5 ms.
// Reductions are per slice (one warp), then per system (one block, in a fixed order).
struct FState {
    double rr, bb, tol2, dq, dr, alpha, beta, rel;
    long long iter;
    int done;  // as KState::done: 0 running, 1 converged, 2 iteration cap, 3 breakdown, 4 b = 0, 5 non-finite
    int restart, pass, restarts, status;
    int shift;  // scale of r32 (cycleShift)
    int bad;  // the right-hand side, the guess or the matrix is not finite: no system of flexible CG
};
constexpr int FLEX_MIN_ROWS = 8192;
constexpr int FLEX_MAX_ITER = 500;  // iterations (20-30 are usual) after which it has failed
constexpr int FLEX_UNROLL = 2;      // iterations per pass of the device loop

struct FP {
    int nprob, nslices;
    const int *slice_prob, *prob_slice0, *sl_off, *col;
    const double *A, *b;
    double *x, *r, *d, *q, *u, *part;  // part: 3 per slice
    float *r32, *z;
    FState* st;
    double tol;
    long long maxit;
};

__global__ void flex_begin_kernel(const FP P) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P.nprob) return;
    FState z{};
    z.restart = 1;
    z.status = PRISM_OK;
    P.st[p] = z;
}

// f(slice, system) for every slice, one warp each
template <typename F>
__device__ __forceinline__ void forSlices(const FP& P, F f) {
    const int nw = gridDim.x * (BS / 32);
    for (int sl = blockIdx.x * (BS / 32) + (threadIdx.x >> 5); sl < P.nslices; sl += nw) f(sl, P.slice_prob[sl]);
}
template <typename X>
__device__ __forceinline__ double sliceDot(const FP& P, int sl, int lane, const X* __restrict__ v) {
    const int b = P.sl_off[sl], width = (P.sl_off[sl + 1] - b) >> 5;
    double sum = 0.0;
    for (int j0 = 0; j0 < width; j0 += 4) {
        int c[4];
        double m[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j0 + j < width) {
                c[j] = __ldcs(P.col + b + 32 * (j0 + j) + lane);
                m[j] = __ldcs(P.A + b + 32 * (j0 + j) + lane);
            }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j0 + j < width) sum += m[j] * (double)__ldg(v + c[j]);
    }
    return sum;
}
__device__ __forceinline__ void slicePartials(const FP& P, int sl, int lane, double a, double b, double c) {
    a = warpSum(a);
    b = warpSum(b);
    c = warpSum(c);
    if (lane == 0) {
        P.part[3 * (int64_t)sl] = a;
        P.part[3 * (int64_t)sl + 1] = b;
        P.part[3 * (int64_t)sl + 2] = c;
    }
}
// the system's sums of the slice partials, valid in thread 0 (one block per system)
__device__ __forceinline__ void systemSums(const FP& P, int pr, double (&t)[3]) {
    __shared__ double sh[3][BS / 32];
    double v[3] = {0.0, 0.0, 0.0};
    for (int c = P.prob_slice0[pr] + threadIdx.x; c < P.prob_slice0[pr + 1]; c += BS)
        for (int k = 0; k < 3; ++k) v[k] += P.part[3 * (int64_t)c + k];
    for (int k = 0; k < 3; ++k) {
        v[k] = warpSum(v[k]);
        if ((threadIdx.x & 31) == 0) sh[k][threadIdx.x >> 5] = v[k];
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 0; k < 3; ++k) {
            t[k] = 0.0;
            for (int w = 0; w < BS / 32; ++w) t[k] += sh[k][w];
        }
}

// a system that met values that are not finite leaves the cycle, whose coarsest solve couples all
// systems (0 x NaN); the whole block, after thread 0 set done
__device__ __forceinline__ void dropNonfinite(const FP& P, int pr) {
    __syncthreads();
    if (P.st[pr].done != 5) return;
    for (int i = 32 * P.prob_slice0[pr] + threadIdx.x; i < 32 * P.prob_slice0[pr + 1]; i += BS) P.r32[i] = 0.f;
}

// (re)started systems: r = b - A x, d = q = 0
__global__ void __launch_bounds__(BS) flex_init_kernel(const FP P) {
    const int lane = threadIdx.x & 31;
    forSlices(P, [&](int sl, int pr) {
        if (!P.st[pr].restart) return;
        const int i = sl * 32 + lane;
        const double bi = P.b[i], ri = bi - sliceDot(P, sl, lane, P.x);
        P.r[i] = ri;
        P.r32[i] = (float)ri;
        P.d[i] = 0.0;
        P.q[i] = 0.0;
        slicePartials(P, sl, lane, ri * ri, bi * bi, 0.0);
    });
}
__global__ void __launch_bounds__(BS) flex_init_reduce_kernel(const FP P) {
    FState& S = P.st[blockIdx.x];
    if (!S.restart) return;
    double t[3];
    systemSums(P, blockIdx.x, t);
    if (threadIdx.x == 0) {
        S.rr = t[0];
        S.bb = t[1];
        S.tol2 = P.tol * P.tol * t[1];
        S.dq = 1.0;
        S.dr = 0.0;
        S.done = !isfinite(t[0]) || !isfinite(t[1]) ? 5 : t[1] == 0.0 ? 4 : t[0] <= S.tol2 ? 1 : 0;
        if (S.done == 5 && S.pass == 0 && S.restarts == 0) S.bad = 1;
        S.shift = cycleShift(t[0]);
    }
    dropNonfinite(P, blockIdx.x);
    if (S.done == 5 || S.shift == 0) return;
    for (int i = 32 * P.prob_slice0[blockIdx.x] + threadIdx.x; i < 32 * P.prob_slice0[blockIdx.x + 1]; i += BS)
        P.r32[i] = cycleCopy(P.r[i], S.shift);
}
// u = A z ; z.q, z.u, z.r
__global__ void __launch_bounds__(BS) flex_spmv_kernel(const FP P) {
    pdlEnter();
    const int lane = threadIdx.x & 31;
    forSlices(P, [&](int sl, int pr) {
        if (P.st[pr].done) return;
        const int i = sl * 32 + lane;
        const double sum = sliceDot(P, sl, lane, P.z), zi = (double)P.z[i];
        P.u[i] = sum;
        slicePartials(P, sl, lane, zi * P.q[i], zi * sum, zi * P.r[i]);
    });
}
__global__ void __launch_bounds__(BS) flex_direction_kernel(const FP P) {
    pdlEnter();
    FState& S = P.st[blockIdx.x];
    if (S.done) return;
    double t[3];
    systemSums(P, blockIdx.x, t);
    if (threadIdx.x) return;
    const double beta = t[0] / S.dq;
    const double dq = t[1] - beta * t[0], dr = t[2] - beta * S.dr, alpha = dr / dq;
    if (!isfinite(t[0]) || !isfinite(t[1]) || !isfinite(t[2])) S.done = 5;
    else if (!(dq > 0.0) || !isfinite(alpha)) S.done = 3;
    S.beta = beta;
    S.alpha = alpha;
}
// d = z - beta d ; q = u - beta q ; x += alpha d ; r -= alpha q ; r.r, d.q, d.r
__global__ void __launch_bounds__(BS) flex_update_kernel(const FP P) {
    pdlEnter();
    const int lane = threadIdx.x & 31;
    forSlices(P, [&](int sl, int pr) {
        const FState& S = P.st[pr];
        if (S.done) return;
        const double alpha = S.alpha, beta = S.beta;
        const int i = sl * 32 + lane;
        const double di = (double)P.z[i] - beta * P.d[i];
        const double qi = P.u[i] - beta * P.q[i];
        const double ri = P.r[i] - alpha * qi;
        P.x[i] += alpha * di;
        P.d[i] = di;
        P.q[i] = qi;
        P.r[i] = ri;
        P.r32[i] = cycleCopy(ri, S.shift);
        slicePartials(P, sl, lane, ri * ri, di * qi, di * ri);
    });
}
__global__ void __launch_bounds__(BS) flex_convergence_kernel(const FP P) {
    pdlEnter();
    FState& S = P.st[blockIdx.x];
    if (S.done) return;
    double t[3];
    systemSums(P, blockIdx.x, t);
    if (threadIdx.x == 0) {
        S.rr = t[0];
        S.dq = t[1];
        S.dr = t[2];
        S.iter += 1;
        if (!isfinite(t[0]) || !isfinite(t[1])) S.done = 5;
        else if (t[0] <= S.tol2) S.done = 1;
        else if (S.iter >= P.maxit) S.done = 2;
        else if (!(t[1] > 0.0)) S.done = 3;
    }
    dropNonfinite(P, blockIdx.x);
}
// the loop goes on while a system is running
__global__ void flex_running_kernel(const FP P, cudaGraphConditionalHandle loop) {
    int any = 0;
    for (int p = threadIdx.x; p < P.nprob; p += blockDim.x) any |= P.st[p].done == 0;
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) cudaGraphSetConditional(loop, any ? 1u : 0u);
}
// b - A x of every system started in this pass (x = 0 where b = 0)
__global__ void __launch_bounds__(BS) flex_residual_kernel(const FP P) {
    const int lane = threadIdx.x & 31;
    forSlices(P, [&](int sl, int pr) {
        if (!P.st[pr].restart) return;
        const int i = sl * 32 + lane;
        const double e = P.b[i] - sliceDot(P, sl, lane, P.x);
        slicePartials(P, sl, lane, e * e, 0.0, 0.0);
    });
}
__global__ void flex_zero_kernel(const FP P) {
    const int lane = threadIdx.x & 31;
    forSlices(P, [&](int sl, int pr) {
        if (P.st[pr].restart && P.st[pr].done == 4) P.x[sl * 32 + lane] = 0.0;
    });
}
// the end of a pass: accept a system whose true residual meets the tolerance, or start again
// from x (the recursive residual drifted, or the recurrence broke down)
constexpr int FLEX_MAX_PASS = 4;
__global__ void __launch_bounds__(BS) flex_pass_kernel(const FP P) {
    FState& S = P.st[blockIdx.x];
    if (!S.restart) return;
    double t[3];
    systemSums(P, blockIdx.x, t);
    if (threadIdx.x) return;
    S.rel = S.bb > 0.0 ? sqrt(t[0] / S.bb) : 0.0;
    S.restart = 0;
    if (S.done == 1) {
        if (S.rel > P.tol) {
            if (++S.pass < FLEX_MAX_PASS) S.restart = 1;
            else S.status = PRISM_NOT_CONVERGED;
        }
    } else if (S.done == 3) {
        if (++S.restarts > 20) S.status = PRISM_BREAKDOWN;
        else S.restart = 1;
    } else if (S.done == 2) {
        S.status = PRISM_NOT_CONVERGED;
    } else if (S.done == 5 || !isfinite(S.rel)) {
        S.status = PRISM_NONFINITE;
    }
}
__global__ void flex_again_kernel(const FP P, cudaGraphConditionalHandle loop) {
    int any = 0;
    for (int p = threadIdx.x; p < P.nprob; p += blockDim.x) any |= P.st[p].restart;
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) cudaGraphSetConditional(loop, any ? 1u : 0u);
}
__global__ void flex_open_kernel(cudaGraphConditionalHandle loop) { cudaGraphSetConditional(loop, 1u); }

// the block-diagonal CSR pattern, one system per launch: row starts (padding rows empty), columns
__global__ void flex_pattern_kernel(int n, int padded, const int* rowptr, const int* col, int nnz, int row0, int entry0,
                                    int* rp, int* cc) {
    const int t = blockIdx.x * BS + threadIdx.x;
    if (t < padded) rp[row0 + t] = entry0 + (t < n ? rowptr[t] : nnz);
    for (int k = t; k < nnz; k += gridDim.x * BS) cc[entry0 + k] = col[k] + row0;
}

// Solves the batch in one graph launch. FLEX_SHORT: every system came close, but a residual did
// not reach the tolerance in FLEX_MAX_PASS passes; FLEX_FAILED: a system failed (its guess is put
// back). The other systems keep their solutions, which BiCGSTAB then finds converged. A system
// whose input is not finite is no failure.
enum FlexEnd { FLEX_OK, FLEX_SHORT, FLEX_FAILED };
FlexEnd runFlex(const std::vector<BatchSystem>& sys, BatchPlan& pl, double tol, long long maxit, bool own_cap,
             std::vector<BatchOut>& out, cudaStream_t s) {
    const int nrows = pl.nslices * 32;
    if (!pl.rowptr) {
        int64_t nnz = 0;
        for (const auto& q : sys) nnz += q.nnz_csr;
        pl.nnz_csr = nnz;
        pl.rowptr.alloc((size_t)nrows + 1);
        pl.csr_col.alloc(std::max<int64_t>(nnz, 1));
        int64_t off = 0;
        for (size_t i = 0; i < sys.size(); ++i) {
            const BatchSystem& q = sys[i];
            flex_pattern_kernel<<<grid(std::max(32 * q.nslices, 1)), BS, 0, s>>>(
                q.n, 32 * q.nslices, q.rowptr, q.col, (int)q.nnz_csr, 32 * pl.slice0[i], (int)off, pl.rowptr.p, pl.csr_col.p); countLaunch();
            off += q.nnz_csr;
        }
        const int last = (int)nnz;
        PB_CUDA(cudaMemcpyAsync(pl.rowptr.p + nrows, &last, sizeof(int), cudaMemcpyHostToDevice, s));
        PB_CUDA(cudaStreamSynchronize(s));
        for (auto* b : {&pl.fr, &pl.fd, &pl.fq, &pl.fu, &pl.x0}) {
            b->alloc(nrows);
            b->zero(s);
        }
        for (auto* b : {&pl.fr32, &pl.fz32}) {
            b->alloc(nrows);
            b->zero(s);
        }
        pl.fstate.alloc(sizeof(FState) * pl.nprob);
        pl.sa = std::make_unique<SaAmg>();
        pl.sa->max_fill = 100.0;  // as for single systems of these sizes: the other way is Jacobi
        pl.cs = std::make_unique<CaptureStreams>();
    }
    const bool fresh = !pl.sa->built;  // the structure is of this call's matrix
    SellMatrix A;
    A.n = nrows;
    A.nslices = pl.nslices;
    A.nnz_padded = pl.nnz;
    A.sl_off = pl.sl_off.p;
    A.col = pl.col.p;
    A.diag_pos = pl.diag.p;
    A.vals = pl.A64.p;
    A.nnz_csr = pl.nnz_csr;
    FP P{};
    P.nprob = pl.nprob;
    P.nslices = pl.nslices;
    P.slice_prob = pl.slice_prob.p;
    P.prob_slice0 = pl.prob_slice0.p;
    P.sl_off = pl.sl_off.p;
    P.col = pl.col.p;
    P.A = pl.A64.p;
    P.b = pl.b64.p;
    P.x = pl.x64.p;
    P.r = pl.fr.p;
    P.d = pl.fd.p;
    P.q = pl.fq.p;
    P.u = pl.fu.p;
    P.part = pl.cdot.p;
    P.r32 = pl.fr32.p;
    P.z = pl.fz32.p;
    P.st = reinterpret_cast<FState*>(pl.fstate.p);
    P.tol = tol;
    P.maxit = std::min<long long>(2 * std::min<long long>(maxit, FLEX_MAX_ITER), FLEX_MAX_ITER);

    std::vector<CopyEntry> tab(sys.size());
    std::vector<uintptr_t> key = {2, (uintptr_t)P.maxit, 0};
    uint64_t bits;
    std::memcpy(&bits, &tol, sizeof bits);
    key[2] = (uintptr_t)bits;
    for (size_t i = 0; i < sys.size(); ++i) {
        const BatchSystem& q = sys[i];
        tab[i] = {q.vals, q.b, q.x, (long long)q.nnz_padded, (long long)pl.nnz_off[i], 32LL * pl.slice0[i], q.n};
        for (uintptr_t v : {(uintptr_t)q.vals, (uintptr_t)q.b, (uintptr_t)q.x}) key.push_back(v);
    }
    const CopyEntry* dtab = reinterpret_cast<const CopyEntry*>(pl.copy_tab.p);
    const dim3 copy_grid(64, (unsigned)sys.size());
    const int sg = std::max(1, std::min(ceil_div(pl.nslices, BS / 32), NUM_SMS * 8));
    auto gather = [&] {
        batch_copy_kernel<<<copy_grid, BS, 0, s>>>(dtab, 0, pl.A64.p, pl.b64.p, pl.x64.p); countLaunch();
        PB_CUDA(cudaMemcpyAsync(pl.x0.p, pl.x64.p, nrows * sizeof(double), cudaMemcpyDeviceToDevice, s));
    };
    auto scatter = [&] {
        batch_copy_kernel<<<copy_grid, BS, 0, s>>>(dtab, 1, pl.A64.p, pl.b64.p, pl.x64.p); countLaunch();
    };
    if (!(pl.graph.g && key == pl.graph_key)) {
        pl.graph.reset();
        pl.graph_key.clear();
        const size_t bytes = tab.size() * sizeof(CopyEntry);
        if (pl.copy_tab.n < bytes) pl.copy_tab.alloc(bytes);
        pl.copy_tab.upload(reinterpret_cast<const unsigned char*>(tab.data()), bytes, s);
        dtab = reinterpret_cast<const CopyEntry*>(pl.copy_tab.p);
        if (!pl.sa->built) {
            gather();
            pl.sa->setup(A, pl.rowptr.p, pl.csr_col.p, true, false, s);
        }
        PB_CUDA(cudaStreamSynchronize(s));
        cudaStream_t passes = pl.cs->at(0), loop = pl.cs->at(1);
        PB_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed));
        cudaGraph_t g = nullptr;
        try {
            gather();
            pl.sa->setup(A, pl.rowptr.p, pl.csr_col.p, true, false, s);
            flex_begin_kernel<<<grid(pl.nprob), BS, 0, s>>>(P); countLaunch();
            cudaGraphConditionalHandle again = createConditional(s, 0);
            flex_open_kernel<<<1, 1, 0, s>>>(again); countLaunch();
            beginConditional(s, cudaGraphCondTypeWhile, again, passes);
            flex_init_kernel<<<sg, BS, 0, passes>>>(P); countLaunch();
            flex_init_reduce_kernel<<<pl.nprob, BS, 0, passes>>>(P); countLaunch();
            cudaGraphConditionalHandle running = createConditional(passes, 0);
            flex_running_kernel<<<1, BS, 0, passes>>>(P, running); countLaunch();
            beginConditional(passes, cudaGraphCondTypeWhile, running, loop);
            for (int k = 0; k < FLEX_UNROLL; ++k) {
                pl.sa->apply(P.r32, P.z, nullptr, loop);
                launchPdl(flex_spmv_kernel, sg, BS, loop, P);
                launchPdl(flex_direction_kernel, pl.nprob, BS, loop, P);
                launchPdl(flex_update_kernel, sg, BS, loop, P);
                launchPdl(flex_convergence_kernel, pl.nprob, BS, loop, P);
            }
            flex_running_kernel<<<1, BS, 0, loop>>>(P, running); countLaunch();
            endConditional(loop);
            flex_zero_kernel<<<sg, BS, 0, passes>>>(P); countLaunch();
            flex_residual_kernel<<<sg, BS, 0, passes>>>(P); countLaunch();
            flex_pass_kernel<<<pl.nprob, BS, 0, passes>>>(P); countLaunch();
            flex_again_kernel<<<1, BS, 0, passes>>>(P, again); countLaunch();
            endConditional(passes);
            scatter();
        } catch (...) {
            cudaStreamEndCapture(s, &g);
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();
            throw;
        }
        PB_CUDA(cudaStreamEndCapture(s, &g));
        const cudaError_t e = cudaGraphInstantiate(&pl.graph.g, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) pl.graph.g = nullptr;
        PB_CUDA(e);
        pl.graph_key = key;
    }
    PB_CUDA(cudaGraphLaunch(pl.graph.g, s));
    graphLaunchCounter().fetch_add(1, std::memory_order_relaxed);
    std::vector<FState> hs(pl.nprob);
    PB_CUDA(cudaMemcpyAsync(hs.data(), P.st, pl.nprob * sizeof(FState), cudaMemcpyDeviceToHost, s));
    PB_CUDA(cudaStreamSynchronize(s));
    out.assign(pl.nprob, BatchOut{});
    FlexEnd end = FLEX_OK;
    bool nonfinite = false;
    for (int i = 0; i < pl.nprob; ++i) {
        out[i].iterations = (hs[i].iter + 1) / 2;  // in place of BiCGSTAB, as for single systems (krylov.cu)
        out[i].passes = hs[i].pass + 1;
        out[i].rel_residual = hs[i].rel;
        out[i].status = hs[i].status;
        const bool capped = own_cap && hs[i].status == PRISM_NOT_CONVERGED && out[i].iterations >= maxit;
        nonfinite = nonfinite || hs[i].status == PRISM_NONFINITE;
        if (hs[i].status == PRISM_OK || capped || hs[i].bad) continue;
        end = std::max(end, hs[i].done == 1 ? FLEX_SHORT : FLEX_FAILED);
        if (hs[i].done == 1) continue;
        const size_t row = (size_t)32 * pl.slice0[i];
        PB_CUDA(cudaMemcpyAsync(pl.x64.p + row, pl.x0.p + row, sizeof(double) * 32 * (pl.slice0[i + 1] - pl.slice0[i]),
                                cudaMemcpyDeviceToDevice, s));
    }
    if (verbose()) {
        long long most = 0;
        for (const auto& q : out) most = std::max<long long>(most, q.iterations);
        std::fprintf(stderr, "[prism] batched flexible CG of %d systems (%d rows): at most %lld iterations, %s\n", pl.nprob,
                     nrows, most, end == FLEX_OK ? "ok" : end == FLEX_SHORT ? "residuals above the tolerance" : "failed");
    }
    if (end == FLEX_FAILED) {
        scatter();
        PB_CUDA(cudaStreamSynchronize(s));  // the systems' own streams go on with the guesses
    }
    // a structure built from such values goes, and one that failed on the matrices of another call
    if (nonfinite ? fresh : end == FLEX_FAILED && !fresh) {
        pl.sa->built = false;
        pl.graph.reset();
        pl.graph_key.clear();
    }
    return end;
}

}  // namespace

std::vector<BatchOut> solveBatch(const std::vector<BatchSystem>& sys, BatchPlan& pl, bool mixed, double tol,
                                 double itol, int max_inner, int max_pass, long long maxit, bool own_cap,
                                 cudaStream_t s) {
    if (sys.empty()) return {};
    std::vector<uintptr_t> key;
    for (const auto& q : sys) {
        key.push_back((uintptr_t)q.sl_off);
        key.push_back((uintptr_t)q.sl_col);
        key.push_back((uintptr_t)q.n);
        key.push_back((uintptr_t)q.nnz_padded);
    }
    if (key != pl.key) {
        BatchPlan fresh;
        pl = std::move(fresh);
        pl.key = key;
        pl.nprob = (int)sys.size();
        std::vector<int> prob_slice0(pl.nprob + 1), prob_n(pl.nprob);
        pl.nnz_off.resize(pl.nprob + 1);
        pl.slice0.resize(pl.nprob + 1);
        int64_t nnz = 0;
        int64_t ns = 0;
        for (int i = 0; i < pl.nprob; ++i) {
            pl.nnz_off[i] = nnz;
            pl.slice0[i] = (int)ns;
            prob_slice0[i] = (int)ns;
            prob_n[i] = sys[i].n;
            nnz += sys[i].nnz_padded;
            ns += sys[i].nslices;
        }
        if (nnz >= ((int64_t)1 << 31) || ns * 32 >= ((int64_t)1 << 31) / 4)
            fail(PRISM_BAD_ARG, "batched solver: batch too large for 32-bit indices");
        if (pl.nprob > 16384) fail(PRISM_BAD_ARG, "batched solver: at most 16384 systems per batch");
        pl.nnz_off[pl.nprob] = nnz;
        pl.slice0[pl.nprob] = (int)ns;
        prob_slice0[pl.nprob] = (int)ns;
        pl.nnz = nnz;
        pl.nslices = (int)ns;
        const int nrows = pl.nslices * 32;
        pl.prob_slice0.upload(prob_slice0, s);
        pl.prob_n.upload(prob_n, s);
        pl.slice_prob.alloc(ns);
        pl.sl_off.alloc(ns + 1);
        pl.col.alloc(std::max<int64_t>(nnz, 1));
        pl.diag.alloc(nrows);
        fill_int_kernel<<<grid(nrows), BS, 0, s>>>(nrows, -1, pl.diag.p); countLaunch();
        for (int i = 0; i < pl.nprob; ++i) {
            const BatchSystem& q = sys[i];
            fill_int_kernel<<<grid(q.nslices), BS, 0, s>>>(q.nslices, i, pl.slice_prob.p + pl.slice0[i]); countLaunch();
            shift_kernel<<<grid(q.nslices), BS, 0, s>>>(q.nslices, q.sl_off, (int)pl.nnz_off[i],
                                                        pl.sl_off.p + pl.slice0[i]); countLaunch();
            const int gs = (int)std::min<int64_t>(grid(q.nnz_padded), NUM_SMS * 8);
            shift_kernel<<<gs, BS, 0, s>>>(q.nnz_padded, q.sl_col, 32 * pl.slice0[i], pl.col.p + pl.nnz_off[i]); countLaunch();
            shift_kernel<<<grid(q.n), BS, 0, s>>>(q.n, q.diag_pos, (int)pl.nnz_off[i],
                                                  pl.diag.p + 32 * (int64_t)pl.slice0[i]); countLaunch();
        }
        const int last = (int)nnz;
        PB_CUDA(cudaMemcpyAsync(pl.sl_off.p + ns, &last, sizeof(int), cudaMemcpyHostToDevice, s));
        pl.A64.alloc(std::max<int64_t>(nnz, 1));
        for (auto* b : {&pl.x64, &pl.b64, &pl.dinv}) {
            b->alloc(nrows);
            b->zero(s);
        }
        pl.cdot.alloc((size_t)ns * 4 * 3 + (size_t)ns * 2);
        pl.state.alloc(sizeof(BState) * pl.nprob);
        pl.ctl.alloc(4);
        PB_CUDA(cudaStreamSynchronize(s));
        PB_LAUNCH("batched plan");
    }
    int64_t rows = 0, entries = 0;
    bool symmetric = !pl.no_flex && !fp64Cycles();
    for (const auto& q : sys) {
        rows += q.n;
        entries += q.nnz_csr;
        symmetric = symmetric && q.symmetric;
    }
    std::vector<BatchOut> flex(sys.size());
    bool failed = false;
    if (symmetric && rows >= FLEX_MIN_ROWS && entries < ((int64_t)1 << 29) && sys.size() <= 65535) {
        try {
            const FlexEnd end = runFlex(sys, pl, tol, maxit, own_cap, flex, s);
            if (end == FLEX_OK) {
                pl.look_at_dominance = false;
                return flex;
            }
            failed = end == FLEX_FAILED;
        } catch (const Error& e) {
            if (!hierarchyDidNotFit(e)) throw;
            // the persistent launch needs a fraction of this memory; nothing was written back yet
            pl.sa.reset();
            for (auto* b : {&pl.fr, &pl.fd, &pl.fq, &pl.fu, &pl.x0}) b->release();
            for (auto* b : {&pl.fr32, &pl.fz32}) b->release();
            for (auto* b : {&pl.rowptr, &pl.csr_col}) b->release();
            pl.fstate.release();
            pl.no_flex = true;
        }
    }
    // flexible CG's iterations count, and against a cap of the caller's
    long long used = 0;
    for (const auto& f : flex) used = std::max<long long>(used, f.iterations);
    const long long left = own_cap ? maxit - used : maxit;
    if (left <= 0) return flex;
    std::vector<BatchOut> out = mixed ? runBatch<float>(sys, pl, tol, itol, max_inner, max_pass, left, s)
                                      : runBatch<double>(sys, pl, tol, itol, max_inner, max_pass, left, s);
    for (size_t i = 0; i < out.size(); ++i) {
        out[i].iterations += flex[i].iterations;
        // values that are not finite in one system's matrix reach all of them, and say nothing
        // about the method
        failed = failed && out[i].status != PRISM_NONFINITE;
    }
    if (failed) (pl.look_at_dominance ? pl.no_flex : pl.look_at_dominance) = true;
    return out;
}

}  // namespace pb
