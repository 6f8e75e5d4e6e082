// small.cu -- a whole ISolver::solve of a small system in one launch of one thread-block
// cluster: the scaled residuals, the outer steps, and in each of them Jacobi-preconditioned
// BiCGSTAB with its restarts and accurate-residual passes (bicgstab() in krylov.cu, whose
// control flow and statuses these are).
//
// Systems of a few thousand rows are bound by launches, not by bytes: an iteration as five
// kernels takes 17 us whatever the size (32^2 to 31^3 rows), and a solve that has nothing to
// do still 130 us. Here a thread owns two or four rows: their vectors stay in registers, the
// matrix in L1, and only the two preconditioned directions pass through shared memory, read
// by the cluster's other blocks as distributed shared memory. An iteration is five barriers,
// three of them carrying a reduction (each block sends its partial sums to every other block
// before it arrives, and all add them in block order, so results repeat bit for bit).
#include <algorithm>
#include <cmath>

#include "cluster.cuh"
#include "krylov.h"

namespace pb {

namespace {

constexpr int NV = 3;  // values of one reduction, at most

struct SmallParams {
    int n;
    const int* sl_off;
    const int* col;
    const double* vals;
    const int* diag_pos;
    const double* b;
    double* x;
    long long from, n_iter, maxit;  // outer steps from <= step < n_iter
    double eps, tol;
    int symmetric;  // the matrix is symmetric by construction
    SolveCtl* out;
};

// THREADS threads of K rows each per block, the first KEPT entries of a row in registers; CL:
// more than one block
template <int THREADS, int K, int KEPT, bool CL>
__global__ void __launch_bounds__(THREADS, 1) small_solve_kernel(const SmallParams P) {
    constexpr int ROWS = THREADS * K;  // rows per block
    __shared__ double ph[ROWS], sh[ROWS];  // the gathered vectors: M^-1 p (or x), M^-1 s
    __shared__ ClusterShared<THREADS, NV> shared;
    ClusterReduce<THREADS, CL, NV> R(shared);
    const int rank = R.rank;

    // the first KEPT entries of a row stay in registers
    int row[K], at[K], width[K], kcol[K][KEPT + 1];
    double kval[K][KEPT + 1];
    double dinv[K], x[K], r[K], r0[K], p[K], v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        row[k] = rank * ROWS + k * THREADS + threadIdx.x;
        const bool in = row[k] < P.n;
        const int s0 = in ? P.sl_off[row[k] >> 5] : 0;
        width[k] = in ? (P.sl_off[(row[k] >> 5) + 1] - s0) >> 5 : 0;
        at[k] = s0 + (row[k] & 31);
        const double d = in ? P.vals[P.diag_pos[row[k]]] : 1.0;
        dinv[k] = d != 0.0 ? 1.0 / d : 1.0;
        x[k] = in ? P.x[row[k]] : 0.0;
        r[k] = r0[k] = p[k] = v[k] = 0.0;
#pragma unroll
        for (int j = 0; j < KEPT; ++j)
            if (j < width[k]) {
                kcol[k][j] = __ldg(P.col + at[k] + 32 * j);
                kval[k][j] = __ldg(P.vals + at[k] + 32 * j);
            }
    }
    auto rhs = [&](int k) { return row[k] < P.n ? __ldg(P.b + row[k]) : 0.0; };
    auto own = [&](int k) { return k * THREADS + (int)threadIdx.x; };
    auto gather = [&](double* a, int j) -> double {
        if constexpr (CL) return *R.cl.map_shared_rank(a + (j & (ROWS - 1)), j / ROWS);
        else return a[j];
    };
    // (A y)_row with y spread over the blocks' shared array a; up to 4 entries in flight
    auto rowOf = [&](int k, double* a) {
        double sum = 0.0;
#pragma unroll
        for (int j = 0; j < KEPT; ++j)
            if (j < width[k]) sum += kval[k][j] * gather(a, kcol[k][j]);
        for (int j0 = KEPT; j0 < width[k]; j0 += 4) {
            int c[4];
            double m[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j0 + j < width[k]) {
                    c[j] = __ldg(P.col + at[k] + 32 * (j0 + j));
                    m[j] = __ldg(P.vals + at[k] + 32 * (j0 + j));
                }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j0 + j < width[k]) sum += m[j] * gather(a, c[j]);
        }
        return sum;
    };
    // ax := A x
    double ax[K];
    auto applyToX = [&] {
#pragma unroll
        for (int k = 0; k < K; ++k) ph[own(k)] = x[k];
        R.barrier();
#pragma unroll
        for (int k = 0; k < K; ++k) ax[k] = row[k] < P.n ? rowOf(k, ph) : 0.0;
    };
    // max|A x - b| / (max|diag x| + eps) from ax; NaN if a term is not finite
    auto scaledResidual = [&] {
        double m[NV] = {};
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (row[k] >= P.n) continue;
            const double e = fabs(ax[k] - rhs(k)), d = fabs(P.vals[P.diag_pos[row[k]]] * x[k]);
            if (!isfinite(e) || !isfinite(d)) {
                m[2] = 1.0;
            } else {
                m[0] = fmax(m[0], e);
                m[1] = fmax(m[1], d);
            }
        }
        R.template all<3, true>(m);
        return m[2] != 0.0 ? __longlong_as_double(0x7ff8000000000000LL) : m[0] / (m[1] + EPSILON);
    };

    double init_res = 0.0, cur_res = 0.0, krylov_rel = 0.0;
    int status = PRISM_OK, converged = 0;
    long long outer = P.from, total = 0;
    bool cg_ok = P.symmetric != 0;
    if (P.from > 0) {  // go on from the record of the launches before
        if (P.out->converged || P.out->outer < P.from) return;
        init_res = P.out->init_res;
        status = P.out->status;
        total = P.out->krylov_iterations;
        cg_ok = cg_ok && !P.out->no_cg;
        R.barrier();  // every block has started before the first write to another's memory
    } else if (P.n_iter > 0) {
        applyToX();
        init_res = scaledResidual();
    }
    // conjugate gradients where the matrix is symmetric and, by its signs and row sums,
    // positive semi-definite: half the products and a third of the reductions of BiCGSTAB. Two of
    // its iterations, with the products of one of BiCGSTAB, count as one: a cap that was enough stays so
    if (cg_ok && P.n_iter > 0) {
        double bad[NV] = {};
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double sum = 0.0, d = 0.0;
            for (int j = 0; j < width[k]; ++j) {
                const double a = __ldg(P.vals + at[k] + 32 * j);
                if (__ldg(P.col + at[k] + 32 * j) == row[k]) d += a;
                else if (a > 0.0) bad[0] = 1.0;
                sum += a;
            }
            if (row[k] < P.n && !(d > 0.0 && sum >= -1e-12 * d)) bad[0] = 1.0;
        }
        R.template all<1, true>(bad);
        cg_ok = bad[0] == 0.0;
    }
    while (outer < P.n_iter) {
        long long left = P.maxit;
        int kstatus = PRISM_OK;
        for (int pass = 0; pass < 4; ++pass) {
            long long iter = 0;
            int restarts = 0, done = 0;
            kstatus = PRISM_OK;
            while (true) {
                applyToX();
                double d[NV] = {};
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const double bk = rhs(k);
                    r[k] = r0[k] = bk - ax[k];
                    p[k] = v[k] = 0.0;
                    d[0] += r[k] * r[k];
                    d[1] += bk * bk;
                }
                R.template all<2>(d);
                const double r0sq = d[0], tol2 = P.tol * P.tol * d[1];
                double rho = d[0], beta = d[0], w = 1.0;
                long long iter_cg = 0;
                done = !isfinite(d[0]) || !isfinite(d[1]) ? 5 : d[1] == 0.0 ? 4 : d[0] <= tol2 ? 1 : 0;
                if (cg_ok) {
                    // Chronopoulos and Gear 1989: one reduction per iteration; q = A p is carried in v
                    double gamma_old = 1.0, alpha = 1.0;
                    beta = 0.0;
                    while (done == 0) {
                        double z[K], az[K];
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            z[k] = dinv[k] * r[k];
                            ph[own(k)] = z[k];
                        }
                        R.barrier();
                        d[0] = d[1] = d[2] = 0.0;
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            az[k] = rowOf(k, ph);
                            d[0] += r[k] * z[k];
                            d[1] += az[k] * z[k];
                            d[2] += r[k] * r[k];
                        }
                        R.template all<3>(d);
                        if (!isfinite(d[0]) || !isfinite(d[1]) || !isfinite(d[2])) done = 5;
                        else if (d[2] <= tol2) done = 1;
                        else if (iter >= left && iter_cg % 2 == 0) done = 2;
                        if (done) break;
                        beta = iter_cg > 0 ? d[0] / gamma_old : 0.0;
                        const double pq = d[1] - (iter_cg > 0 ? beta * d[0] / alpha : 0.0);
                        alpha = d[0] / pq;
                        if (!(pq > 0.0) || !isfinite(alpha)) {
                            done = 3;
                            cg_ok = false;
                            break;
                        }
                        gamma_old = d[0];
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            p[k] = z[k] + beta * p[k];
                            v[k] = az[k] + beta * v[k];
                            x[k] += alpha * p[k];
                            r[k] -= alpha * v[k];
                        }
                        if (++iter_cg % 2 == 1) ++iter;
                    }
                } else if (done == 0 && iter >= left) {
                    done = 2;  // conjugate gradients broke down within the last pair
                }
                while (done == 0) {
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        p[k] = r[k] + beta * (p[k] - w * v[k]);
                        ph[own(k)] = dinv[k] * p[k];
                    }
                    R.barrier();
                    d[0] = 0.0;
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        v[k] = rowOf(k, ph);
                        d[0] += r0[k] * v[k];
                    }
                    R.template all<1>(d);
                    const double alpha = rho / d[0];
                    if (d[0] == 0.0 || !isfinite(alpha)) {  // breakdown: restart from the current x
                        done = isfinite(d[0]) ? 3 : 5;
                        break;
                    }
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        r[k] -= alpha * v[k];  // s
                        sh[own(k)] = dinv[k] * r[k];
                    }
                    R.barrier();
                    double t[K];  // A M^-1 s
                    d[0] = d[1] = 0.0;
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        t[k] = rowOf(k, sh);
                        d[0] += t[k] * r[k];
                        d[1] += t[k] * t[k];
                    }
                    R.template all<2>(d);
                    w = d[1] > 0.0 ? d[0] / d[1] : 0.0;
                    // r0.r of the updated r (as r0.s - w r0.t it loses its accuracy where r
                    // vanishes on r0's support: krylov.cu)
                    d[0] = d[1] = 0.0;
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        x[k] += alpha * (dinv[k] * p[k]) + w * (dinv[k] * r[k]);
                        r[k] -= w * t[k];
                        d[0] += r0[k] * r[k];
                        d[1] += r[k] * r[k];
                    }
                    R.template all<2>(d);
                    ++iter;
                    const double rho_new = d[0], rr = d[1];
                    if (!isfinite(rho_new) || !isfinite(rr)) done = 5;
                    else if (rr <= tol2) done = 1;
                    else if (iter >= left) done = 2;
                    else if (w == 0.0 || fabs(rho_new) < EPSILON * EPSILON * r0sq) done = 3;
                    else {
                        beta = (rho_new / rho) * (alpha / w);
                        rho = rho_new;
                    }
                }
                if (done != 3) break;
                if (++restarts > 20) {
                    kstatus = PRISM_BREAKDOWN;
                    break;
                }
            }
            if (done == 2) kstatus = PRISM_NOT_CONVERGED;
            if (done == 5) kstatus = PRISM_NONFINITE;
            if (done == 4) {  // b = 0: x = 0
#pragma unroll
                for (int k = 0; k < K; ++k) x[k] = 0.0;
            }
            total += iter;
            left -= iter;
            // accurate residual: the recursive one drifts from b - A x
            applyToX();
            double d[NV] = {};
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const double bk = rhs(k), e = bk - ax[k];
                d[0] += e * e;
                d[1] += bk * bk;
            }
            R.template all<2>(d);
            krylov_rel = d[1] > 0 ? sqrt(d[0] / d[1]) : 0.0;
            if (kstatus != PRISM_OK || krylov_rel <= 10 * P.tol || left <= 0 || d[1] == 0) break;
        }
        cur_res = scaledResidual();
        ++outer;
        if (kstatus != PRISM_OK && status == PRISM_OK) status = kstatus;
        if (isnan(cur_res)) status = PRISM_NONFINITE;
        if (cur_res < P.eps) {
            converged = 1;
            break;
        }
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (row[k] < P.n) P.x[row[k]] = x[k];
    if (rank == 0 && threadIdx.x == 0) {
        SolveCtl z{};
        z.n_iter = P.n_iter;
        z.outer = outer;
        z.eps = P.eps;
        z.init_res = init_res;
        z.cur_res = cur_res;
        z.converged = converged;
        z.status = status;
        z.kmax = P.maxit;
        z.krylov_iterations = total;
        z.tol = P.tol;
        z.krylov_rel = krylov_rel;
        z.no_cg = !cg_ok;
        *P.out = z;
    }
}

// blocks of the largest cluster the device places (8 is always allowed)
int maxCtas() {
    static PerDevice c;
    return c.get([] {
        return clusterPlaced(small_solve_kernel<256, 1, 7, true>, 256) &&
                       clusterPlaced(small_solve_kernel<512, 2, 5, true>, 512) &&
                       clusterPlaced(small_solve_kernel<512, 2, 7, true>, 512) &&
                       clusterPlaced(small_solve_kernel<512, 4, 0, true>, 512)
                   ? CLUSTER_MAX
                   : 8;
    });
}

template <int T, int K, int KEPT>
void launchSmall(const SmallParams& P, cudaStream_t s) {
    const int ctas = ceil_div(P.n, T * K);
    if (ctas == 1) launchCluster(small_solve_kernel<T, K, KEPT, false>, 1, T, s, false, P);
    else launchCluster(small_solve_kernel<T, K, KEPT, true>, ctas, T, s, false, P);
}

// iterations that one launch holds at most: 5 s at 4.6 us a pair of CG iterations on 1,024 rows, 10 s at
// 10 us a BiCGSTAB iteration on 32,768
constexpr long long LAUNCH_ITERATIONS = 1LL << 20;

}  // namespace

bool smallSolveFits(const SellMatrix& A, long long maxit, long long n_iter) {
    return A.n > 0 && A.n <= maxCtas() * 2048 && maxit <= LAUNCH_ITERATIONS && n_iter <= 4096;
}

// Rows per block: one block up to 1,024 rows, whose barriers cost a fraction of a cluster's;
// then as few rows per block as 16 blocks allow. Entries kept in registers (two rows per
// thread): five for the rows of 2-D meshes (32^2 Poisson 0.31 ms, with seven 0.37, none 0.39),
// seven for longer ones (22^3 transport 4.46 ms, with five 4.94, none 5.25); four rows per
// thread leave no room.
long long smallSolve(const SellMatrix& A, const double* b, double* x, long long from, long long n_iter, double eps,
                     double tol, long long maxit, bool symmetric, SolveCtl* out, cudaStream_t s) {
    const long long to = std::min(n_iter, from + std::max(1LL, LAUNCH_ITERATIONS / std::max(1LL, maxit)));
    const SmallParams P{A.n, A.sl_off, A.col, A.vals, A.diag_pos, b, x, from, to, maxit, eps, tol, symmetric ? 1 : 0, out};
    const int max = maxCtas();
    const bool two = (A.n > 256 && A.n <= 1024) || (A.n > max * 256 && A.n <= max * 1024);
    if (two && A.nnz_padded <= 5LL * 32 * A.nslices) launchSmall<512, 2, 5>(P, s);
    else if (two) launchSmall<512, 2, 7>(P, s);
    else if (A.n <= max * 256) launchSmall<256, 1, 7>(P, s);
    else launchSmall<512, 4, 0>(P, s);
    return to;
}

}  // namespace pb
