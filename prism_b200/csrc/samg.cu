// samg.cu -- smoothed-aggregation multigrid (Vanek, Mandel and Brezina 1996): the FP32
// V-cycle that preconditions flexible CG on symmetric positive (semi-)definite systems and
// BiCGSTAB on convection-diffusion.
//
//   * Aggregates: a maximal independent set at distance two of the strong couplings
//     (w_ij = |a_ij| / sqrt(a_ii a_jj) >= 0.25 of the larger of both rows' strongest),
//     found in rounds of neighbour maxima over hashed priorities (Bell, Dalton and Olson
//     2012); the rows next to a root join it, the rows beyond join their strongest
//     neighbour's aggregate. Deterministic: integer maxima only.
//   * Prolongation P = (I - omega_p D^-1 A) P0, Galerkin operators P^T A P. A smoothed
//     prolongation needs about half the iterations of a piecewise-constant one and its
//     aggregates of 7-11 rows leave fewer, smaller levels (2.1M-cell cavity: 5 levels
//     against 7), which matters as much: the coarse levels are latency-bound.
//   * Cycle: V(1,1) with damped Jacobi. With Q = (I - omega D^-1 A) P, the whole cycle of a level is two passes:
//       down   b_next = Q^T b          (pre-smoothing from zero, residual, restriction)
//              y = omega D^-1 (2 b - A omega D^-1 b)   (both smoothing steps of b itself)
//       up     x = y + Q x_next        (prolongation and its post-smoothing)
//     because the post-smoothed prolongation (I - omega D^-1 A) P is Q.
//     The two halves of `down` share a launch; A is stored scaled by omega D^-1, so its
//     pass gathers one vector. Q^T and Q hold fewer entries than A on 2-D meshes.
//   * The smallest levels (TAIL_ROWS, TAIL_NNZ) run in one launch of a thread-block cluster.
// The structure is built once per pattern; every new matrix refreshes
// the values by gathers in a fixed order. For a symmetric matrix (A P)^T stands for P^T A;
// otherwise the restriction is smoothed with A^T's values: R^T = (I - omega_p D^-1 A^T) P0
// takes P^T's place and (S R^T)^T, S with A^T, that of Q^T (Sala and Tuminaro 2008).
#include <cub/cub.cuh>

#include <atomic>
#include <chrono>
#include <cmath>
#include <type_traits>

#include "amg.h"
#include "cluster.cuh"
#include "samg.h"

namespace pb {

namespace {

constexpr int BS = 256;
constexpr int WARPS = BS / 32;
constexpr int COARSE_MAX = 96;  // rows solved by a dense inverse
constexpr int MAX_LEVELS = 12;
constexpr int MIS_ROUNDS = 24;   // 6-9 rounds leave nothing undecided on the meshes seen
constexpr int MIS_BATCH = 8;     // rounds between two looks at the number left
constexpr double STRONG = 0.25;
// Coarse symmetric levels are smoothed (omega 1.1) and their prolongation is smoothed (0.95) as if
// the spectrum of D^-1 A ended near 1.5, which holds for diffusion. With a time term it may reach 3 from
// the third level on, where both amplify: 2.1M rows with off-diagonal sums of 0.9 of the diagonal took
// 242 iterations, of 0.8 13. A diagonal raised to half of its row's sum keeps it below 2 (15 iterations, as
// many as before without a time term; 1.8 costs 5-8% more there, for convection the bound only costs).
constexpr double SPECTRUM = 2.0;
// Products per entry (A P: of A; P^T A P: of P and A P) beyond which a row that does not fit its
// table makes the hierarchy give way to one with a piecewise-constant prolongation: a row coupled to
// all others fills A P. Meshes have 2 to 10; one such row among 26,000 has 740, whose structure and
// values took 26 s against 1 s.
constexpr long long MAX_PRODUCTS = 32;

inline int grid(int64_t n) { return std::max(1, ceil_div(n, BS)); }

// ---------------------------------------------------------------- structure
__device__ __forceinline__ double valueAt(const double* vals, const int* csr_pos, int k) {
    if (!csr_pos) return vals[k];
    const int at = csr_pos[k];
    return at >= 0 ? vals[at] : 0.0;
}

__global__ void csr_pos_kernel(int n, const int* rowptr, const int* sl_off, int* csr_pos) {
    const int r = blockIdx.x * BS + threadIdx.x;
    if (r >= n) return;
    const int base = sl_off[r >> 5] + (r & 31);
    for (int k = rowptr[r]; k < rowptr[r + 1]; ++k) csr_pos[k] = base + 32 * (k - rowptr[r]);
}

// D^-1 and omega D^-1 (0 for a zero diagonal). bound > 0: a diagonal below 1/bound of its row's sum of
// magnitudes is taken as that, which keeps the spectrum of D^-1 A within it
__global__ void scaling_kernel(int n, const int* rowptr, const int* col, const int* csr_pos, const double* vals,
                               double omega, double bound, double* dinv, float* wd) {
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i >= n) return;
    double d = 0.0, sum = 0.0;
    for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) {
        const double a = valueAt(vals, csr_pos, k);
        if (col[k] == i) d = a;
        sum += fabs(a);
    }
    if (bound > 0.0 && d != 0.0 && sum > bound * fabs(d)) d = copysign(sum / bound, d);
    const double di = d != 0.0 ? 1.0 / d : 0.0;
    dinv[i] = di;
    wd[i] = (float)(omega * di);
}

// |a_ij| / sqrt(a_ii a_jj), a_ij averaged with a_ji where the matrix is not symmetric
__device__ __forceinline__ float coupling(const int* csr_pos, const int* tr_pos, const double* vals, int k, double di,
                                          double dj) {
    double a = fabs(valueAt(vals, csr_pos, k));
    if (tr_pos) a = 0.5 * (a + (tr_pos[k] >= 0 ? fabs(vals[tr_pos[k]]) : 0.0));
    return (float)(a * sqrt(fabs(di * dj)));
}

// place in vals of the transposed entry of every CSR entry (-1: none)
__global__ void transposed_kernel(int n, const int* rowptr, const int* col, const int* csr_pos, int* tr_pos) {
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i >= n) return;
    for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) {
        const int j = col[k];
        int at = -1;
        if (csr_pos) {  // level 0: columns in the mesh's order
            for (int q = rowptr[j]; q < rowptr[j + 1]; ++q)
                if (col[q] == i) at = csr_pos[q];
        } else {
            int lo = rowptr[j], hi = rowptr[j + 1];
            const int end = hi;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (col[mid] < i) lo = mid + 1;
                else hi = mid;
            }
            if (lo < end && col[lo] == i) at = lo;
        }
        tr_pos[k] = at;
    }
}

__global__ void strongest_kernel(int n, const int* rowptr, const int* col, const int* csr_pos, const int* tr_pos,
                                 const double* vals, const double* dinv, float* wmax) {
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i >= n) return;
    float best = 0.f;
    const double di = dinv[i];
    for (int k = rowptr[i]; k < rowptr[i + 1]; ++k)
        if (col[k] != i) best = fmaxf(best, coupling(csr_pos, tr_pos, vals, k, di, dinv[col[k]]));
    wmax[i] = best;
}

// strong[k] = the column of a strong entry, else the row itself (which every neighbour
// maximum below includes anyway)
__global__ void strong_kernel(int n, const int* rowptr, const int* col, const int* csr_pos, const int* tr_pos,
                              const double* vals, const double* dinv, const float* wmax, int* strong) {
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i >= n) return;
    const double di = dinv[i];
    const float wi = wmax[i];
    for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) {
        const int j = col[k];
        const float w = j == i ? 0.f : coupling(csr_pos, tr_pos, vals, k, di, dinv[j]);
        strong[k] = (w > 0.f && w >= (float)STRONG * fmaxf(wi, wmax[j])) ? j : i;
    }
}

// priority of a row: undecided 1 | hash | index; in the set 3 << 62; out 0
constexpr unsigned long long MIS_IN = 3ull << 62;
__global__ void mis_init_kernel(int n, unsigned long long* key, int* undecided) {
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i == 0) undecided[0] = n;
    if (i >= n) return;
    unsigned long long h = ((unsigned long long)i + 0x632BE59BD9B4E019ull) * 0x9E3779B97F4A7C15ull;
    h ^= h >> 31;
    h *= 0xBF58476D1CE4E5B9ull;
    h ^= h >> 29;
    key[i] = (1ull << 62) | ((h >> 34) << 32) | (unsigned)i;
}
__global__ void mis_near_kernel(int n, const int* rowptr, const int* strong, const unsigned long long* key,
                                unsigned long long* near, const int* undecided) {
    if (*undecided == 0) return;
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i >= n) return;
    unsigned long long m = key[i];
    for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) m = max(m, key[strong[k]]);
    near[i] = m;
}
__global__ void mis_decide_kernel(int n, const int* rowptr, const int* strong, unsigned long long* key,
                                  const unsigned long long* near, const int* undecided, int* left) {
    if (*undecided == 0) return;
    const int i = blockIdx.x * BS + threadIdx.x;
    bool open = false;
    if (i < n) {
        const unsigned long long mine = key[i];
        if (mine != 0 && mine != MIS_IN) {
            unsigned long long m = near[i];
            for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) m = max(m, near[strong[k]]);
            if (m == mine) key[i] = MIS_IN;
            else if (m == MIS_IN) key[i] = 0;
            else open = true;
        }
    }
    const int c = __syncthreads_count(open);
    if (threadIdx.x == 0 && c) atomicAdd(left, c);
}
// in the set (or still undecided after every round); a row without couplings needs no coarse
// row: the smoother solves it
__global__ void mis_root_kernel(int n, const unsigned long long* key, const float* wmax, int* root) {
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i < n) root[i] = key[i] != 0 && wmax[i] > 0.f;
}
__global__ void root_label_kernel(int n, const int* root, const int* id, int* label) {
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i < n) label[i] = root[i] ? id[i] : -1;
}
// an unlabelled row joins its strongest labelled strong neighbour (ties: lower label)
__global__ void join_kernel(int n, const int* rowptr, const int* col, const int* csr_pos, const int* tr_pos,
                            const double* vals, const double* dinv, const int* strong, const int* label, int* out) {
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i >= n) return;
    int l = label[i];
    if (l < 0) {
        float best = -1.f;
        const double di = dinv[i];
        for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) {
            const int j = strong[k];
            if (j == i || label[j] < 0) continue;
            const float w = coupling(csr_pos, tr_pos, vals, k, di, dinv[j]);
            if (w > best || (w == best && label[j] < l)) {
                best = w;
                l = label[j];
            }
        }
    }
    out[i] = l;
}

// keys (row, aggregate) of P's pattern: every entry of A; rows outside every aggregate give the
// key past the last row
__global__ void p_keys_kernel(int n, const int* rowptr, const int* col, const int* agg, long long nc, long long* keys) {
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i >= n) return;
    for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) {
        const int a = agg[col[k]];
        keys[k] = a >= 0 ? i * nc + a : agg[i] >= 0 ? i * nc + agg[i] : n * nc;
    }
}
// keys of a row product's pattern, one left entry per thread: the output row of entry k
// with every column of row idx[k] of the right matrix
__global__ void product_count_kernel(int64_t m, const int* idx, const int* b_rowptr, long long* count) {
    const int64_t k = blockIdx.x * (int64_t)BS + threadIdx.x;
    if (k < m) count[k] = b_rowptr[idx[k] + 1] - b_rowptr[idx[k]];
}
__global__ void product_keys_kernel(int64_t m, const int* orow, const int* idx, const int* b_rowptr, const int* b_col,
                                    const long long* off, long long nc, long long* keys) {
    const int64_t k = blockIdx.x * (int64_t)BS + threadIdx.x;
    if (k >= m) return;
    long long o = off[k];
    const long long r = orow[k] * nc;
    for (int e = b_rowptr[idx[k]]; e < b_rowptr[idx[k] + 1]; ++e) keys[o++] = r + b_col[e];
}
// CSR of the sorted distinct keys: columns, and each row's start by binary search
__global__ void key_cols_kernel(int64_t m, const long long* keys, long long nc, int* col) {
    const int64_t q = blockIdx.x * (int64_t)BS + threadIdx.x;
    if (q < m) col[q] = (int)(keys[q] % nc);
}
__global__ void key_rows_kernel(int nrows, int64_t m, const long long* keys, long long nc, int* rowptr) {
    const int r = blockIdx.x * BS + threadIdx.x;
    if (r > nrows) return;
    const long long want = r * nc;
    int64_t lo = 0, hi = m;
    while (lo < hi) {
        const int64_t mid = (lo + hi) / 2;
        if (keys[mid] < want) lo = mid + 1;
        else hi = mid;
    }
    rowptr[r] = (int)lo;
}
__global__ void iota_kernel(int64_t n, int* v) {
    const int64_t i = blockIdx.x * (int64_t)BS + threadIdx.x;
    if (i < n) v[i] = (int)i;
}
// transpose of a CSR pattern, its entries sorted by column (stable): rows, place of every entry
__global__ void transpose_kernel(int64_t m, const int* src, const int* erow, int* trow, int* place) {
    const int64_t q = blockIdx.x * (int64_t)BS + threadIdx.x;
    if (q >= m) return;
    const int e = src[q];
    trow[q] = erow[e];
    if (place) place[e] = (int)q;
}
__global__ void entry_rows_kernel(int n, const int* rowptr, int* erow) {
    const int r = blockIdx.x * BS + threadIdx.x;
    if (r >= n) return;
    for (int e = rowptr[r]; e < rowptr[r + 1]; ++e) erow[e] = r;
}
__global__ void sorted_starts_kernel(int nrows, int64_t m, const int* sorted, int* rowptr) {
    const int r = blockIdx.x * BS + threadIdx.x;
    if (r > nrows) return;
    int64_t lo = 0, hi = m;
    while (lo < hi) {
        const int64_t mid = (lo + hi) / 2;
        if (sorted[mid] < r) lo = mid + 1;
        else hi = mid;
    }
    rowptr[r] = (int)lo;
}

// Patterns of row products by row: the distinct columns of the right rows that the left row
// names, collected in shared memory, counted first and then written in increasing order (pass
// two: out_rowptr given). Against sorting one 64-bit key per product this needs no memory
// beyond the result: the keys of a 128^3 hex level 0 alone took 1.7 GB, whose mapping made
// first solves wait for up to a second. A row with more columns than its table holds sets
// *overflow and the sort takes over.
struct Union {
    int rows;
    const int *l_rowptr, *l_idx;
    const int *b_rowptr, *b_col;  // b_rowptr null: row j of B is the single column b_col[j] (none if negative)
    const int* out_rowptr;
    int *count, *out_col, *overflow;
};

template <int CAP>
__global__ void __launch_bounds__(BS) union_thread_kernel(const Union U) {
    __shared__ int cols[CAP][BS];
    const int r = blockIdx.x * BS + threadIdx.x, t = threadIdx.x;
    if (r >= U.rows) return;
    int len = 0;
    bool over = false;
    auto insert = [&](int c) {
        for (int k = 0; k < len; ++k)
            if (cols[k][t] == c) return;
        if (len == CAP) {
            over = true;
            return;
        }
        int k = len++;
        for (; k > 0 && cols[k - 1][t] > c; --k) cols[k][t] = cols[k - 1][t];
        cols[k][t] = c;
    };
    for (int q = U.l_rowptr[r]; q < U.l_rowptr[r + 1]; ++q) {
        const int j = U.l_idx[q];
        if (!U.b_rowptr) {
            if (U.b_col[j] >= 0) insert(U.b_col[j]);
        } else {
            for (int e = U.b_rowptr[j]; e < U.b_rowptr[j + 1]; ++e) insert(U.b_col[e]);
        }
    }
    if (over) *U.overflow = 1;
    if (!U.out_rowptr) {
        U.count[r] = len;
        return;
    }
    const int o = U.out_rowptr[r];
    for (int k = 0; k < len; ++k) U.out_col[o + k] = cols[k][t];
}

// T threads per row; groups of GL lanes take one left entry each; H slots (open addressing)
template <int T, int GL, int H>
__global__ void __launch_bounds__(BS) union_team_kernel(const Union U) {
    constexpr int TEAMS = BS / T, G = T / GL, FULL = H / 4 * 3;
    __shared__ int table[TEAMS][H], list[TEAMS][FULL + T], cnt[TEAMS];
    const int team = threadIdx.x / T, t = threadIdx.x % T, grp = t / GL, gl = t % GL;
    const int r = blockIdx.x * TEAMS + team;
    if (r >= U.rows) return;  // whole teams
    auto sync = [] {
        if constexpr (T == 32) __syncwarp();
        else __syncthreads();
    };
    for (int k = t; k < H; k += T) table[team][k] = -1;
    if (t == 0) cnt[team] = 0;
    sync();
    volatile int* count = &cnt[team];
    for (int q = U.l_rowptr[r] + grp; q < U.l_rowptr[r + 1]; q += G) {
        const int j = U.l_idx[q];
        for (int e = U.b_rowptr[j] + gl; e < U.b_rowptr[j + 1]; e += GL) {
            if (*count >= FULL) break;  // overflow: set below
            const int c = U.b_col[e];
            unsigned at = ((unsigned)c * 2654435761u) & (H - 1);
            for (int probe = 0; probe < H; ++probe, at = (at + 1) & (H - 1)) {
                const int old = atomicCAS(&table[team][at], -1, c);
                if (old == c) break;
                if (old == -1) {
                    atomicAdd(&cnt[team], 1);
                    break;
                }
            }
        }
    }
    sync();
    const int len = cnt[team];
    if (len >= FULL) {
        if (t == 0) *U.overflow = 1;
        if (t == 0 && !U.out_rowptr) U.count[r] = 0;
        return;
    }
    if (!U.out_rowptr) {
        if (t == 0) U.count[r] = len;
        return;
    }
    sync();
    if (t == 0) cnt[team] = 0;
    sync();
    for (int k = t; k < H; k += T)
        if (table[team][k] >= 0) list[team][atomicAdd(&cnt[team], 1)] = table[team][k];
    sync();
    const int o = U.out_rowptr[r];
    for (int a = t; a < len; a += T) {  // the place of a column: how many are smaller
        const int c = list[team][a];
        int rank = 0;
        for (int b = 0; b < len; ++b) rank += list[team][b] < c;
        U.out_col[o + rank] = c;
    }
}

// Transpose of a CSR pattern: rows spread over the columns by counting, then every column's
// rows put in increasing order
__global__ void column_count_kernel(int64_t m, const int* col, int* count) {
    const int64_t k = blockIdx.x * (int64_t)BS + threadIdx.x;
    if (k < m) atomicAdd(&count[col[k]], 1);
}
__global__ void column_fill_kernel(int n, const int* rowptr, const int* col, const int* t_rowptr, int* cursor, int* t_row) {
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i >= n) return;
    for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) t_row[t_rowptr[col[k]] + atomicAdd(&cursor[col[k]], 1)] = i;
}
// src: transposed entry -> entry; place: entry -> transposed entry
template <int T, int CAP>
__global__ void __launch_bounds__(BS) column_sort_kernel(int nc, const int* t_rowptr, int* t_row, const int* rowptr,
                                                         const int* col, int* src, int* place, int* overflow) {
    constexpr int TEAMS = BS / T;
    __shared__ int rows[TEAMS][CAP];
    const int team = threadIdx.x / T, t = threadIdx.x % T;
    const int c = blockIdx.x * TEAMS + team;
    if (c >= nc) return;
    auto sync = [] {
        if constexpr (T == 32) __syncwarp();
        else __syncthreads();
    };
    const int o = t_rowptr[c], len = t_rowptr[c + 1] - o;
    if (len > CAP) {
        if (t == 0) *overflow = 1;
        return;
    }
    for (int k = t; k < len; k += T) rows[team][k] = t_row[o + k];
    sync();
    for (int a = t; a < len; a += T) {
        const int i = rows[team][a];
        int rank = 0;
        for (int b = 0; b < len; ++b) rank += rows[team][b] < i;
        t_row[o + rank] = i;
        int e = rowptr[i], hi = rowptr[i + 1];  // the entry (i, c), columns sorted
        while (e < hi) {
            const int mid = (e + hi) >> 1;
            if (col[mid] < c) e = mid + 1;
            else hi = mid;
        }
        if (src) src[o + rank] = e;
        if (place) place[e] = o + rank;
    }
}

// ---------------------------------------------------------------- values
// position of column c in the sorted list col[lo, hi), or -1
__device__ __forceinline__ int findColumn(const int* __restrict__ col, int lo, int hi, int c) {
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const int v = __ldg(col + mid);
        if (v == c) return mid;
        if (v < c) lo = mid + 1;
        else hi = mid;
    }
    return -1;
}

// P[i, c] = [agg(i) = c] - omega_p dinv_i sum_{agg(j) = c} a_ij; LPR lanes per row, one
// entry per lane at a time
template <int LPR>
__global__ void __launch_bounds__(BS) p_values_kernel(
    int n, const int* __restrict__ rowptr, const int* __restrict__ col, const int* __restrict__ csr_pos,
    const double* __restrict__ vals, const double* __restrict__ dinv, const int* __restrict__ agg,
    const int* __restrict__ p_rowptr, const int* __restrict__ p_col, double omega_p, double* __restrict__ p_val) {
    const int64_t gt = blockIdx.x * (int64_t)BS + threadIdx.x;
    const int i = (int)(gt / LPR), sub = (int)(gt % LPR);
    if (i >= n) return;
    const double f = omega_p * dinv[i];
    const int own = agg[i];
    for (int p = p_rowptr[i] + sub; p < p_rowptr[i + 1]; p += LPR) {
        const int c = p_col[p];
        double sum = 0.0;
        for (int k = rowptr[i]; k < rowptr[i + 1]; ++k)
            if (agg[col[k]] == c) sum += valueAt(vals, csr_pos, k);
        p_val[p] = (own == c ? 1.0 : 0.0) - f * sum;
    }
}

// Row products of two sparse matrices on a known pattern: out[r, :] = sum_q w_q B[idx_q, :]
// over the entries q of row r of the left matrix. Both Galerkin products are of this form:
// A P (left A, right P) and P^T (A P) (left P^T, right A P).
struct Product {
    int rows;
    const int *out_rowptr, *out_col;
    const int *l_rowptr, *l_idx, *l_src;  // left entry -> row of B, and its value's place (null: the entry itself)
    const double* l_val;
    const int *b_rowptr, *b_col;
    const double* b_val;
    double* out;  // null: not kept
    // where B is P: Q = P - omega D^-1 A P, written to q_val and, transposed, to t_val (null: none)
    double omega;
    const double* dinv;
    const int* q_tpos;
    float *q_val, *t_val;
};
__device__ __forceinline__ void storeProduct(const Product& P, int r, int e, double v) {
    if (P.out) P.out[e] = v;
    if (P.q_val || P.t_val) {
        const int own = findColumn(P.b_col, P.b_rowptr[r], P.b_rowptr[r + 1], P.out_col[e]);
        const float q = (float)((own >= 0 ? P.b_val[own] : 0.0) - P.omega * P.dinv[r] * v);
        if (P.q_val) P.q_val[e] = q;
        if (P.t_val) P.t_val[P.q_tpos[e]] = q;
    }
}

// T threads per row (part of a warp, or the whole block) in groups of GL lanes: a group takes one left
// entry at a time, its lanes the entries of that row of B (distinct columns, so no two lanes
// of a group meet in one sum), into sums of its own; the groups' sums are added in order.
template <int T, int GL, int CH>
__global__ void __launch_bounds__(BS) product_team_kernel(const Product P) {
    constexpr int TEAMS = BS / T, G = T / GL;
    __shared__ double acc[TEAMS][G][CH];
    __shared__ int cols[TEAMS][CH];
    const int team = threadIdx.x / T, t = threadIdx.x % T, grp = t / GL, gl = t % GL;
    const unsigned mask = GL == 32 ? 0xffffffffu : ((1u << GL) - 1u) << (threadIdx.x & 31 & ~(GL - 1));
    const int r = blockIdx.x * TEAMS + team;
    if (r >= P.rows) return;  // whole teams
    auto sync = [&] {
        if constexpr (T <= 32) __syncwarp(T == 32 ? 0xffffffffu : ((1u << (T & 31)) - 1u) << (threadIdx.x & 31 & ~(T - 1)));
        else __syncthreads();
    };
    const int o1 = P.out_rowptr[r + 1], l0 = P.l_rowptr[r], l1 = P.l_rowptr[r + 1];
    for (int base = P.out_rowptr[r]; base < o1; base += CH) {
        const int len = min(CH, o1 - base);
        for (int k = t; k < len; k += T) cols[team][k] = P.out_col[base + k];
        for (int k = gl; k < len; k += GL) acc[team][grp][k] = 0.0;
        sync();
        for (int q = l0 + grp; q < l1; q += G) {
            const int j = P.l_idx[q];
            const double w = valueAt(P.l_val, P.l_src, q);
            for (int e = P.b_rowptr[j] + gl; e < P.b_rowptr[j + 1]; e += GL) {
                const int c = P.b_col[e];
                int lo = 0, hi = len;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (cols[team][mid] < c) lo = mid + 1;
                    else hi = mid;
                }
                if (lo < len && cols[team][lo] == c) acc[team][grp][lo] += w * P.b_val[e];
            }
            __syncwarp(mask);
        }
        sync();
        for (int k = t; k < len; k += T) {
            double v = 0.0;
            for (int g = 0; g < G; ++g) v += acc[team][g][k];
            storeProduct(P, r, base + k, v);
        }
        sync();
    }
}

// nnz_out, nnz_b: entries of the product and of B (n_b rows)
void launchProduct(const Product& P, int64_t nnz_out, int n_b, int64_t nnz_b, cudaStream_t s) {
    const double out = (double)nnz_out / std::max(P.rows, 1), right = (double)nnz_b / std::max(n_b, 1);
    // four lanes per row where rows are short and fill the chip (2.1M seven-point rows: 584 us;
    // one thread per row 1,078, eight lanes 699), a warp per row for longer ones (218,566 rows of
    // 37: 607 us, half a warp 610, a quarter 670), the whole block where rows are few
    if (P.rows > 8192 && out <= 12.0 && right <= 4.0) {
        product_team_kernel<4, 4, 16><<<ceil_div(P.rows, BS / 4), BS, 0, s>>>(P);
    } else if (P.rows > 16384) {
        const int g = ceil_div(P.rows, BS / 32);
        if (right <= 12.0) product_team_kernel<32, 8, 64><<<g, BS, 0, s>>>(P);
        else product_team_kernel<32, 32, 64><<<g, BS, 0, s>>>(P);
    } else if (right <= 12.0) {
        product_team_kernel<BS, 8, 96><<<P.rows, BS, 0, s>>>(P);
    } else {
        product_team_kernel<BS, 32, 256><<<P.rows, BS, 0, s>>>(P);
    }
    countLaunch();
}

// Inverse of a symmetric matrix of at most COARSE_MAX rows by Gauss-Jordan elimination
// without pivoting, one block: 32 x 32 threads hold 3 x 3 entries each in registers, and the
// next step's pivot row, column and reciprocal pass through shared memory, one barrier per
// step (the pivoting kernel of amg.cu takes seven over shared memory: 548 us at 148 rows;
// 5 x 5 entries per thread spill). A pivot below 1e-12 of the largest diagonal entry marks a
// singular direction (the constant vector of an all-Neumann Laplacian): its row and column
// are zeroed, which yields the solution of a consistent system with that unknown set to zero.
constexpr int INV_T = 3;
static_assert(32 * INV_T >= COARSE_MAX, "register tile too small");
__global__ void __launch_bounds__(1024) sym_inverse_kernel(int n, const int* __restrict__ rowptr,
                                                           const int* __restrict__ col,
                                                           const int* __restrict__ csr_pos,
                                                           const double* __restrict__ vals, double* __restrict__ M,
                                                           float* __restrict__ inv32) {
    __shared__ double row[2][COARSE_MAX], colv[2][COARSE_MAX], rec[2], amax;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int e = threadIdx.x; e < n * n; e += 1024) M[e] = 0.0;
    __syncthreads();
    for (int r = ty; r < n; r += 32)
        for (int k = rowptr[r] + tx; k < rowptr[r + 1]; k += 32) M[r * n + col[k]] = valueAt(vals, csr_pos, k);
    __syncthreads();
    if (ty == 0) {
        double m = 0.0;
        for (int i = tx; i < n; i += 32) m = fmax(m, fabs(M[i * n + i]));
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (tx == 0) amax = m;
    }
    __syncthreads();
    const double least = 1e-12 * amax;
    auto reciprocal = [&](double piv) { return fabs(piv) > least ? 1.0 / piv : 0.0; };  // 0: dropped
    double a[INV_T][INV_T];
#pragma unroll
    for (int u = 0; u < INV_T; ++u)
#pragma unroll
        for (int v = 0; v < INV_T; ++v) {
            const int i = ty + 32 * u, j = tx + 32 * v;
            a[u][v] = i < n && j < n ? M[i * n + j] : 0.0;
            if (i == 0 && j < n) row[0][j] = a[u][v];
            if (j == 0 && i < n) colv[0][i] = a[u][v];
        }
    if (threadIdx.x == 0) rec[0] = reciprocal(a[0][0]);
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        const int cur = k & 1, nxt = cur ^ 1;
        const double ip = rec[cur];
        double rk[INV_T], ck[INV_T];
#pragma unroll
        for (int v = 0; v < INV_T; ++v) {
            const int j = tx + 32 * v;
            rk[v] = j < n ? row[cur][j] * ip : 0.0;
        }
#pragma unroll
        for (int u = 0; u < INV_T; ++u) {
            const int i = ty + 32 * u;
            ck[u] = i < n ? colv[cur][i] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < INV_T; ++u)
#pragma unroll
            for (int v = 0; v < INV_T; ++v) {
                const int i = ty + 32 * u, j = tx + 32 * v;
                double x = a[u][v];
                if (i == k) x = j == k ? ip : rk[v];
                else if (j == k) x = -ck[u] * ip;
                else x -= ck[u] * rk[v];
                a[u][v] = x;
                if (i == k + 1 && j < n) row[nxt][j] = x;
                if (j == k + 1 && i < n) colv[nxt][i] = x;
                if (i == k + 1 && j == k + 1 && i < n) rec[nxt] = reciprocal(x);
            }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < INV_T; ++u)
#pragma unroll
        for (int v = 0; v < INV_T; ++v) {
            const int i = ty + 32 * u, j = tx + 32 * v;
            if (i < n && j < n) inv32[i * n + j] = (float)a[u][v];
        }
}

// A (omega D^-1) in FP32
__global__ void scaled_values_kernel(int64_t m, const int* __restrict__ col, const double* __restrict__ vals,
                                     const double* __restrict__ dinv, double omega, float* __restrict__ out) {
    for (int64_t k = blockIdx.x * (int64_t)BS + threadIdx.x; k < m; k += (int64_t)gridDim.x * BS)
        out[k] = (float)(vals[k] * (omega * dinv[col[k]]));
}

// ---------------------------------------------------------------- cycle kernels
// sum over CSR row [lo, hi) split over LPR adjacent lanes; valid in every lane of the group
template <int LPR, typename F>
__device__ __forceinline__ float csrSum(int lo, int hi, int sub, const int* __restrict__ col,
                                        const float* __restrict__ val, F x) {
    constexpr int W = LPR == 1 ? 8 : 4;  // entries in flight per lane
    float sum = 0.f;
    for (int k = lo + sub; k < hi; k += W * LPR) {
        int c[W];
        float v[W];
#pragma unroll
        for (int u = 0; u < W; ++u)
            if (k + u * LPR < hi) {
                c[u] = col[k + u * LPR];
                v[u] = val[k + u * LPR];
            }
#pragma unroll
        for (int u = 0; u < W; ++u)
            if (k + u * LPR < hi) sum += v[u] * x(c[u]);
    }
    if constexpr (LPR > 1)
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return sum;
}

// the SELL-32 row sum of the level-0 matrix, four slots in flight (eight: 58 against 53 us in
// the down-sweep of 2.1M five-point rows)
__device__ __forceinline__ float sellSum(const int* __restrict__ col, const float* __restrict__ val,
                                         const float* __restrict__ x, int base, int width) {
    float sum = 0.f;
    for (int j0 = 0; j0 < width; j0 += 4) {
        int c[4];
        float v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (j0 + k < width) {
                c[k] = col[base + 32 * (j0 + k)];
                v[k] = val[base + 32 * (j0 + k)];
            }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (j0 + k < width) sum += v[k] * __ldg(x + c[k]);
    }
    return sum;
}

// the matrix half of a down-sweep: y = omega D^-1 (2 b - (A omega D^-1) b)
struct SmoothArgs {
    int n;
    const int* rowptr;  // CSR (coarser levels) or the SELL slice offsets (level 0)
    const int* col;
    const float* val;
    const float* wd;
    const float* b;
    float* y;
};
// the transfer half: bc = Q^T b
struct RestrictArgs {
    int n;
    const int* rowptr;
    const int* col;
    const float* val;
    const float* b;
    float* bc;
};

template <int LT>
__device__ __forceinline__ void restrictRows(const RestrictArgs& R, int64_t gt) {
    const int row = (int)(gt / LT), sub = (int)(gt % LT);
    const bool valid = row < R.n;
    const int lo = valid ? R.rowptr[row] : 0, hi = valid ? R.rowptr[row + 1] : 0;
    const float sum = csrSum<LT>(lo, hi, sub, R.col, R.val, [&](int c) { return __ldg(R.b + c); });
    if (valid && sub == 0) R.bc[row] = sum;
}

// down-sweep of level 0: blocks below `rblocks` restrict, the others smooth
template <int LT>
__global__ void __launch_bounds__(BS) down0_kernel(const SmoothArgs A, const RestrictArgs R, int rblocks,
                                                   const KState* S) {
    pdlEnter();
    if (S && S->done) return;
    if ((int)blockIdx.x < rblocks) {
        restrictRows<LT>(R, (int64_t)blockIdx.x * BS + threadIdx.x);
        return;
    }
    const int row = (blockIdx.x - rblocks) * BS + threadIdx.x;
    if (row >= A.n) return;
    const int s0 = A.rowptr[row >> 5], width = (A.rowptr[(row >> 5) + 1] - s0) >> 5;
    const float sum = sellSum(A.col, A.val, A.b, s0 + (row & 31), width);
    A.y[row] = A.wd[row] * (2.f * A.b[row] - sum);
}

// down-sweep of a coarser level
template <int LA, int LT>
__global__ void __launch_bounds__(BS) down_kernel(const SmoothArgs A, const RestrictArgs R, int rblocks,
                                                  const KState* S) {
    pdlEnter();
    if (S && S->done) return;
    if ((int)blockIdx.x < rblocks) {
        restrictRows<LT>(R, (int64_t)blockIdx.x * BS + threadIdx.x);
        return;
    }
    const int64_t gt = (int64_t)(blockIdx.x - rblocks) * BS + threadIdx.x;
    const int row = (int)(gt / LA), sub = (int)(gt % LA);
    const bool valid = row < A.n;
    const int lo = valid ? A.rowptr[row] : 0, hi = valid ? A.rowptr[row + 1] : 0;
    const float sum = csrSum<LA>(lo, hi, sub, A.col, A.val, [&](int c) { return __ldg(A.b + c); });
    if (valid && sub == 0) A.y[row] = A.wd[row] * (2.f * A.b[row] - sum);
}

// up-sweep: x = y + Q e; LQ lanes per row
template <int LQ>
__global__ void __launch_bounds__(BS) up_kernel(int n, const int* __restrict__ rowptr, const int* __restrict__ col,
                                                const float* __restrict__ val, const float* __restrict__ e,
                                                const float* __restrict__ y, float* __restrict__ x, const KState* S) {
    pdlEnter();
    if (S && S->done) return;
    const int64_t gt = (int64_t)blockIdx.x * BS + threadIdx.x;
    const int row = (int)(gt / LQ), sub = (int)(gt % LQ);
    const bool valid = row < n;
    const int lo = valid ? rowptr[row] : 0, hi = valid ? rowptr[row + 1] : 0;
    const float sum = csrSum<LQ>(lo, hi, sub, col, val, [&](int c) { return __ldg(e + c); });
    if (valid && sub == 0) x[row] = y[row] + sum;
}

// coarsest level outside the tail: dense inverse, one warp per row
__global__ void coarse_kernel(int n, const float* __restrict__ inv, const float* __restrict__ b, float* __restrict__ x,
                              const KState* S) {
    pdlEnter();
    if (S && S->done) return;
    const int row = (blockIdx.x * BS + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= n) return;
    float sum = 0.f;
    for (int c = lane; c < n; c += 32) sum += inv[(size_t)row * n + c] * b[c];
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if (lane == 0) x[row] = sum;
}
// coarsest level too large for it (aggregation stagnated): damped Jacobi sweeps
__global__ void sweep_kernel(int n, const int* __restrict__ rowptr, const int* __restrict__ col,
                             const float* __restrict__ as, const float* __restrict__ wd, const float* __restrict__ b,
                             const float* __restrict__ x, float* __restrict__ out, int first, const KState* S) {
    pdlEnter();
    if (S && S->done) return;
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i >= n) return;
    // x holds u with the iterate omega D^-1 u (A is stored scaled): u += b - (A omega D^-1) u
    if (first) {
        out[i] = b[i];
        return;
    }
    float sum = 0.f;
    for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) sum += as[k] * x[col[k]];
    out[i] = x[i] + (b[i] - sum);
}
__global__ void sweep_end_kernel(int n, const float* __restrict__ wd, const float* __restrict__ u,
                                 float* __restrict__ x, const KState* S) {
    pdlEnter();
    if (S && S->done) return;
    const int i = blockIdx.x * BS + threadIdx.x;
    if (i < n) x[i] = wd[i] * u[i];
}

// ---- fused coarse tail: every level of at most TAIL_ROWS rows in one launch of one
// thread-block cluster, its phases separated by cluster barriers. Vectors written inside
// the launch are read through L2 (ld.global.cg).
constexpr int TAIL_BS = 1024;
constexpr int TAIL_ROWS = 4096;
constexpr int TAIL_NNZ = 98304;

struct TailLevel {
    int n;
    const int *rowptr, *col;
    const float *as, *wd;
    const int *t_rowptr, *t_col;
    const float* t_val;
    const int *q_rowptr, *q_col;
    const float* q_val;
    float *b, *x, *y;
};
struct TailParams {
    int nlev;
    const float* inv;
    const KState* S;
    TailLevel L[MAX_LEVELS];
};

// Row sums of a CSR matrix over the cluster's threads: as many lanes per row (8 to 32) as
// leave every row a group of its own; f(row, sum) runs in the first lane of each row.
template <int LPR, typename X, typename F>
__device__ __forceinline__ void tailRowsBy(int n, int g, int nthreads, const int* __restrict__ rowptr,
                                           const int* __restrict__ col, const float* __restrict__ val, X x, F f) {
    constexpr int RPW = 32 / LPR;
    const int lane = g & 31;
    for (int rb = (g >> 5) * RPW; rb < n; rb += (nthreads >> 5) * RPW) {  // uniform across a warp
        const int row = rb + lane / LPR;
        const bool valid = row < n;
        const int lo = valid ? rowptr[row] : 0, hi = valid ? rowptr[row + 1] : 0;
        const float sum = csrSum<LPR>(lo, hi, lane % LPR, col, val, x);
        if (valid && lane % LPR == 0) f(row, sum);
    }
}
template <typename X, typename F>
__device__ __forceinline__ void tailRows(int n, int g, int nthreads, const int* __restrict__ rowptr,
                                         const int* __restrict__ col, const float* __restrict__ val, X x, F f) {
    if (n * 32 <= nthreads) tailRowsBy<32>(n, g, nthreads, rowptr, col, val, x, f);
    else if (n * 16 <= nthreads) tailRowsBy<16>(n, g, nthreads, rowptr, col, val, x, f);
    else tailRowsBy<8>(n, g, nthreads, rowptr, col, val, x, f);
}

__global__ void __launch_bounds__(TAIL_BS) tail_kernel(const __grid_constant__ TailParams P) {
    pdlEnter();
    if (P.S && P.S->done) return;  // uniform: the state does not change during this launch
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int nthreads = (int)cl.num_blocks() * TAIL_BS;
    const int g = (int)cl.block_rank() * TAIL_BS + threadIdx.x;
    const int lane = threadIdx.x & 31;
    for (int l = 0; l + 1 < P.nlev; ++l) {
        const TailLevel& L = P.L[l];
        const TailLevel& N = P.L[l + 1];
        auto xb = [&](int c) { return __ldcg(L.b + c); };
        // both halves in one phase: the next level's right-hand side, then this level's y
        tailRows(N.n, g, nthreads, L.t_rowptr, L.t_col, L.t_val, xb, [&](int row, float sum) { N.b[row] = sum; });
        tailRows(L.n, g, nthreads, L.rowptr, L.col, L.as, xb,
                 [&](int row, float sum) { L.y[row] = L.wd[row] * (2.f * __ldcg(L.b + row) - sum); });
        cl.sync();
    }
    {
        const TailLevel& C = P.L[P.nlev - 1];
        const int nw = nthreads >> 5;
        for (int row = g >> 5; row < C.n; row += nw) {
            float sum = 0.f;
            for (int c = lane; c < C.n; c += 32) sum += P.inv[(size_t)row * C.n + c] * __ldcg(C.b + c);
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
            if (lane == 0) C.x[row] = sum;
        }
    }
    for (int l = P.nlev - 2; l >= 0; --l) {
        cl.sync();
        const TailLevel& L = P.L[l];
        const float* e = P.L[l + 1].x;
        tailRows(L.n, g, nthreads, L.q_rowptr, L.q_col, L.q_val, [&](int c) { return __ldcg(e + c); },
                 [&](int row, float sum) { L.x[row] = __ldcg(L.y + row) + sum; });
    }
}

// CTAs of the tail's cluster: 16 where the device can place it, else 8
int tailCluster() {
    static PerDevice c;
    return c.get([] { return clusterPlaced(tail_kernel, TAIL_BS) ? CLUSTER_MAX : 8; });
}

// ---------------------------------------------------------------- host side of the structure
int readInt(const int* d, cudaStream_t s) {
    int v = 0;
    PB_CUDA(cudaMemcpyAsync(&v, d, sizeof(int), cudaMemcpyDeviceToHost, s));
    PB_CUDA(cudaStreamSynchronize(s));
    return v;
}

// CSR pattern (sorted columns) of the distinct keys row * ncols + col among keys[0, m); keys is overwritten
int64_t patternOf(DevArena& ar, long long* keys, int64_t m, int nrows, long long ncols, ArenaBuf<int>& rowptr,
                  ArenaBuf<int>& col, cudaStream_t s) {
    if (m >= (int64_t(1) << 31)) fail(PRISM_BAD_ARG, "multigrid structure too large for 32-bit indices");
    TmpBuf<long long> sorted(std::max<int64_t>(m, 1), s);
    TmpBuf<int> count(1, s);
    int end_bit = 1;
    while (end_bit < 63 && ((long long)1 << end_bit) <= (long long)nrows * ncols) ++end_bit;
    size_t t0 = 0, t1 = 0;
    PB_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, t0, keys, sorted.p, m, 0, end_bit, s));
    PB_CUDA(cub::DeviceSelect::Unique(nullptr, t1, sorted.p, keys, count.p, m, s));
    TmpBuf<unsigned char> tmp(std::max<size_t>(std::max(t0, t1), 1), s);
    PB_CUDA(cub::DeviceRadixSort::SortKeys(tmp.p, t0, keys, sorted.p, m, 0, end_bit, s));
    PB_CUDA(cub::DeviceSelect::Unique(tmp.p, t1, sorted.p, keys, count.p, m, s));
    int64_t nnz = readInt(count.p, s);
    if (nnz > 0) {  // a key past the last row is no entry
        long long last = 0;
        PB_CUDA(cudaMemcpyAsync(&last, keys + nnz - 1, sizeof(long long), cudaMemcpyDeviceToHost, s));
        PB_CUDA(cudaStreamSynchronize(s));
        if (last == (long long)nrows * ncols) --nnz;
    }
    rowptr.alloc(ar, (size_t)nrows + 1, s);
    col.alloc(ar, std::max<int64_t>(nnz, 1), s);
    key_cols_kernel<<<grid(nnz), BS, 0, s>>>(nnz, keys, ncols, col.p); countLaunch();
    key_rows_kernel<<<grid(nrows + 1), BS, 0, s>>>(nrows, nnz, keys, ncols, rowptr.p); countLaunch();
    return nnz;
}

// exclusive offsets of count[0, n) into rowptr[0, n]; returns the total
int64_t rowOffsets(TmpBuf<int>& count, int n, int* rowptr, cudaStream_t s) {
    PB_CUDA(cudaMemsetAsync(count.p + n, 0, sizeof(int), s));
    size_t tb = 0;
    PB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, count.p, rowptr, n + 1, s));
    TmpBuf<unsigned char> tmp(std::max<size_t>(tb, 1), s);
    PB_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tb, count.p, rowptr, n + 1, s));
    return readInt(rowptr + n, s);
}

// U's pattern (U.rows rows; the average numbers of left and right entries choose the kernel);
// false if a row did not fit
bool unionPattern(DevArena& ar, Union U, double left, double right, ArenaBuf<int>& rowptr, ArenaBuf<int>& col,
                  int64_t& nnz, cudaStream_t s) {
    TmpBuf<int> count((size_t)U.rows + 1, s), overflow(1, s);
    PB_CUDA(cudaMemsetAsync(overflow.p, 0, sizeof(int), s));
    U.count = count.p;
    U.overflow = overflow.p;
    auto run = [&] {
        if (!U.b_rowptr || left * right <= 64.0) {
            union_thread_kernel<32><<<grid(U.rows), BS, 0, s>>>(U);
        } else if (U.rows > 16384) {
            if (right <= 12.0) union_team_kernel<32, 8, 256><<<ceil_div(U.rows, BS / 32), BS, 0, s>>>(U);
            else union_team_kernel<32, 32, 256><<<ceil_div(U.rows, BS / 32), BS, 0, s>>>(U);
        } else {
            if (right <= 12.0) union_team_kernel<BS, 8, 4096><<<U.rows, BS, 0, s>>>(U);
            else union_team_kernel<BS, 32, 4096><<<U.rows, BS, 0, s>>>(U);
        }
        countLaunch();
    };
    run();
    rowptr.alloc(ar, (size_t)U.rows + 1, s);
    nnz = rowOffsets(count, U.rows, rowptr.p, s);
    if (readInt(overflow.p, s)) return false;
    col.alloc(ar, std::max<int64_t>(nnz, 1), s);
    U.out_rowptr = rowptr.p;
    U.out_col = col.p;
    run();
    PB_LAUNCH("smoothed aggregation: pattern");
    return true;
}

// Pattern of the row product of m left entries (output row orow[k], right row idx[k]) with B;
// entries: of the matrices that it is made from
int64_t productPattern(DevArena& ar, int64_t entries, int64_t m, const int* orow, const int* idx, const int* b_rowptr, const int* b_col,
                       int nrows, long long ncols, ArenaBuf<int>& rowptr, ArenaBuf<int>& col, cudaStream_t s) {
    TmpBuf<long long> count(m + 1, s), off(m + 1, s);
    product_count_kernel<<<grid(m), BS, 0, s>>>(m, idx, b_rowptr, count.p); countLaunch();
    PB_CUDA(cudaMemsetAsync(count.p + m, 0, sizeof(long long), s));
    size_t tb = 0;
    PB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, count.p, off.p, m + 1, s));
    TmpBuf<unsigned char> tmp(std::max<size_t>(tb, 1), s);
    PB_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tb, count.p, off.p, m + 1, s));
    long long total = 0;
    PB_CUDA(cudaMemcpyAsync(&total, off.p + m, sizeof(long long), cudaMemcpyDeviceToHost, s));
    PB_CUDA(cudaStreamSynchronize(s));
    if (total > MAX_PRODUCTS * entries) fail(PRISM_BAD_ARG, "multigrid structure too dense for smoothed aggregation");
    TmpBuf<long long> keys(std::max<long long>(total, 1), s);
    product_keys_kernel<<<grid(m), BS, 0, s>>>(m, orow, idx, b_rowptr, b_col, off.p, ncols, keys.p); countLaunch();
    return patternOf(ar, keys.p, total, nrows, ncols, rowptr, col, s);
}

// the transpose by sorting the entries (columns of more rows than columnTranspose holds)
void sortedTranspose(DevArena& ar, int n, int nc, int64_t nnz, const int* rowptr, const int* col, ArenaBuf<int>& t_rowptr,
                 ArenaBuf<int>& t_row, ArenaBuf<int>* src, ArenaBuf<int>* place, cudaStream_t s) {
    const size_t m = std::max<int64_t>(nnz, 1);
    TmpBuf<int> erow(m, s), ids(m, s), col_s(m, s), src_t(src ? 0 : m, s);
    if (src) src->alloc(ar, m, s);
    int* order = src ? src->p : src_t.p;
    entry_rows_kernel<<<grid(n), BS, 0, s>>>(n, rowptr, erow.p); countLaunch();
    iota_kernel<<<grid(nnz), BS, 0, s>>>(nnz, ids.p); countLaunch();
    int end_bit = 1;
    while (end_bit < 31 && (1 << end_bit) < nc) ++end_bit;
    size_t tb = 0;
    PB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, col, col_s.p, ids.p, order, nnz, 0, end_bit, s));
    TmpBuf<unsigned char> tmp(std::max<size_t>(tb, 1), s);
    PB_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, col, col_s.p, ids.p, order, nnz, 0, end_bit, s));
    t_rowptr.alloc(ar, (size_t)nc + 1, s);
    t_row.alloc(ar, m, s);
    if (place) place->alloc(ar, m, s);
    sorted_starts_kernel<<<grid(nc + 1), BS, 0, s>>>(nc, nnz, col_s.p, t_rowptr.p); countLaunch();
    transpose_kernel<<<grid(nnz), BS, 0, s>>>(nnz, order, erow.p, t_row.p, place ? place->p : nullptr); countLaunch();
}

// Transpose of the pattern (n rows, nc columns): row starts, the row of every entry, and
// src (entry of the transpose -> entry) or place (entry -> entry of the transpose)
void transposeOf(DevArena& ar, int n, int nc, int64_t nnz, const int* rowptr, const int* col, ArenaBuf<int>& t_rowptr,
                 ArenaBuf<int>& t_row, ArenaBuf<int>* src, ArenaBuf<int>* place, cudaStream_t s) {
    const DevArena::Mark before = ar.mark();
    const size_t m = std::max<int64_t>(nnz, 1);
    t_rowptr.alloc(ar, (size_t)nc + 1, s);
    t_row.alloc(ar, m, s);
    if (src) src->alloc(ar, m, s);
    if (place) place->alloc(ar, m, s);
    TmpBuf<int> count((size_t)nc + 1, s), overflow(1, s);
    PB_CUDA(cudaMemsetAsync(overflow.p, 0, sizeof(int), s));
    PB_CUDA(cudaMemsetAsync(count.p, 0, nc * sizeof(int), s));
    column_count_kernel<<<grid(nnz), BS, 0, s>>>(nnz, col, count.p); countLaunch();
    rowOffsets(count, nc, t_rowptr.p, s);
    PB_CUDA(cudaMemsetAsync(count.p, 0, nc * sizeof(int), s));
    column_fill_kernel<<<grid(n), BS, 0, s>>>(n, rowptr, col, t_rowptr.p, count.p, t_row.p); countLaunch();
    int* sp = src ? src->p : nullptr;
    int* pp = place ? place->p : nullptr;
    if (nc > 16384)
        column_sort_kernel<32, 512><<<ceil_div(nc, BS / 32), BS, 0, s>>>(nc, t_rowptr.p, t_row.p, rowptr, col, sp, pp, overflow.p);
    else
        column_sort_kernel<BS, 8192><<<nc, BS, 0, s>>>(nc, t_rowptr.p, t_row.p, rowptr, col, sp, pp, overflow.p);
    countLaunch();
    PB_LAUNCH("smoothed aggregation: transpose");
    if (readInt(overflow.p, s)) {
        ar.rewind(before);
        sortedTranspose(ar, n, nc, nnz, rowptr, col, t_rowptr, t_row, src, place, s);
    }
}

// aggregates of level L into L.agg; returns their number
int aggregate(DevArena& ar, SaLevel& L, cudaStream_t s) {
    const int n = L.n;
    TmpBuf<float> wmax(n, s);
    TmpBuf<int> strong(std::max<int64_t>(L.nnz, 1), s), left(MIS_ROUNDS + 1, s), root(n + 1, s), id(n + 1, s), lab(n, s);
    TmpBuf<unsigned long long> key(n, s), near(n, s);
    strongest_kernel<<<grid(n), BS, 0, s>>>(n, L.rowptr, L.col, L.csr_pos, L.tr_pos.p, L.vals, L.dinv.p, wmax.p); countLaunch();
    strong_kernel<<<grid(n), BS, 0, s>>>(n, L.rowptr, L.col, L.csr_pos, L.tr_pos.p, L.vals, L.dinv.p, wmax.p, strong.p); countLaunch();
    PB_CUDA(cudaMemsetAsync(left.p, 0, (MIS_ROUNDS + 1) * sizeof(int), s));
    mis_init_kernel<<<grid(n), BS, 0, s>>>(n, key.p, left.p); countLaunch();
    for (int r = 0; r < MIS_ROUNDS; ++r) {
        mis_near_kernel<<<grid(n), BS, 0, s>>>(n, L.rowptr, strong.p, key.p, near.p, left.p + r); countLaunch();
        mis_decide_kernel<<<grid(n), BS, 0, s>>>(n, L.rowptr, strong.p, key.p, near.p, left.p + r, left.p + r + 1); countLaunch();
        if (r % MIS_BATCH == MIS_BATCH - 1 && readInt(left.p + r + 1, s) == 0) break;
    }
    PB_CUDA(cudaMemsetAsync(root.p + n, 0, sizeof(int), s));
    mis_root_kernel<<<grid(n), BS, 0, s>>>(n, key.p, wmax.p, root.p); countLaunch();
    size_t tb = 0;
    PB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, root.p, id.p, n + 1, s));
    TmpBuf<unsigned char> tmp(std::max<size_t>(tb, 1), s);
    PB_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tb, root.p, id.p, n + 1, s));
    const int nc = readInt(id.p + n, s);
    L.agg.alloc(ar, n, s);
    // the rows next to a root, then the rows next to those
    root_label_kernel<<<grid(n), BS, 0, s>>>(n, root.p, id.p, L.agg.p); countLaunch();
    join_kernel<<<grid(n), BS, 0, s>>>(n, L.rowptr, L.col, L.csr_pos, L.tr_pos.p, L.vals, L.dinv.p, strong.p, L.agg.p, lab.p); countLaunch();
    join_kernel<<<grid(n), BS, 0, s>>>(n, L.rowptr, L.col, L.csr_pos, L.tr_pos.p, L.vals, L.dinv.p, strong.p, lab.p, L.agg.p); countLaunch();
    PB_LAUNCH("smoothed aggregation: aggregates");
    return nc;
}

// lanes per CSR row: about four entries per lane, more where the rows alone leave most of
// the chip idle
int lanesFor(int n, int64_t nnz) {
    const double mean = n > 0 ? (double)nnz / n : 1.0;
    int l = 2;
    while (l < 32 && l * 4 < mean) l *= 2;
    while (l < 32 && l < mean && (int64_t)n * l < (int64_t)NUM_SMS * 1024) l *= 2;
    return l;
}

template <typename F>
void withLanes(int l, F&& f) {
    switch (l) {
        case 2: f(std::integral_constant<int, 2>{}); break;
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 16: f(std::integral_constant<int, 16>{}); break;
        default: f(std::integral_constant<int, 32>{}); break;
    }
}

}  // namespace

// D^-1 and the FP32 copy of A from the current values of level L
void SaAmg::levelScaling(SaLevel& L, cudaStream_t s) {
    scaling_kernel<<<grid(L.n), BS, 0, s>>>(L.n, L.rowptr, L.col, L.csr_pos, L.vals, L.omega, L.csr_pos || L.tr_pos.p ? 0.0 : SPECTRUM,
                                            L.dinv.p, L.wd.p); countLaunch();
    const int64_t m = L.csr_pos ? L.sell_nnz : L.nnz;
    const int* col = L.csr_pos ? L.sl_col : L.col;
    scaled_values_kernel<<<(int)std::min<int64_t>(grid(m), NUM_SMS * 32), BS, 0, s>>>(m, col, L.vals, L.dinv.p, L.omega,
                                                                                     L.as32.p); countLaunch();
}

// P, A P, Q, Q^T of level l and the values of level l + 1, from level l's current values
void SaAmg::levelValues(size_t l, cudaStream_t s) {
    SaLevel& L = *levels[l];
    SaLevel& C = *levels[l + 1];
    const bool sym = !L.tr_pos.p;
    auto prolongation = [&](const int* pos, double* val) {
        withLanes(L.lpr_p, [&](auto c) {
            constexpr int LP = decltype(c)::value;
            p_values_kernel<LP><<<grid((int64_t)L.n * LP), BS, 0, s>>>(L.n, L.rowptr, L.col, pos, L.vals, L.dinv.p,
                                                                       L.agg.p, L.p_rowptr.p, L.p_col.p, L.omega_p, val); countLaunch();
        });
    };
    prolongation(L.csr_pos, L.p_val.p);
    Product AP{};
    AP.rows = L.n;
    AP.out_rowptr = L.q_rowptr.p;
    AP.out_col = L.q_col.p;
    AP.l_rowptr = L.rowptr;
    AP.l_idx = L.col;
    AP.l_src = L.csr_pos;
    AP.l_val = L.vals;
    AP.b_rowptr = L.p_rowptr.p;
    AP.b_col = L.p_col.p;
    AP.b_val = L.p_val.p;
    AP.out = L.ap_val.p;
    AP.omega = L.omega;
    AP.dinv = L.dinv.p;
    AP.q_tpos = L.q_tpos.p;
    AP.q_val = L.q_val.p;
    AP.t_val = sym ? L.t_val.p : nullptr;
    launchProduct(AP, L.q_nnz, L.n, L.p_nnz, s);
    if (!sym) {
        // the restriction from A^T in A's place: R^T, and (S R^T) stored transposed
        prolongation(L.tr_pos.p, L.r_val.p);
        AP.l_src = L.tr_pos.p;
        AP.b_val = L.r_val.p;
        AP.out = nullptr;
        AP.q_val = nullptr;
        AP.t_val = L.t_val.p;
        launchProduct(AP, L.q_nnz, L.n, L.p_nnz, s);
    }
    Product AC{};
    AC.rows = C.n;
    AC.out_rowptr = C.rowptr;
    AC.out_col = C.col;
    AC.l_rowptr = L.pt_rowptr.p;
    AC.l_idx = L.pt_row.p;
    AC.l_src = L.pt_src.p;
    AC.l_val = sym ? L.p_val.p : L.r_val.p;
    AC.b_rowptr = L.q_rowptr.p;
    AC.b_col = L.q_col.p;
    AC.b_val = L.ap_val.p;
    AC.out = C.o_vals.p;
    launchProduct(AC, C.nnz, L.n, L.q_nnz, s);
}

void SaAmg::build(const SellMatrix& A, const int* rowptr, const int* col, bool sym, cudaStream_t s) {
    symmetric = sym;
    levels.clear();
    arena.reset();  // stream order keeps earlier work on the old hierarchy ahead of its reuse
    coarse_a.release();
    coarse_inv32.release();
    const auto t0 = std::chrono::steady_clock::now();
    auto L0 = std::make_unique<SaLevel>();
    L0->n = A.n;
    L0->nnz = A.nnz_csr;
    L0->rowptr = rowptr;
    L0->col = col;
    L0->o_csr_pos.alloc(arena, std::max<int64_t>(A.nnz_csr, 1), s);
    csr_pos_kernel<<<grid(A.n), BS, 0, s>>>(A.n, rowptr, A.sl_off, L0->o_csr_pos.p); countLaunch();
    L0->csr_pos = L0->o_csr_pos.p;
    L0->vals = A.vals;
    L0->nslices = A.nslices;
    L0->sell_nnz = A.nnz_padded;
    L0->sl_off = A.sl_off;
    L0->sl_col = A.col;
    L0->diag_pos = A.diag_pos;
    levels.push_back(std::move(L0));
    double filled = 0.0;
    while (true) {
        const size_t l = levels.size() - 1;
        SaLevel& L = *levels[l];
        // Smoother weights. Symmetric: the spectrum of D^-1 A reaches 2 on the finest level and
        // 1.2-1.5 on the Galerkin levels (measured on 2-D, 3-D and tetrahedral diffusion);
        // omega_p is 4/3 over it, omega the largest that leaves the stiffest modes damped. With
        // convection the spectrum is complex and the larger weights diverge: a CPU model of the
        // cycle took 22 BiCGSTAB iterations on 48^3 MUSCL transport with (0.8, 0.66) on every
        // level against 64 with piecewise-constant aggregation, 26 / 54 at a cell Peclet number
        // of 3,000, 30 / 68 on tetrahedra, and failed with (0.9, 0.95).
        L.omega = !sym ? 0.8 : l == 0 ? 0.9 : 1.1;
        L.omega_p = !sym ? 0.66 : l == 0 ? 0.7 : 0.95;
        if (!sym) {
            L.tr_pos.alloc(arena, std::max<int64_t>(L.nnz, 1), s);
            transposed_kernel<<<grid(L.n), BS, 0, s>>>(L.n, L.rowptr, L.col, L.csr_pos, L.tr_pos.p); countLaunch();
        }
        L.dinv.alloc(arena, L.n, s);
        L.wd.alloc(arena, L.n, s);
        L.as32.alloc(arena, std::max<int64_t>(std::max(L.nnz, L.sell_nnz), 1), s);
        L.y.alloc(arena, L.n, s);
        if (l > 0) {  // level 0 works on the caller's vectors
            L.b.alloc(arena, L.n, s);
            L.x.alloc(arena, L.n, s);
        }
        L.lpr_a = lanesFor(L.n, L.nnz);
        levelScaling(L, s);
        if (L.n <= COARSE_MAX || levels.size() >= (size_t)MAX_LEVELS) break;
        const int nc = aggregate(arena, L, s);
        if (nc == 0 || nc > (int)(0.8 * L.n)) break;
        // P: the aggregates of a row's neighbours
        Union U{};
        U.rows = L.n;
        U.l_rowptr = L.rowptr;
        U.l_idx = L.col;
        U.b_col = L.agg.p;
        const double left = (double)L.nnz / L.n;
        DevArena::Mark before = arena.mark();
        if (!unionPattern(arena, U, left, 1.0, L.p_rowptr, L.p_col, L.p_nnz, s)) {
            arena.rewind(before);
            TmpBuf<long long> keys(std::max<int64_t>(L.nnz, 1), s);
            p_keys_kernel<<<grid(L.n), BS, 0, s>>>(L.n, L.rowptr, L.col, L.agg.p, nc, keys.p); countLaunch();
            L.p_nnz = patternOf(arena, keys.p, L.nnz, L.n, nc, L.p_rowptr, L.p_col, s);
        }
        L.p_val.alloc(arena, std::max<int64_t>(L.p_nnz, 1), s);
        if (!sym) L.r_val.alloc(arena, std::max<int64_t>(L.p_nnz, 1), s);
        transposeOf(arena, L.n, nc, L.p_nnz, L.p_rowptr.p, L.p_col.p, L.pt_rowptr, L.pt_row, &L.pt_src, nullptr, s);
        // A P, the pattern of Q
        U.b_rowptr = L.p_rowptr.p;
        U.b_col = L.p_col.p;
        before = arena.mark();
        if (!unionPattern(arena, U, left, (double)L.p_nnz / L.n, L.q_rowptr, L.q_col, L.q_nnz, s)) {
            arena.rewind(before);
            TmpBuf<int> erow(std::max<int64_t>(L.nnz, 1), s);
            entry_rows_kernel<<<grid(L.n), BS, 0, s>>>(L.n, L.rowptr, erow.p); countLaunch();
            L.q_nnz = productPattern(arena, L.nnz, L.nnz, erow.p, L.col, L.p_rowptr.p, L.p_col.p, L.n, nc, L.q_rowptr, L.q_col, s);
        }
        L.ap_val.alloc(arena, std::max<int64_t>(L.q_nnz, 1), s);
        L.q_val.alloc(arena, std::max<int64_t>(L.q_nnz, 1), s);
        L.t_val.alloc(arena, std::max<int64_t>(L.q_nnz, 1), s);
        transposeOf(arena, L.n, nc, L.q_nnz, L.q_rowptr.p, L.q_col.p, L.t_rowptr, L.t_col, nullptr, &L.q_tpos, s);
        L.lpr_p = lanesFor(L.n, L.p_nnz);
        L.lpr_q = lanesFor(L.n, L.q_nnz);
        L.lpr_t = lanesFor(nc, L.q_nnz);
        // P^T A P
        auto C = std::make_unique<SaLevel>();
        U.rows = nc;
        U.l_rowptr = L.pt_rowptr.p;
        U.l_idx = L.pt_row.p;
        U.b_rowptr = L.q_rowptr.p;
        U.b_col = L.q_col.p;
        before = arena.mark();
        if (!unionPattern(arena, U, (double)L.p_nnz / nc, (double)L.q_nnz / L.n, C->o_rowptr, C->o_col, C->nnz, s)) {
            arena.rewind(before);
            TmpBuf<int> erow(std::max<int64_t>(L.p_nnz, 1), s);
            entry_rows_kernel<<<grid(L.n), BS, 0, s>>>(L.n, L.p_rowptr.p, erow.p); countLaunch();
            C->nnz = productPattern(arena, L.p_nnz + L.q_nnz, L.p_nnz, L.p_col.p, erow.p, L.q_rowptr.p, L.q_col.p, nc, nc,
                                    C->o_rowptr, C->o_col, s);
        }
        C->n = nc;
        C->rowptr = C->o_rowptr.p;
        C->col = C->o_col.p;
        C->o_vals.alloc(arena, std::max<int64_t>(C->nnz, 1), s);
        C->vals = C->o_vals.p;
        C->lpr_a = lanesFor(nc, C->nnz);
        levels.push_back(std::move(C));
        filled += (double)levels.back()->nnz * levels.back()->nnz / nc;
        if (filled > max_fill * A.nnz_csr * A.nnz_csr / A.n) fail(PRISM_BAD_ARG, "multigrid levels too dense for smoothed aggregation");
        levelValues(l, s);
        PB_LAUNCH("smoothed aggregation: level");
    }
    coarse_n = levels.back()->n;
    if (coarse_n <= COARSE_MAX) {
        const size_t nn = (size_t)coarse_n * coarse_n;
        coarse_a.alloc(arena, nn, s);
        coarse_inv32.alloc(arena, nn, s);
    }
    // the fused tail needs a dense coarsest level
    tail = -1;
    for (size_t l = 1; l < levels.size() && coarse_inv32.p; ++l)
        if (levels[l]->n <= TAIL_ROWS && levels[l]->nnz <= TAIL_NNZ) {
            tail = (int)l;
            break;
        }
    built = true;
    static std::atomic<uint64_t> next{0};  // process-wide: no two hierarchies share a value
    generation = ++next;
    if (verbose()) {
        PB_CUDA(cudaStreamSynchronize(s));
        std::fprintf(stderr, "[prism samg] hierarchy:");
        for (auto& L : levels) std::fprintf(stderr, " %d/%lld", L->n, (long long)L->nnz);
        std::fprintf(stderr, " (rows/entries), P/Q:");
        for (auto& L : levels)
            if (L->q_nnz) std::fprintf(stderr, " %lld/%lld", (long long)L->p_nnz, (long long)L->q_nnz);
        std::fprintf(stderr, ", fused tail from level %d, %.1f MB, built in %.2f ms\n", tail, arena.used() / 1e6,
                     std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count());
    }
}

void SaAmg::setup(const SellMatrix& A, const int* rowptr, const int* col, bool sym, bool keep_values, cudaStream_t s) {
    const bool same = built && symmetric == sym && !levels.empty() && levels[0]->n == A.n && levels[0]->sl_off == A.sl_off;
    if (same && keep_values && levels[0]->vals == A.vals) return;
    fresh = !same;
    if (!same) {
        build(A, rowptr, col, sym, s);
    } else {
        levels[0]->vals = A.vals;
        levelScaling(*levels[0], s);
        for (size_t l = 0; l + 1 < levels.size(); ++l) {
            levelValues(l, s);
            levelScaling(*levels[l + 1], s);
        }
    }
    if (coarse_inv32.p) {
        const SaLevel& C = *levels.back();
        sym_inverse_kernel<<<1, 1024, 0, s>>>(coarse_n, C.rowptr, C.col, C.csr_pos, C.vals, coarse_a.p, coarse_inv32.p); countLaunch();
    }
    PB_LAUNCH("smoothed aggregation: setup");
}

void SaAmg::apply(const float* r, float* z, const KState* S, cudaStream_t s, bool sample) {
    const size_t last = levels.size() - 1;
    const size_t stop = tail > 0 ? (size_t)tail : last;  // levels below `stop` run their own launches
    auto rhs = [&](size_t l) { return l == 0 ? r : (const float*)levels[l]->b.p; };
    auto sol = [&](size_t l) { return l == 0 ? z : levels[l]->x.p; };
    for (size_t l = 0; l < stop; ++l) {
        SaLevel& L = *levels[l];
        SaLevel& N = *levels[l + 1];
        const SmoothArgs A{L.n, l == 0 ? L.sl_off : L.rowptr, l == 0 ? L.sl_col : L.col, L.as32.p, L.wd.p, rhs(l), L.y.p};
        const RestrictArgs R{N.n, L.t_rowptr.p, L.t_col.p, L.t_val.p, rhs(l), N.b.p};
        // algorithmic bytes: the entries of A and Q^T, their row offsets, b, D^-1, y and the restricted b
        const int slot = sample && l == 0 ? profBegin(PROF_AMG_DOWN, true,
                                                      8.0 * (L.nnz + L.q_nnz) + 4.0 * (L.n + N.n + 2) + 12.0 * L.n +
                                                          4.0 * N.n, s)
                                          : -1;
        withLanes(L.lpr_t, [&](auto ct) {
            constexpr int LT = decltype(ct)::value;
            const int rb = grid((int64_t)N.n * LT);
            if (l == 0) {
                launchPdl(down0_kernel<LT>, rb + grid(L.n), BS, s, A, R, rb, S);
            } else {
                withLanes(L.lpr_a, [&](auto ca) {
                    constexpr int LA = decltype(ca)::value;
                    launchPdl(down_kernel<LA, LT>, rb + grid((int64_t)L.n * LA), BS, s, A, R, rb, S);
                });
            }
        });
        profEnd(slot, s);
    }
    if (tail > 0) {
        TailParams P{};
        P.nlev = (int)(levels.size() - tail);
        P.inv = coarse_inv32.p;
        P.S = S;
        for (int k = 0; k < P.nlev; ++k) {
            SaLevel& L = *levels[tail + k];
            P.L[k] = TailLevel{L.n, L.rowptr, L.col, L.as32.p, L.wd.p, L.t_rowptr.p, L.t_col.p, L.t_val.p,
                               L.q_rowptr.p, L.q_col.p, L.q_val.p, L.b.p, L.x.p, L.y.p};
        }
        launchCluster(tail_kernel, tailCluster(), TAIL_BS, s, true, P);
    } else if (coarse_inv32.p) {
        launchPdl(coarse_kernel, grid((int64_t)coarse_n * 32), BS, s, coarse_n, (const float*)coarse_inv32.p, rhs(last),
                  sol(last), S);
    } else if (last == 0) {
        // nothing to aggregate (no strong couplings): the two smoothing steps alone
        SaLevel& L = *levels[0];
        const SmoothArgs A{L.n, L.sl_off, L.sl_col, L.as32.p, L.wd.p, r, z};
        launchPdl(down0_kernel<2>, grid(L.n), BS, s, A, RestrictArgs{}, 0, S);
    } else {
        SaLevel& C = *levels[last];
        const int* rp = C.rowptr;
        const int* cl = C.col;
        const float* as = C.as32.p;
        float* cur = C.y.p;
        float* nxt = C.x.p;
        launchPdl(sweep_kernel, grid(C.n), BS, s, C.n, rp, cl, as, (const float*)C.wd.p, rhs(last), (const float*)nxt,
                  cur, 1, S);
        for (int k = 0; k < 8; ++k) {
            launchPdl(sweep_kernel, grid(C.n), BS, s, C.n, rp, cl, as, (const float*)C.wd.p, rhs(last),
                      (const float*)cur, nxt, 0, S);
            std::swap(cur, nxt);
        }
        launchPdl(sweep_end_kernel, grid(C.n), BS, s, C.n, (const float*)C.wd.p, (const float*)cur, sol(last), S);
    }
    for (size_t l = stop; l-- > 0;) {
        SaLevel& L = *levels[l];
        const float* e = levels[l + 1]->x.p;
        const int slot = sample && l == 0
                             ? profBegin(PROF_AMG_POST, true, 8.0 * L.q_nnz + 4.0 * (L.n + 1) + 8.0 * L.n +
                                                                  4.0 * levels[l + 1]->n, s)
                             : -1;
        // one thread per row where rows are short and fill the chip (2.1M rows of 4.3 entries: 26
        // us, with two lanes 35, with four 61)
        if ((double)L.q_nnz <= 16.0 * L.n && L.n > 32 * NUM_SMS * WARPS) {
            launchPdl(up_kernel<1>, grid(L.n), BS, s, L.n, (const int*)L.q_rowptr.p, (const int*)L.q_col.p,
                      (const float*)L.q_val.p, e, (const float*)L.y.p, sol(l), S);
        } else {
            withLanes(L.lpr_q, [&](auto c) {
                constexpr int P = decltype(c)::value;
                launchPdl(up_kernel<P>, grid((int64_t)L.n * P), BS, s, L.n, (const int*)L.q_rowptr.p,
                          (const int*)L.q_col.p, (const float*)L.q_val.p, e, (const float*)L.y.p, sol(l), S);
            });
        }
        profEnd(slot, s);
    }
}

}  // namespace pb
