// samg.h -- smoothed-aggregation multigrid, the preconditioner of flexible CG on symmetric
// positive (semi-)definite systems and of BiCGSTAB on other transport equations.
#pragma once

#include <memory>
#include <vector>

#include "common.h"
#include "krylov.h"

namespace pb {

// One level. Level 0 borrows the equation's SELL-32 matrix; coarser matrices are CSR.
// For the transfer to the next level, P = (I - omega_p D^-1 A) P0 is the smoothed
// prolongation and Q = (I - omega D^-1 A) P: the up-sweep adds Q e, and for symmetric A the
// down-sweep is b_next = Q^T b. Otherwise R^T is P made with A^T and the down-sweep's matrix
// that Q^T made with A^T and R^T.
struct SaLevel {
    int n = 0;
    int64_t nnz = 0;
    // A: CSR pattern; the values sit at vals[csr_pos[k]] (level 0) or vals[k] (csr_pos null)
    const int* rowptr = nullptr;
    const int* col = nullptr;
    const int* csr_pos = nullptr;
    const double* vals = nullptr;
    ArenaBuf<int> o_rowptr, o_col, o_csr_pos;
    ArenaBuf<int> tr_pos;  // A not symmetric: place in vals of each entry's transpose (-1: none)
    ArenaBuf<double> o_vals;
    // level 0: the SELL-32 view
    int nslices = 0;
    int64_t sell_nnz = 0;
    const int* sl_off = nullptr;
    const int* sl_col = nullptr;
    const int* diag_pos = nullptr;
    double omega = 0.0, omega_p = 0.0;
    ArenaBuf<double> dinv;
    ArenaBuf<float> wd;    // omega D^-1
    ArenaBuf<float> as32;  // A (omega D^-1) in FP32: SELL layout on level 0, CSR below
    int lpr_a = 1;         // lanes per row of the CSR passes over A, Q and Q^T
    int lpr_p = 1, lpr_q = 1, lpr_t = 1;
    // transfer to the next level
    ArenaBuf<int> agg;
    ArenaBuf<int> p_rowptr, p_col;           // P
    ArenaBuf<double> p_val, r_val;           // r_val: R^T on P's pattern (A not symmetric)
    ArenaBuf<int> pt_rowptr, pt_row, pt_src; // P^T: fine row and P entry of each
    ArenaBuf<int> q_rowptr, q_col, q_tpos;   // Q (the pattern of A P); q_tpos: its place in Q^T
    ArenaBuf<double> ap_val;                 // A P
    ArenaBuf<float> q_val;
    int64_t p_nnz = 0, q_nnz = 0;
    ArenaBuf<int> t_rowptr, t_col;           // Q^T
    ArenaBuf<float> t_val;
    ArenaBuf<float> b, x, y;                 // cycle vectors (FP32)
};

struct SaAmg {
    DevArena arena;  // declared first: released last
    std::vector<std::unique_ptr<SaLevel>> levels;
    bool built = false, symmetric = true;
    bool fresh = false;  // the last setup built the structure: it belongs to the matrix of that call
    uint64_t generation = 0;
    // rows x (entries per row)^2 of the coarse levels over the matrix's: beyond it setup throws
    double max_fill = 25.0;
    int tail = -1;  // first level of the fused coarse tail (-1: none)
    int coarse_n = 0;
    ArenaBuf<double> coarse_a;
    ArenaBuf<float> coarse_inv32;

    // Builds the hierarchy (first call on a pattern) or refreshes its values for the
    // matrix A, whose CSR pattern lists each row's entries in the order of its SELL slots.
    // sym: A is symmetric. keep_values: the matrix is unchanged since the last call.
    void setup(const SellMatrix& A, const int* rowptr, const int* col, bool sym, bool keep_values, cudaStream_t s);
    // z = B r, one V(1,1) cycle in FP32; S (optional): skip the work once the solve has
    // stopped; sample: time the finest-level kernels when a profiling window is open
    void apply(const float* r, float* z, const KState* S, cudaStream_t s, bool sample = false);

private:
    void build(const SellMatrix& A, const int* rowptr, const int* col, bool sym, cudaStream_t s);
    void levelScaling(SaLevel& L, cudaStream_t s);
    void levelValues(size_t l, cudaStream_t s);
};

}  // namespace pb
