// solve.cuh -- the record kernels of a block-PCG solve (k_solve.cu) and the device-side stopping
// rule, as solver.cu drives them.
#pragma once

#include "internal.cuh"

namespace globe {

// State of the device-side PCG loop
struct PcgLoopState {
    double last;          // last max ratio (PCGsolver rule, stagnation)
    long long rhs_iters;  // sum over iterations of active columns
    int it;               // iterations completed
    int stag;             // iterations in a row with < 0.5% improvement
    int status;           // 0 running, 1 converged, 2 stagnated, 3 iteration cap, 4 breakdown
    int err_col;          // column of a breakdown
};
// The rule that an iteration's last kernel applies (st null: the host checks)
struct PcgLoop {
    PcgLoopState* st = nullptr;
    cudaGraphConditionalHandle h = 0;
    double tol = 0;
    int rule = 0, maxit = 0, k = 0;
    const double* bb = nullptr;     // |b|^2
    const double* unsc = nullptr;   // per-column factors of a double-float solve
};

// Device vectors of one solve: x, r, p (Nrec x k, column fastest), five values per individual and
// column, and the per-column scalars (k entries each; rz is followed by 2 k entries of scratch)
struct SolveVecs {
    bool df = false;                // double-float pairs, else FP64
    int k = 0;
    const int32_t* cols = nullptr;  // the active columns (null: all)
    void *x = nullptr, *r = nullptr, *p = nullptr, *ind = nullptr;
    void *alpha = nullptr, *beta = nullptr;   // in the vectors' arithmetic
    double *rz = nullptr, *pvp = nullptr, *rr = nullptr;
    const double* unsc = nullptr;   // double-float: column c runs at 1 / unsc[c]
};

int col_unscales(globe_ctx* ctx, const double* bb, int k, double* unsc);   // unsc[c] = col_unscale(bb[c])
int solve_load(globe_ctx* ctx, const SolveVecs& v, const double* in, void* out);    // column-major -> v's layout
int solve_store(globe_ctx* ctx, const SolveVecs& v, bool pending, double* out);     // x (+ alpha p, pending) -> column-major
int solve_init(globe_ctx* ctx, const SolveVecs& v);   // from r, all columns: Q^-1's factors and r'z
// zhi: the statistics words of Zi's columns to raise (null: none)
int solve_dir(globe_ctx* ctx, const SolveVecs& v, int kact, bool first, double* Zi, unsigned* zhi);
int solve_step(globe_ctx* ctx, const SolveVecs& v, int kact, const double* GZ);
int solve_update(globe_ctx* ctx, const SolveVecs& v, int kact, const PcgLoop& loop);

}  // namespace globe
