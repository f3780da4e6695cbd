// The BiCGStab engine of the FP64, JACOBI, MIXED and LEARNED solvers with the Jacobi
// preconditioner (krylov.cu).
#pragma once
#include "solver.cuh"

namespace lsmps_gpu {

// Vectors of U + 1 doubles. The solvers that scale the columns iterate on y = D x, kept in x.
struct KrylovVecs {
    double *x, *r, *r0, *p, *v, *s, *t;
    const double* b = nullptr;
    const double* keep = nullptr;  // the warm start that a network correction replaced
};

struct KrylovOpts {
    double tol = 0;    // converged when |r| <= tol max(1, |b|)
    double delta = 0;  // mixed: residual drop between replacements by the true residual
    int chunk = 8;     // iterations between those decisions
    int max_iter = 0;
    long long max_chunks = 0;        // bound on the restarts
    int stall = 0;                   // window of the stall rule (network start)
    int use_x = 0;                   // start from x (else from zero)
    int use_nn = 0;                  // x holds a network guess or correction
    const double* warm_rn2 = nullptr;  // |b - A x|^2 of the warm start the network corrected
    const double* dinv = nullptr;    // column scaling undone at the end (null: none)
    const double* xe = nullptr;      // p*, for the error sums
};

struct KrylovResult {
    double rn, bnorm;     // |r| of the last residual, |b|
    double err2, ref2;    // |x - p*|^2, |p*|^2
    unsigned long long maxbits;  // max |x - p*|, as bits
    int iterations, outer, converged, fallback, nonfinite;
};

// A whole solve in one cooperative launch on the context stream; records event 11 after it and
// waits for the result. Af: the FP32 copy the mixed solvers iterate with (null: iterate with A).
KrylovResult krylov_solve(lsmps_ctx* ctx, const Sell<float>* Af, const Sell<double>& A, const KrylovVecs& V,
                          const KrylovOpts& o);
// The blocks of a solve of nslices slices.
unsigned krylov_blocks(lsmps_ctx* ctx, long long nslices);
// v = A p and the block partials of r0.v over a solve's blocks, whose first slices cut holds (no wait).
template <class TM>
void krylov_row_product(lsmps_ctx* ctx, const Sell<TM>& A, const int* cut, const double* p, double* v, const double* r0);

}  // namespace lsmps_gpu
