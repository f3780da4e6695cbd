// REFERENCE solver: the reference's unpreconditioned FP64 BiCGStab (src/lsmps.cpp:65-67) bit
// for bit on sm_100a: exactly rounded FP64 updates in the reference's expression order, row
// products in stored entry order, and dot products with the rounding of a sequential sum over
// the unknowns in the reference's order.
//
// What bounds it is the dependent chain of those sums: six dots of U products per iteration,
// each U rounded additions one after another (one thread adding from memory took 144 us per
// dot at U = 6,000). The chain is cut in three ways, all with the same bits:
//   * the sums run in parallel where their rounding allows it (block_seq_sum, seqsum.cuh);
//   * the products are written in the reference's order by the kernels that form their
//     factors, and independent dots (s.s, t.t, t.s; r.r, r0.r) run side by side in one launch;
//   * p and s are formed where the row products gather them, so an iteration is six launches
//     instead of 18: v = A p, its dot, t = A s, three dots, the x / r update, two dots.
// Per iteration of the shipped rain_injection configuration (U = 6,000; iterations 40 to 140; B200):
// 918 us before, 100 us now = 4.4 (v) + 34.7 (r0.v) + 3.3 (t) + 19.6 (s.s, t.t, t.s) + 2.2 (x, r) +
// 35.8 (r.r, r0.r); 507 and 81 us at U = 2,888 (smoke).
// What is left is the additions of r0.v and r0.r, whose running value leaves its binade at
// every second element, one after another: 6,000 of them at 8.2 cycles each are 25 us.
#include <algorithm>
#include <cmath>

#include "ops.cuh"
#include "seqsum.cuh"
#include "solver.cuh"

namespace lsmps_gpu {
namespace {

// ---- the iteration ----------------------------------------------------------------------------
struct ExactState {
    double rho, rho0, alpha, omega, beta, bnorm, thresh;
    double dot[3];
    double fin[3];  // final statistics: |A x - b|^2, |x - p*|^2, |p*|^2
    unsigned long long maxbits;
    unsigned ticket;
    int done;  // 1 converged, 2 break
    int s_conv;
    int iters;
    int it;
    int converged;
};

enum ExactOp { OP_START, OP_DEN, OP_ST, OP_RN, OP_FINAL };

// rho of the next iteration (src/lsmps.cpp:67: a vanishing rho ends the loop before any update)
__device__ void next_rho(ExactState* st, double rho) {
    st->rho = rho;
    if (fabs(rho) < 1e-30) st->done = 2;
    else st->beta = xmul(xdiv(st->rho, st->rho0), xdiv(st->alpha, st->omega));
}

// One block per dot over the product arrays prod + k stride; the last block to finish makes the
// iteration's scalar step. The sequential sums of a step are independent, so they overlap.
__global__ void __launch_bounds__(SEQ_THREADS) k_x_dots(const double* __restrict__ prod, long long stride,
                                                        long long U, ExactState* st, int op, double tol,
                                                        int max_iter) {
    extern __shared__ double el[];
    __shared__ SeqShared sh;
    pdl_begin();
    if (op != OP_FINAL && st->done) return;
    if (op == OP_RN && st->s_conv) {  // the |s| test passed: x took its last update
        if (blockIdx.x == 0 && threadIdx.x == 0) st->done = 1;
        return;
    }
    const double s = block_seq_sum(prod + blockIdx.x * stride, U, el, sh);
    if (threadIdx.x) return;
    st->dot[blockIdx.x] = s;
    __threadfence();
    if (atomicAdd(&st->ticket, 1u) != gridDim.x - 1) return;
    __threadfence();
    st->ticket = 0;
    const volatile double* dot = st->dot;
    const double d0 = dot[0], d1 = dot[1], d2 = dot[2];
    switch (op) {
        case OP_START:  // b.b, which is r0.r too
            st->bnorm = __dsqrt_rn(d0);
            st->thresh = xmul(tol, fmax(1.0, st->bnorm));
            st->rho0 = st->alpha = st->omega = 1.0;
            if (max_iter <= 0) st->done = 2;
            else next_rho(st, d0);
            break;
        case OP_DEN:  // r0.v
            if (fabs(d0) < 1e-30) st->done = 2;
            else st->alpha = xdiv(st->rho, d0);
            break;
        case OP_ST:  // s.s, t.t, t.s
            if (__dsqrt_rn(d0) <= st->thresh) {
                st->s_conv = 1;
                st->iters = st->it + 1;
                st->converged = 1;
            } else if (d1 < 1e-30) {
                st->done = 2;
            } else {
                st->omega = xdiv(d2, d1);
            }
            break;
        case OP_RN:  // r.r, r0.r
            st->iters = st->it + 1;
            if (__dsqrt_rn(d0) <= st->thresh) {
                st->converged = 1;
                st->done = 1;
                break;
            }
            if (fabs(st->omega) < 1e-30) {
                st->done = 2;
                break;
            }
            st->rho0 = st->rho;
            st->it += 1;
            if (st->it >= max_iter) st->done = 2;
            else next_rho(st, d1);
            break;
        case OP_FINAL:
            st->fin[0] = d0;
            st->fin[1] = d1;
            st->fin[2] = d2;
            break;
    }
}

struct ExactSystem {
    long long U;
    const int *row, *col;
    const double* val;
    const int* ref_of_u;
    double* prod;      // three product arrays in the reference's order
    long long stride;  // between them
};

// The row product sum_e val_e f(col_e) in entry order, eight lanes per row: the lanes form the
// products of 32 entries at a time (four per lane, all loads in flight together) and every lane
// adds them in entry order.
constexpr int XG = 8;
template <class F>
__device__ __forceinline__ double exact_row(const ExactSystem& A, int e0, int e1, int sub, int gbase, F&& f) {
    double s = 0.0;
    const int len = e1 - e0;
    const int most = __reduce_max_sync(0xffffffffu, len);  // the warp's rows step together
    for (int b = 0; b < most; b += 4 * XG) {
        double p[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int e = e0 + b + XG * k + sub;
            p[k] = e < e1 ? xmul(A.val[e], f(A.col[e])) : 0.0;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (b + XG * k >= most) break;
#pragma unroll
            for (int j = 0; j < XG; ++j) {
                const double pj = __shfl_sync(0xffffffffu, p[k], gbase + j);
                if (b + XG * k + j < len) s = xadd(s, pj);
            }
        }
    }
    return s;
}

// v = A p with p = r + beta (p - omega v), and the products r0 v. The old p and v are gathered
// while the new ones are written, so both have two buffers.
__global__ void __launch_bounds__(256) k_x_v(ExactSystem A, const double* __restrict__ r,
                                             const double* __restrict__ r0, const double* __restrict__ p_old,
                                             const double* __restrict__ v_old, double* __restrict__ p,
                                             double* __restrict__ v, const ExactState* st) {
    pdl_begin();
    if (st->done) return;
    const double beta = st->beta, omega = st->omega;
    auto f = [&](long long i) { return xadd(r[i], xmul(beta, xsub(p_old[i], xmul(omega, v_old[i])))); };
    const int lane = threadIdx.x & 31, sub = lane & (XG - 1), gbase = lane & ~(XG - 1);
    const long long step = (long long)gridDim.x * blockDim.x / XG;
    for (long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / 32 * (32 / XG); w < A.U; w += step) {
        const long long i = w + lane / XG;
        const bool live = i < A.U;
        const int e0 = live ? A.row[i] : 0, e1 = live ? A.row[i + 1] : 0;
        const double y = exact_row(A, e0, e1, sub, gbase, f);
        if (live && sub == 0) {
            p[i] = f(i);
            v[i] = y;
            A.prod[A.ref_of_u[i]] = xmul(r0[i], y);
        }
    }
}

// t = A s with s = r - alpha v, and the products s s, t t, t s
__global__ void __launch_bounds__(256) k_x_t(ExactSystem A, const double* __restrict__ r,
                                             const double* __restrict__ v, double* __restrict__ t,
                                             const ExactState* st) {
    pdl_begin();
    if (st->done) return;
    const double alpha = st->alpha;
    auto f = [&](long long i) { return xsub(r[i], xmul(alpha, v[i])); };
    const int lane = threadIdx.x & 31, sub = lane & (XG - 1), gbase = lane & ~(XG - 1);
    const long long step = (long long)gridDim.x * blockDim.x / XG;
    for (long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / 32 * (32 / XG); w < A.U; w += step) {
        const long long i = w + lane / XG;
        const bool live = i < A.U;
        const int e0 = live ? A.row[i] : 0, e1 = live ? A.row[i + 1] : 0;
        const double y = exact_row(A, e0, e1, sub, gbase, f);
        if (live && sub == 0) {
            const double si = f(i);
            double* q = A.prod + A.ref_of_u[i];
            t[i] = y;
            q[0] = xmul(si, si);
            q[A.stride] = xmul(y, y);
            q[2 * A.stride] = xmul(y, si);
        }
    }
}

// x += alpha p + omega s, r = s - omega t and the products r r, r0 r (or, when the |s| test
// passed, x += alpha p and r = s)
__global__ void __launch_bounds__(256) k_x_xr(ExactSystem A, double* __restrict__ x, double* __restrict__ r,
                                              const double* __restrict__ r0, const double* __restrict__ p,
                                              const double* __restrict__ v, const double* __restrict__ t,
                                              const ExactState* st) {
    pdl_begin();
    if (st->done) return;
    const double alpha = st->alpha, omega = st->omega;
    const bool last = st->s_conv != 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < A.U;
         i += (long long)gridDim.x * blockDim.x) {
        const double si = xsub(r[i], xmul(alpha, v[i]));
        if (last) {
            x[i] = xadd(x[i], xmul(alpha, p[i]));
            r[i] = si;
            continue;
        }
        x[i] = xadd(x[i], xadd(xmul(alpha, p[i]), xmul(omega, si)));
        const double ri = xsub(si, xmul(omega, t[i]));
        r[i] = ri;
        double* q = A.prod + A.ref_of_u[i];
        q[0] = xmul(ri, ri);
        q[A.stride] = xmul(r0[i], ri);
    }
}

// x = p = v = 0, r = r0 = b and the products b b
__global__ void __launch_bounds__(256) k_x_start(ExactSystem A, const double* __restrict__ b, double* __restrict__ x,
                                                 double* __restrict__ r, double* __restrict__ r0,
                                                 double* __restrict__ p, double* __restrict__ v) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < A.U;
         i += (long long)gridDim.x * blockDim.x) {
        const double bi = b[i];
        x[i] = p[i] = v[i] = 0.0;
        r[i] = r0[i] = bi;
        A.prod[A.ref_of_u[i]] = xmul(bi, bi);
    }
}

// The products of the final statistics (src/lsmps.cpp:67 tail) and max |x - p*|
__global__ void __launch_bounds__(256) k_x_final(ExactSystem A, const double* __restrict__ b,
                                                 const double* __restrict__ x, const double* __restrict__ xe,
                                                 ExactState* st) {
    pdl_begin();
    const int lane = threadIdx.x & 31, sub = lane & (XG - 1), gbase = lane & ~(XG - 1);
    const long long step = (long long)gridDim.x * blockDim.x / XG;
    double mx = 0.0;
    auto f = [&](long long i) { return x[i]; };
    for (long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / 32 * (32 / XG); w < A.U; w += step) {
        const long long i = w + lane / XG;
        const bool live = i < A.U;
        const int e0 = live ? A.row[i] : 0, e1 = live ? A.row[i + 1] : 0;
        const double y = exact_row(A, e0, e1, sub, gbase, f);
        if (live && sub == 0) {
            const double d = xsub(y, b[i]), e = xsub(x[i], xe[i]);
            double* q = A.prod + A.ref_of_u[i];
            q[0] = xmul(d, d);
            q[A.stride] = xmul(e, e);
            q[2 * A.stride] = xmul(xe[i], xe[i]);
            mx = fmax(mx, fabs(e));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0 && mx > 0) atomicMax(&st->maxbits, (unsigned long long)__double_as_longlong(mx));
}

}  // namespace

void solve_exact(lsmps_ctx* ctx, const lsmps_solver_opts* o, lsmps_ppe_stats* ps) {
    cudaStream_t s = ctx->stream;
    const long long U = ctx->U;
    double* x = ctx->vx.ensure<double>(U + 2);
    double* r = ctx->vr.ensure<double>(U + 1);
    double* r0 = ctx->vr0.ensure<double>(U + 1);
    double* p[2] = {ctx->vp.ensure<double>(U + 1), ctx->vs.ensure<double>(U + 1)};
    double* v[2] = {ctx->vv.ensure<double>(U + 1), ctx->vsh.ensure<double>(U + 1)};
    double* t = ctx->vt.ensure<double>(U + 1);
    double* prod = ctx->vph.ensure<double>(3 * (U + 1));
    ExactState* st = reinterpret_cast<ExactState*>(ctx->red.ensure<double>(64));
    static_assert(sizeof(ExactState) <= 64 * sizeof(double), "exact solver state");
    const double* b = ctx->A_b.get<double>();
    const ExactSystem A{U, ctx->A_row.get<int>(), ctx->A_col.get<int>(), ctx->A_val.get<double>(),
                        ctx->ref_of_u.get<int>(), prod, U + 1};
    LSMPS_CUDA(cudaFuncSetAttribute(k_x_dots, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SEQ_SMEM));
    LSMPS_CUDA(cudaMemsetAsync(st, 0, sizeof(ExactState), s));
    const unsigned rows = std::max(1u, std::min(blocks_for((size_t)U * XG, 256), 148u * 8));
    const unsigned vecs = std::max(1u, std::min(blocks_for((size_t)U, 256), 148u * 8));
    const int max_iter = o->max_iter;
    auto dots = [&](unsigned n, int op) {
        launch_pdl(k_x_dots, n, SEQ_THREADS, SEQ_SMEM, s, prod, U + 1, U, st, op, o->tol, max_iter);
    };
    ev_record(ctx, 10);
    ctx->have_solution = false;  // until the solve has succeeded: x is overwritten from here on
    k_x_start<<<vecs, 256, 0, s>>>(A, b, x, r, r0, p[0], v[0]);
    LSMPS_CHECK_LAUNCH();
    dots(1, OP_START);
    note_launches(1);
    const int check = std::max(1, o->check_every > 0 ? o->check_every : 16);
    for (int it = 0; it < max_iter; ++it) {
        const int cur = it & 1, nxt = cur ^ 1;
        launch_pdl(k_x_v, rows, 256, 0, s, A, r, r0, p[cur], v[cur], p[nxt], v[nxt], st);
        dots(1, OP_DEN);
        launch_pdl(k_x_t, rows, 256, 0, s, A, r, v[nxt], t, st);
        dots(3, OP_ST);
        launch_pdl(k_x_xr, vecs, 256, 0, s, A, x, r, r0, p[nxt], v[nxt], t, st);
        dots(2, OP_RN);
        note_launches(6);
        if ((it + 1) % check == 0) {
            int done = 0;
            read_back(ctx, {{&st->done, &done, sizeof(int)}}, nullptr);
            if (done) break;
        }
    }
    ev_record(ctx, 11);
    launch_pdl(k_x_final, rows, 256, 0, s, A, b, x, ctx->A_xexact.get<double>(), st);
    dots(3, OP_FINAL);
    note_launches(2);
    ExactState h{};
    read_back(ctx, {{st, &h, sizeof(h)}}, nullptr);
    double mx;
    static_assert(sizeof(mx) == sizeof(h.maxbits), "double bits");
    std::copy_n(reinterpret_cast<const char*>(&h.maxbits), sizeof(mx), reinterpret_cast<char*>(&mx));
    ps->iterations = h.iters;
    ps->converged = h.converged;
    ps->initial_residual = h.bnorm;
    ps->final_residual = std::sqrt(h.fin[0]);
    ps->relative_l2_error = std::sqrt(h.fin[1] / std::fmax(h.fin[2], 1e-30));
    ps->max_error = mx;
    ps->relative_residual = ps->final_residual / std::max(h.bnorm, 1e-300);
    ps->solve_ms = ev_elapsed(ctx, 10, 11);
}

}  // namespace lsmps_gpu
