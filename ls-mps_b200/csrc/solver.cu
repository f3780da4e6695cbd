// PPE solvers on sm_100a.
//
// * REFERENCE: the reference's unpreconditioned FP64 BiCGStab (src/lsmps.cpp:65-67)
//   reproduced bit for bit (exact.cu).
// * FP64 / JACOBI: the same iteration with GPU reductions. Jacobi right preconditioning
//   is applied as a column scaling of the matrix (A D^-1, solve for y, x = D^-1 y), which
//   costs nothing per iteration.
// * MIXED / LEARNED: the Jacobi iteration with an FP32 copy of the matrix and residual
//   replacement by the FP64 one; LEARNED starts from the message-passing network's guess.
// These run in one cooperative launch per solve (krylov.cu). Here are the SELL copies, the
// multigrid-preconditioned MIXED / LEARNED iteration and MIXED_F32, whose kernels the host
// launches: each reduction is fused into the kernel that produces its operands; the last block
// of the grid to finish (atomic ticket) sums the per-block partials in a fixed order, so results
// are deterministic, and updates the scalars in device memory. Every kernel returns at once when
// the run is done, so the host reads the status once per chunk of iterations.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <tuple>
#include <utility>

#include "krylov.cuh"
#include "ops.cuh"
#include "scan.cuh"
#include "sell.cuh"

namespace lsmps_gpu {


namespace {

constexpr int RB = 256;            // threads per block
constexpr int RGRID = 148 * 6;     // persistent grid of the vector / SpMV kernels

// ---------------------------------------------------------------------------------------
// Fast engine
// ---------------------------------------------------------------------------------------
struct Partials {
    double* a;   // RGRID entries
    double* b;   // RGRID entries
};

// Block sum of two doubles into partials[blockIdx]; returns true in the last block to
// arrive, after which the caller may read all partials (fixed-order final sum).
__device__ __forceinline__ bool block_partials(double va, double vb, Partials P, unsigned int* counter) {
    __shared__ double sa[RB / 32], sb[RB / 32];
    __shared__ bool last;
    va = warp_sum(va);
    vb = warp_sum(vb);
    int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) { sa[w] = va; sb[w] = vb; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ta = 0, tb = 0;
        for (int k = 0; k < RB / 32; ++k) { ta += sa[k]; tb += sb[k]; }
        P.a[blockIdx.x] = ta;
        P.b[blockIdx.x] = tb;
        __threadfence();
        unsigned int ticket = atomicAdd(counter, 1u);
        last = ticket == gridDim.x - 1;
    }
    __syncthreads();
    return last;
}

// In the last block: fixed-order sum of the partials (thread t sums entries t, t+RB, ...
// then a fixed tree), result in *ra / *rb for thread 0.
__device__ __forceinline__ void final_sum(Partials P, double* ra, double* rb) {
    __shared__ double sa[RB / 32], sb[RB / 32];
    double va = 0, vb = 0;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += RB) {
        va += __ldcg(P.a + k);
        vb += __ldcg(P.b + k);
    }
    va = warp_sum(va);
    vb = warp_sum(vb);
    if ((threadIdx.x & 31) == 0) { sa[threadIdx.x >> 5] = va; sb[threadIdx.x >> 5] = vb; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ta = 0, tb = 0;
        for (int k = 0; k < RB / 32; ++k) { ta += sa[k]; tb += sb[k]; }
        *ra = ta;
        *rb = tb;
    }
}

// grid of the row-product kernels: the pipelined products take 64 registers
template <class TM, bool C16>
constexpr int spmv_blocks_per_sm() {
    return C16 && sizeof(TM) == 4 ? 4 : 6;
}
template <class TM, bool C16>
constexpr unsigned spmv_grid() {
    return 148u * spmv_blocks_per_sm<TM, C16>();
}

#define SELL_LOOP(A)                                                              \
    const int lane = threadIdx.x & 31;                                            \
    const long long w0 = (blockIdx.x * (long long)RB + threadIdx.x) >> 5;         \
    const long long nw = ((long long)gridDim.x * RB) >> 5;                        \
    for (long long s = w0; s < (A).nslices; s += nw)

// Four consecutive vector elements per thread and access (float4, or two double2), so
// the elementwise kernels keep 16-32 bytes per array in flight per thread.
template <class T>
struct V4 {
    T a[4];
};
__device__ __forceinline__ V4<float> ld_v4(const float* p) {
    float4 q = *reinterpret_cast<const float4*>(p);
    return {{q.x, q.y, q.z, q.w}};
}
__device__ __forceinline__ V4<double> ld_v4(const double* p) {
    double2 u = reinterpret_cast<const double2*>(p)[0], w = reinterpret_cast<const double2*>(p)[1];
    return {{u.x, u.y, w.x, w.y}};
}
__device__ __forceinline__ void st_v4(float* p, const V4<float>& v) {
    *reinterpret_cast<float4*>(p) = make_float4(v.a[0], v.a[1], v.a[2], v.a[3]);
}
__device__ __forceinline__ void st_v4(double* p, const V4<double>& v) {
    reinterpret_cast<double2*>(p)[0] = make_double2(v.a[0], v.a[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(v.a[2], v.a[3]);
}

// Calls f4(i) for i = 0, 4, 8, ... (groups of four elements), then f1(i) for the tail.
template <class F4, class F1>
__device__ __forceinline__ void vec_loop(long long n, F4&& f4, F1&& f1) {
    const long long n4 = n >> 2;
    for (long long q = blockIdx.x * (long long)RB + threadIdx.x; q < n4; q += (long long)gridDim.x * RB) f4(q << 2);
    for (long long i = (n4 << 2) + blockIdx.x * (long long)RB + threadIdx.x; i < n; i += (long long)gridDim.x * RB)
        f1(i);
}

// p = r + beta (p - omega v)
template <class T>
__global__ void __launch_bounds__(RB) k_bcg_p(long long n, const T* __restrict__ r, T* __restrict__ p,
                                              const T* __restrict__ v, const BcgScalars* S) {
    pdl_begin();
    if (S->done) return;
    const T beta = (T)S->beta, omega = (T)S->omega;
    vec_loop(n, [&](long long i) {
        V4<T> rr = ld_v4(r + i), pp = ld_v4(p + i), vv = ld_v4(v + i);
#pragma unroll
        for (int j = 0; j < 4; ++j) pp.a[j] = rr.a[j] + beta * (pp.a[j] - omega * vv.a[j]);
        st_v4(p + i, pp);
    }, [&](long long i) { p[i] = r[i] + beta * (p[i] - omega * v[i]); });
}

// v = A p; den = (r0, v); alpha = rho / den
template <class T, class TM = T, bool C16 = false>
__global__ void __launch_bounds__(RB, spmv_blocks_per_sm<TM, C16>()) k_bcg_v(Sell<TM> A, const T* __restrict__ p, T* __restrict__ v,
                                              const T* __restrict__ r0, BcgScalars* S, Partials P) {
    pdl_begin();
    if (S->done) return;
    double acc = 0;
    SELL_LOOP(A) {
        double y = sell_product<C16>(A, s, lane, p);
        long long i = (s << 5) + lane;
        if (i < A.n) {
            T yi = (T)y;
            v[i] = yi;
            acc += (double)r0[i] * (double)yi;
        }
    }
    if (block_partials(acc, 0.0, P, &S->counter[0])) {
        double den, unused;
        final_sum(P, &den, &unused);
        if (threadIdx.x == 0) {
            S->counter[0] = 0;
            if (!isfinite(den)) { S->nonfinite = 1; S->done = 2; }
            else if (fabs(den) < 1e-30) S->done = 2;
            else S->alpha = S->rho / den;
        }
    }
}

// s = r - alpha v; |s|
template <class T>
__global__ void __launch_bounds__(RB) k_bcg_s(long long n, const T* __restrict__ r, const T* __restrict__ v,
                                              T* __restrict__ s, BcgScalars* S, Partials P) {
    pdl_begin();
    if (S->done) return;
    const T alpha = (T)S->alpha;
    double acc = 0;
    vec_loop(n, [&](long long i) {
        V4<T> rr = ld_v4(r + i), vv = ld_v4(v + i), ss;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            ss.a[j] = rr.a[j] - alpha * vv.a[j];
            acc += (double)ss.a[j] * (double)ss.a[j];
        }
        st_v4(s + i, ss);
    }, [&](long long i) {
        T si = r[i] - alpha * v[i];
        s[i] = si;
        acc += (double)si * (double)si;
    });
    if (block_partials(acc, 0.0, P, &S->counter[1])) {
        double ss, unused;
        final_sum(P, &ss, &unused);
        if (threadIdx.x == 0) {
            S->counter[1] = 0;
            S->sn = sqrt(ss);
            if (S->sn <= S->thresh) { S->s_conv = 1; S->iters = S->it + 1; }
        }
    }
}

// With the multigrid, the p and s updates also restrict the new vector to level 1
// (r1 = P^T p, a sum over each aggregate's contiguous rows). A warp takes AGG_W consecutive
// aggregates, i.e. the rows ustart[Ia] .. ustart[Ia + AGG_W], and walks them 32 consecutive rows
// per step, so every load and store is coalesced. A segmented shuffle scan sums each step's
// rows per aggregate and the segment's last lane adds that sum into the aggregate's shared-
// memory slot; steps run in order, so the summation order is fixed.
constexpr int AGG_W = 16;  // aggregates per warp task

inline unsigned agg_blocks(long long n1) {
    return (unsigned)(((n1 + AGG_W - 1) / AGG_W + RB / 32 - 1) / (RB / 32));
}

// Calls f(i) (which returns the new value of row i) for every row of aggregates [Ia, Ib) and
// returns, in lane l < Ib - Ia, the sum over aggregate Ia + l. `sh` is the warp's AGG_W slots.
template <class F>
__device__ __forceinline__ double warp_agg_sums(const MgFine& G, long long Ia, long long Ib, double* sh, F&& f) {
    const int lane = threadIdx.x & 31;
    if (lane < AGG_W) sh[lane] = 0.0;
    __syncwarp();
    const int rb = G.ustart[Ia], re = G.ustart[Ib];
    // segment sums of one step: inclusive scan within runs of equal a, the run's last lane adds
    auto deliver = [&](double x, int a, bool live) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, x, o);
            const int ay = __shfl_up_sync(0xffffffffu, a, o);
            if (lane >= o && ay == a) x += y;
        }
        const int an = __shfl_down_sync(0xffffffffu, a, 1);
        if (live && (lane == 31 || an != a)) sh[a] += x;
        __syncwarp();
    };
    // two steps per pass: both steps' loads are in flight before either scan
    for (int base = rb; base < re; base += 64) {
        const int i0 = base + lane, i1 = base + 32 + lane;
        const bool l0 = i0 < re, l1 = i1 < re;
        int a0 = AGG_W + lane, a1 = AGG_W + lane;  // past the last row: a key of its own, in no run
        if (l0) a0 = G.agg0[i0] - (int)Ia;
        if (l1) a1 = G.agg0[i1] - (int)Ia;
        const double x0 = l0 ? f(i0) : 0.0;
        const double x1 = l1 ? f(i1) : 0.0;
        deliver(x0, a0, l0);
        deliver(x1, a1, l1);
    }
    const double sum = lane < AGG_W ? sh[lane] : 0.0;
    __syncwarp();  // before the next task clears the slots
    return sum;
}

__global__ void __launch_bounds__(RB) k_bcg_p_agg(MgFine G, const double* __restrict__ r, double* __restrict__ p,
                                                  const double* __restrict__ v, const BcgScalars* S) {
    pdl_begin();
    if (S->done) return;
    __shared__ double sh[RB / 32][AGG_W];
    const double beta = S->beta, omega = S->omega;
    const int lane = threadIdx.x & 31;
    const long long nt = (G.n1 + AGG_W - 1) / AGG_W;
    for (long long task = (blockIdx.x * (long long)RB + threadIdx.x) >> 5; task < nt;
         task += ((long long)gridDim.x * RB) >> 5) {
        const long long Ia = task * AGG_W, Ib = min(Ia + AGG_W, G.n1);
        const double a = warp_agg_sums(G, Ia, Ib, sh[threadIdx.x >> 5], [&](int i) {
            const double pi = r[i] + beta * (p[i] - omega * v[i]);
            p[i] = pi;
            return pi;
        });
        if (Ia + lane < Ib) {
            G.r1[Ia + lane] = (float)a;
            G.x1[Ia + lane] = G.omega * (float)a * G.dinv1[Ia + lane];
        }
    }
}

// s = r - alpha v, |s|, and r1 = P^T s in one pass (grid at most RGRID blocks: one partial
// sum of |s|^2 per block).
__global__ void __launch_bounds__(RB) k_bcg_s_agg(MgFine G, const double* __restrict__ r,
                                                  const double* __restrict__ v, double* __restrict__ s,
                                                  BcgScalars* S, Partials P) {
    pdl_begin();
    if (S->done) return;
    __shared__ double sh[RB / 32][AGG_W];
    const double alpha = S->alpha;
    const int lane = threadIdx.x & 31;
    const long long nt = (G.n1 + AGG_W - 1) / AGG_W;
    double acc = 0;
    for (long long task = (blockIdx.x * (long long)RB + threadIdx.x) >> 5; task < nt;
         task += ((long long)gridDim.x * RB) >> 5) {
        const long long Ia = task * AGG_W, Ib = min(Ia + AGG_W, G.n1);
        const double a = warp_agg_sums(G, Ia, Ib, sh[threadIdx.x >> 5], [&](int i) {
            const double si = r[i] - alpha * v[i];
            s[i] = si;
            acc += si * si;
            return si;
        });
        if (Ia + lane < Ib) {
            G.r1[Ia + lane] = (float)a;
            G.x1[Ia + lane] = G.omega * (float)a * G.dinv1[Ia + lane];
        }
    }
    if (block_partials(acc, 0.0, P, &S->counter[1])) {
        double ss, unused;
        final_sum(P, &ss, &unused);
        if (threadIdx.x == 0) {
            S->counter[1] = 0;
            S->sn = sqrt(ss);
            if (S->sn <= S->thresh) { S->s_conv = 1; S->iters = S->it + 1; }
        }
    }
}

// t = A s; omega = (t, s) / (t, t). sd: the s of the dot where sv is a preconditioned M s.
template <class T, class TM = T, bool C16 = false>
__global__ void __launch_bounds__(RB, spmv_blocks_per_sm<TM, C16>()) k_bcg_t(Sell<TM> A, const T* __restrict__ sv, T* __restrict__ t,
                                              BcgScalars* S, Partials P, const T* __restrict__ sd) {
    pdl_begin();
    if (S->done || S->s_conv) return;
    double ats = 0, att = 0;
    SELL_LOOP(A) {
        double y = sell_product<C16>(A, s, lane, sv);
        long long i = (s << 5) + lane;
        if (i < A.n) {
            T ti = (T)y;
            t[i] = ti;
            ats += (double)ti * (double)sd[i];
            att += (double)ti * (double)ti;
        }
    }
    if (block_partials(ats, att, P, &S->counter[2])) {
        double ts, tt;
        final_sum(P, &ts, &tt);
        if (threadIdx.x == 0) {
            S->counter[2] = 0;
            S->tt = tt;
            if (!isfinite(tt) || !isfinite(ts)) { S->nonfinite = 1; S->done = 2; }
            else if (tt < 1e-30) S->done = 2;
            else S->omega = ts / tt;
        }
    }
}

// x += alpha p + omega s; r = s - omega t; |r|, rho' = (r0, r); beta
// (or, when the |s| test passed: x += alpha p and finish). PRE: the x update takes the
// preconditioned directions ph = M p and sh = M s instead of p and s.
template <class T, bool PRE = false>
__global__ void __launch_bounds__(RB) k_bcg_x(long long n, T* __restrict__ x, T* __restrict__ r,
                                              const T* __restrict__ p, const T* __restrict__ s,
                                              const T* __restrict__ t, const T* __restrict__ r0,
                                              BcgScalars* S, Partials P, const T* __restrict__ ph = nullptr,
                                              const T* __restrict__ sh = nullptr) {
    pdl_begin();
    if (S->done) return;
    const T alpha = (T)S->alpha, omega = (T)S->omega;
    const T* __restrict__ xp = PRE ? ph : p;
    const T* __restrict__ xs = PRE ? sh : s;
    if (S->s_conv) {
        for (long long i = blockIdx.x * (long long)RB + threadIdx.x; i < n; i += (long long)gridDim.x * RB) {
            x[i] += alpha * xp[i];
            r[i] = s[i];
        }
        __syncthreads();
        if (block_partials(0.0, 0.0, P, &S->counter[3]) && threadIdx.x == 0) {
            S->counter[3] = 0;
            S->rn = S->sn;
            S->done = 1;
        }
        return;
    }
    double arr = 0, ar0r = 0;
    vec_loop(n, [&](long long i) {
        V4<T> xx = ld_v4(x + i), pp = ld_v4(xp + i), ss = ld_v4(s + i), tt = ld_v4(t + i), q0 = ld_v4(r0 + i), rr;
        V4<T> xsv = PRE ? ld_v4(xs + i) : ss;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            xx.a[j] += alpha * pp.a[j] + omega * xsv.a[j];
            rr.a[j] = ss.a[j] - omega * tt.a[j];
            arr += (double)rr.a[j] * (double)rr.a[j];
            ar0r += (double)q0.a[j] * (double)rr.a[j];
        }
        st_v4(x + i, xx);
        st_v4(r + i, rr);
    }, [&](long long i) {
        T si = s[i];
        x[i] += alpha * xp[i] + omega * (PRE ? xs[i] : si);
        T ri = si - omega * t[i];
        r[i] = ri;
        arr += (double)ri * (double)ri;
        ar0r += (double)r0[i] * (double)ri;
    });
    if (block_partials(arr, ar0r, P, &S->counter[3])) {
        double rr, rho;
        final_sum(P, &rr, &rho);
        if (threadIdx.x == 0) {
            S->counter[3] = 0;
            S->iters = S->it + 1;
            S->it += 1;
            double rn = sqrt(rr);
            S->rn = rn;
            if (!isfinite(rn)) { S->nonfinite = 1; S->done = 2; return; }
            if (rn <= S->thresh) { S->done = 1; return; }
            // stall bookkeeping (learned solver fallback rule)
            if (rn < 0.99 * S->best_rn) { S->best_rn = rn; S->since_best = 0; }
            else if (++S->since_best >= S->stall_window && S->stall_window > 0) { S->done = 4; return; }
            if (fabs(S->omega) < 1e-30) { S->done = 2; return; }
            if (S->it >= S->max_iter) { S->done = 3; return; }
            if (fabs(rho) < 1e-30) { S->done = 2; return; }
            S->beta = (rho / S->rho) * (S->alpha / S->omega);
            S->rho0 = S->rho;
            S->rho = rho;
        }
    }
}

// Initialisation: r = b - A x (or r = b when x = 0), r0 = r, p = v = 0, |b|, rho = (r0, r).
template <class T, class TM = T, bool C16 = false>
__global__ void __launch_bounds__(RB, 6) k_bcg_init(Sell<TM> A, const T* __restrict__ b, const T* __restrict__ x,
                                                 int use_x, T* __restrict__ r, T* __restrict__ r0,
                                                 T* __restrict__ p, T* __restrict__ v, BcgScalars* S,
                                                 Partials P, double tol, double bnorm_override) {
    double abb = 0, arr = 0;
    SELL_LOOP(A) {
        double ax = use_x ? sell_row<C16>(A, s, lane, x) : 0.0;
        long long i = (s << 5) + lane;
        if (i < A.n) {
            T bi = b[i];
            T ri = use_x ? (T)((double)bi - ax) : bi;
            r[i] = ri;
            r0[i] = ri;
            p[i] = 0;
            v[i] = 0;
            abb += (double)bi * (double)bi;
            arr += (double)ri * (double)ri;
        }
    }
    if (block_partials(abb, arr, P, &S->counter[4])) {
        double bb, rr;
        final_sum(P, &bb, &rr);
        if (threadIdx.x == 0) {
            S->counter[4] = 0;
            double bnorm = bnorm_override >= 0 ? bnorm_override : sqrt(bb);
            S->bnorm = sqrt(bb);
            S->thresh = tol * fmax(1.0, bnorm);
            S->rho0 = S->alpha = S->omega = 1.0;
            S->rho = rr;
            S->beta = rr;  // (rho / rho0) (alpha / omega) with rho0 = alpha = omega = 1
            S->rn = sqrt(rr);
            S->best_rn = S->rn;
            S->since_best = 0;
            S->it = 0;
            S->iters = 0;
            S->s_conv = 0;
            S->nonfinite = !isfinite(rr) ? 1 : 0;
            S->done = 0;
            if (S->nonfinite) S->done = 2;
            else if (S->rn <= S->thresh) S->done = 1;  // already converged
            else if (fabs(rr) < 1e-30) S->done = 2;
            else if (S->max_iter <= 0) S->done = 3;
        }
    }
}

// r = b - A x (FP64), |r|^2 and |b|^2 into out2 (fixed-order partials).
template <bool C16 = false>
__global__ void __launch_bounds__(RB, 6) k_residual64(Sell<double> A, const double* __restrict__ b,
                                                   const double* __restrict__ x, double* __restrict__ r,
                                                   double* out2, Partials P, unsigned int* counter) {
    double arr = 0, abb = 0;
    SELL_LOOP(A) {
        double ax = sell_row<C16>(A, s, lane, x);
        long long i = (s << 5) + lane;
        if (i < A.n) {
            double ri = b[i] - ax;
            r[i] = ri;
            arr += ri * ri;
            abb += b[i] * b[i];
        }
    }
    if (block_partials(arr, abb, P, counter)) {
        double rr, bb;
        final_sum(P, &rr, &bb);
        if (threadIdx.x == 0) {
            *counter = 0;
            out2[0] = rr;
            out2[1] = bb;
        }
    }
}

// ---- SELL-32 construction from the CSR rows ----
// slice lengths: one warp per slice
__global__ void k_sell_len(long long n, long long nslices, const int* __restrict__ row, int* __restrict__ slen,
                           int* __restrict__ ssize) {
    const int lane = threadIdx.x & 31;
    long long s = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    if (s >= nslices) return;
    long long i = (s << 5) + lane;
    int len = i < n ? row[i + 1] - row[i] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) len = max(len, __shfl_xor_sync(0xffffffffu, len, o));
    len = (len + 3) & ~3;  // chunks of four entries
    if (lane == 0) {
        slen[s] = len;
        ssize[s] = len * 32;
    }
}

// All SELL arrays of a slice of 32 rows in one pass, SB_WARPS warps per slice: the slice's CSR
// entries (one contiguous range) are staged in shared memory with asynchronous copies, all in
// flight at once, and scaled there in CSR order; then a thread writes every SB_WARPS-th group of
// four entries of its row with 16-byte stores: columns (the diagonal moved to its place in column
// order, padding repeating the last column), values A (padding 0), the column steps and the row's
// first column (any row that does not ascend or steps by more than 65535 sets *bad), and the
// column-scaled copies A D^-1 in FP64 and FP32. Slices of more than `cap` entries read their rows
// from global memory instead. Same values as a per-row fill followed by the column-scaling passes
// (each scaled value is the same single product, rounded once).
// What bounds it: the copies' and the row loop's latency, so it is the number of warps per SM that
// counts: 416 us for 911k unknowns and 102 for 181k when one warp staged a slice with one load
// per step and slices above 1,024 entries (an interior slice has 1,056) were read in place, 286
// and 58 with one warp and asynchronous copies, 196 and 45 with four warps (227 and 52 with two,
// 227 and 48 with eight).
constexpr int SB_MAX = 4000;  // entries staged at most (48 KB)
constexpr int SB_WARPS = 4;
template <int N>
__device__ __forceinline__ void copy_async(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "n"(N)
                 : "memory");
}
__global__ void __launch_bounds__(32 * SB_WARPS) k_sell_build(
    long long n, const int* __restrict__ row, const int* __restrict__ acol, const double* __restrict__ aval,
    const double* __restrict__ dinv, const int* __restrict__ sptr, const int* __restrict__ slen, int* __restrict__ col,
    double* __restrict__ val, unsigned short* __restrict__ dcol, int* __restrict__ rbase, double* __restrict__ vals,
    float* __restrict__ valf, int* bad, int raw, int cap) {
    extern __shared__ double sval[];  // cap values, then cap columns
    int* scol = reinterpret_cast<int*>(sval + cap);
    __shared__ int diag[32];  // where each row's diagonal goes
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long s = blockIdx.x;
    const long long u0 = s << 5, i = u0 + lane;
    const int b0 = row[u0], b1 = row[min(u0 + 32, n)], total = b1 - b0;
    const bool staged = total <= cap;
    if (staged)
        for (int t = threadIdx.x; t < total; t += 32 * SB_WARPS) {
            copy_async<4>(scol + t, acol + b0 + t);
            copy_async<8>(sval + t, aval + b0 + t);
        }
    int e0 = 0, len = 0;
    if (i < n) {
        e0 = row[i];
        len = row[i + 1] - e0;
    }
    if (w == 0) diag[lane] = max(len - 1, 0);
    const int L = slen[s];
    const long long base = (long long)sptr[s] + 4 * lane;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const bool scaled = staged && !raw;  // the staged values are scaled in place
    if (scaled)
#pragma unroll 4
        for (int t = threadIdx.x; t < total; t += 32 * SB_WARPS) sval[t] *= dinv[scol[t]];
    auto C = [&](int e) { return staged ? scol[e - b0] : acol[e]; };
    auto V = [&](int e) { return staged ? sval[e - b0] : aval[e]; };
    // the CSR row's last entry is its diagonal: it goes before the first entry of a larger column
    // (each warp looks at a part of the row)
    const int part = (len + SB_WARPS - 2) / SB_WARPS;
    for (int k = w * part; k < min((w + 1) * part, len - 1); ++k)
        if (C(e0 + k) >= (int)i) {
            atomicMin(&diag[lane], k);
            break;
        }
    __syncthreads();
    const int pos = diag[lane];
    auto at = [&](int k) { return k < pos ? e0 + k : (k == pos ? e0 + len - 1 : e0 + k - 1); };  // the row's k-th entry
    const int last = len > 0 ? C(at(len - 1)) : (i < n ? (int)i : 0);
    bool ok = true;
    for (int k4 = 4 * w; k4 < L; k4 += 4 * SB_WARPS) {
        int cc[4];
        double vv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k4 + j;
            cc[j] = k < len ? C(at(k)) : last;
            vv[j] = k < len ? V(at(k)) : 0.0;
        }
        if (k4 == 0) rbase[i] = cc[0];
        int prev = k4 == 0 ? cc[0] : k4 - 1 < len ? C(at(k4 - 1)) : last;
        unsigned short dd[4];
        double sv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int d = cc[j] - prev;
            ok = ok && d >= 0 && d <= 65535;
            dd[j] = (unsigned short)(d >= 0 && d <= 65535 ? d : 0);
            prev = cc[j];
            sv[j] = scaled ? vv[j] : vv[j] * dinv[cc[j]];
        }
        const long long e = base + 128LL * (k4 >> 2);
        if (raw) {  // unscaled values and 32-bit columns: only the plain FP64 solver reads them
            *reinterpret_cast<int4*>(col + e) = make_int4(cc[0], cc[1], cc[2], cc[3]);
            *reinterpret_cast<double2*>(val + e) = make_double2(vv[0], vv[1]);
            *reinterpret_cast<double2*>(val + e + 2) = make_double2(vv[2], vv[3]);
        }
        *reinterpret_cast<ushort4*>(dcol + e) = make_ushort4(dd[0], dd[1], dd[2], dd[3]);
        *reinterpret_cast<double2*>(vals + e) = make_double2(sv[0], sv[1]);
        *reinterpret_cast<double2*>(vals + e + 2) = make_double2(sv[2], sv[3]);
        *reinterpret_cast<float4*>(valf + e) =
            make_float4((float)sv[0], (float)sv[1], (float)sv[2], (float)sv[3]);
    }
    if (!ok) atomicOr(bad, 1);
}

// cut[b]: the first slice of a solve's block b
template <class T>
__global__ void k_sell_cuts(Sell<T> A, unsigned blocks, int* __restrict__ cut) {
    for (unsigned b = threadIdx.x; b <= blocks; b += blockDim.x) cut[b] = (int)sell_cut(A, b, blocks);
}

// ---------------------------------------------------------------------------------------
// Mixed-precision helpers
// ---------------------------------------------------------------------------------------
template <class T>
__global__ void k_fill(long long n, T* __restrict__ x, T v) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        x[i] = v;
}

__global__ void k_unscale(long long n, double* __restrict__ x, const double* __restrict__ dinv) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        x[i] *= dinv[i];
}

__global__ void k_scale_by_diag(long long n, double* __restrict__ x, const double* __restrict__ dinv) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        x[i] = dinv[i] != 0 ? x[i] / dinv[i] : x[i];
}

// error statistics against p*: |x - p*|^2, |p*|^2, max |x - p*| (fixed-order partials)
__global__ void __launch_bounds__(RB) k_error_stats(long long n, const double* __restrict__ x,
                                                    const double* __restrict__ xe, double* out3, Partials P,
                                                    unsigned int* counter, unsigned long long* maxbits) {
    double se = 0, ee = 0, mx = 0;
    for (long long i = blockIdx.x * (long long)RB + threadIdx.x; i < n; i += (long long)gridDim.x * RB) {
        double e = x[i] - xe[i];
        se += e * e;
        ee += xe[i] * xe[i];
        mx = fmax(mx, fabs(e));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) atomicMax(maxbits, (unsigned long long)__double_as_longlong(mx));
    if (block_partials(se, ee, P, counter)) {
        double a, b;
        final_sum(P, &a, &b);
        if (threadIdx.x == 0) {
            *counter = 0;
            out3[0] = a;
            out3[1] = b;
        }
    }
}

// ---- reliable updates of the mixed-precision solver ----
// x_hi += sigma D^-1 y_lo (FP64), y_lo = 0
__global__ void k_reliable_x(long long n, double* __restrict__ x, float* __restrict__ y,
                             const double* __restrict__ dinv, const double* sigma) {
    const double sg = *sigma;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        x[i] += sg * dinv[i] * (double)y[i];
        y[i] = 0.f;
    }
}

// r = r64 / sigma in FP32 replaces the recursive residual; rho' = (r0, r) and the next
// beta follow, so the iteration continues with its search direction (van der Vorst & Ye
// residual replacement).
__global__ void __launch_bounds__(RB) k_reliable_r(long long n, const double* __restrict__ r64,
                                                   const double* sigma, float* __restrict__ r,
                                                   const float* __restrict__ r0, BcgScalars* S, Partials P) {
    const double inv = 1.0 / *sigma;
    double arr = 0, ar0r = 0;
    for (long long i = blockIdx.x * (long long)RB + threadIdx.x; i < n; i += (long long)gridDim.x * RB) {
        float ri = (float)(r64[i] * inv);
        r[i] = ri;
        arr += (double)ri * (double)ri;
        ar0r += (double)r0[i] * (double)ri;
    }
    if (block_partials(arr, ar0r, P, &S->counter[7])) {
        double rr, rho;
        final_sum(P, &rr, &rho);
        if (threadIdx.x == 0) {
            S->counter[7] = 0;
            S->rn = sqrt(rr);
            if (S->rn < S->best_rn) S->best_rn = S->rn;
            S->beta = (rho / S->rho0) * (S->alpha / S->omega);
            S->rho = rho;
            S->done = 0;
            S->s_conv = 0;
            if (!isfinite(rho) || fabs(rho) < 1e-30) S->done = 2;
        }
    }
}

// rf = r64 / sigma (start of an FP32 run), sigma = |r64| given as its square in scal[0]
__global__ void k_start_rhs(long long n, const double* __restrict__ r64, const double* scal, double* sigma,
                            float* __restrict__ rf, float* __restrict__ y) {
    const double sg = sqrt(scal[0]);
    if (blockIdx.x == 0 && threadIdx.x == 0) *sigma = sg;
    const double inv = sg > 0 ? 1.0 / sg : 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        rf[i] = (float)(r64[i] * inv);
        y[i] = 0.f;
    }
}

// Residual replacement of the mixed solver (FP64 vectors, FP32 matrix in the iteration):
// r = b - (A D^-1) y with the FP64 matrix; rho' = (r0, r) and the next beta follow, so the
// iteration continues with its search direction (van der Vorst & Ye). |r| goes to S->rn.
template <bool C16 = false>
__global__ void __launch_bounds__(RB, 6) k_replace_residual(Sell<double> A, const double* __restrict__ b,
                                                            const double* __restrict__ y, double* __restrict__ r,
                                                            const double* __restrict__ r0, BcgScalars* S,
                                                            Partials P) {
    double arr = 0, ar0r = 0;
    SELL_LOOP(A) {
        double ay = sell_row<C16>(A, s, lane, y);
        long long i = (s << 5) + lane;
        if (i < A.n) {
            double ri = b[i] - ay;
            r[i] = ri;
            arr += ri * ri;
            ar0r += r0[i] * ri;
        }
    }
    if (block_partials(arr, ar0r, P, &S->counter[7])) {
        double rr, rho;
        final_sum(P, &rr, &rho);
        if (threadIdx.x == 0) {
            S->counter[7] = 0;
            S->rn = sqrt(rr);
            if (S->rn < S->best_rn) S->best_rn = S->rn;
            S->beta = (rho / S->rho0) * (S->alpha / S->omega);
            S->rho = rho;
            S->done = 0;
            S->s_conv = 0;
            if (!isfinite(rr)) { S->nonfinite = 1; S->done = 2; }
            else if (S->rn <= S->thresh) S->done = 1;
            else if (!isfinite(rho) || fabs(rho) < 1e-30) S->done = 2;
        }
    }
}

// |b|^2 into scal[0], fixed-order partials (once per learned solve)
__global__ void __launch_bounds__(RB) k_norm2(long long n, const double* __restrict__ b, double* scal, Partials P,
                                              unsigned int* counter) {
    double acc = 0;
    for (long long i = blockIdx.x * (long long)RB + threadIdx.x; i < n; i += (long long)gridDim.x * RB)
        acc += b[i] * b[i];
    if (block_partials(acc, 0.0, P, counter)) {
        double tot, unused;
        final_sum(P, &tot, &unused);
        if (threadIdx.x == 0) {
            *counter = 0;
            scal[0] = tot;
        }
    }
}

// network input b / |b| (FP32)
__global__ void k_rhs_unit(long long n, const double* __restrict__ b, float* __restrict__ rf, const double* scal) {
    const double inv = scal[0] > 0 ? 1.0 / sqrt(scal[0]) : 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        rf[i] = (float)(b[i] * inv);
}

// y0 = |b| net(b / |b|)
__global__ void k_y_from_net(long long n, const float* __restrict__ yf, const double* scal, double* __restrict__ y) {
    const double nb = sqrt(scal[0]);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] = nb * (double)yf[i];
}

// y += |r0| net(r0 / |r0|) (network correction of a warm start), keeping y in keep
__global__ void k_y_add_net(long long n, const float* __restrict__ yf, const double* scal, double* __restrict__ y,
                            double* __restrict__ keep) {
    const double nr = sqrt(scal[0]);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        keep[i] = y[i];
        y[i] += nr * (double)yf[i];
    }
}

// initial guess of the unknowns from a per-particle field (caller order): unknown u is
// particle perm[sorted_of_u[u]]
__global__ void k_guess_from_particles(long long U, const int* __restrict__ sorted_of_u, const int* __restrict__ perm,
                                       const double* __restrict__ pp, double* __restrict__ x) {
    for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < U; u += (long long)gridDim.x * blockDim.x)
        x[u] = pp[perm[sorted_of_u[u]]];
}

__global__ void k_fill_value(size_t n, double v, double* __restrict__ out) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) out[i] = v;
}

__global__ void k_solution_to_particles(long long U, const int* __restrict__ sorted_of_u, const int* __restrict__ perm,
                                        const double* __restrict__ x, double* __restrict__ pp) {
    for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < U; u += (long long)gridDim.x * blockDim.x)
        pp[perm[sorted_of_u[u]]] = x[u];
}

// ---------------------------------------------------------------------------------------
// host side of the engine
// ---------------------------------------------------------------------------------------
struct Engine {
    lsmps_ctx* ctx;
    cudaStream_t s;
    BcgScalars* S;
    Partials P;
};

template <class T>
struct Vecs {
    T *x, *r, *r0, *p, *v, *s, *t;
    T *ph = nullptr, *sh = nullptr;  // preconditioned directions M p, M s (multigrid)
};

Engine make_engine(lsmps_ctx* ctx) {
    Engine E{ctx, ctx->stream, nullptr, {}};
    double* red = ctx->red.ensure<double>(2 * RGRID + 256);
    E.P = Partials{red, red + RGRID};
    E.S = reinterpret_cast<BcgScalars*>(red + 2 * RGRID);
    return E;
}

double* engine_scalars(lsmps_ctx* ctx) { return ctx->red.get<double>() + 2 * RGRID + 128; }

static_assert(sizeof(BcgScalars) <= 128 * sizeof(double), "engine scalar layout");

// One BiCGStab iteration (MIXED_F32)
template <class T>
void iteration(Engine& E, const Sell<T>& A, const Vecs<T>& V) {
    note_launches(5);
    launch_pdl(k_bcg_p<T>, RGRID, RB, 0, E.s, A.n, V.r, V.p, V.v, E.S);
    if (A.dcol) launch_pdl(k_bcg_v<T, T, true>, spmv_grid<T, true>(), RB, 0, E.s, A, V.p, V.v, V.r0, E.S, E.P);
    else launch_pdl(k_bcg_v<T, T, false>, RGRID, RB, 0, E.s, A, V.p, V.v, V.r0, E.S, E.P);
    launch_pdl(k_bcg_s<T>, RGRID, RB, 0, E.s, A.n, V.r, V.v, V.s, E.S, E.P);
    if (A.dcol) launch_pdl(k_bcg_t<T, T, true>, spmv_grid<T, true>(), RB, 0, E.s, A, V.s, V.t, E.S, E.P, V.s);
    else launch_pdl(k_bcg_t<T, T, false>, RGRID, RB, 0, E.s, A, V.s, V.t, E.S, E.P, V.s);
    launch_pdl(k_bcg_x<T, false>, RGRID, RB, 0, E.s, A.n, V.x, V.r, V.p, V.s, V.t, V.r0, E.S, E.P, (const T*)nullptr,
               (const T*)nullptr);
}

// One iteration with the multigrid V-cycle as the right preconditioner: p (and s) and its
// level-1 restriction in one pass, the rest of the V-cycle, then the row product.
void iteration_mg(Engine& E, const Sell<float>& A, const Vecs<double>& V) {
    note_launches(5);
    const MgFine G = mg_fine(E.ctx);
    launch_pdl(k_bcg_p_agg, agg_blocks(G.n1), RB, 0, E.s, G, V.r, V.p, V.v, E.S);
    mg_apply(E.ctx, V.p, V.ph, E.S, 0, true);
    if (A.dcol) launch_pdl(k_bcg_v<double, float, true>, spmv_grid<float, true>(), RB, 0, E.s, A, V.ph, V.v, V.r0, E.S, E.P);
    else launch_pdl(k_bcg_v<double, float, false>, RGRID, RB, 0, E.s, A, V.ph, V.v, V.r0, E.S, E.P);
    launch_pdl(k_bcg_s_agg, std::min<unsigned>(RGRID, agg_blocks(G.n1)), RB, 0, E.s, G, V.r, V.v, V.s, E.S, E.P);
    mg_apply(E.ctx, V.s, V.sh, E.S, 1, true);
    if (A.dcol) launch_pdl(k_bcg_t<double, float, true>, spmv_grid<float, true>(), RB, 0, E.s, A, V.sh, V.t, E.S, E.P, V.s);
    else launch_pdl(k_bcg_t<double, float, false>, RGRID, RB, 0, E.s, A, V.sh, V.t, E.S, E.P, V.s);
    launch_pdl(k_bcg_x<double, true>, RGRID, RB, 0, E.s, A.n, V.x, V.r, V.p, V.s, V.t, V.r0, E.S, E.P, V.ph, V.sh);
}

template <class T, class TM = T>
void init(Engine& E, const Sell<TM>& A, const T* b, const Vecs<T>& V, bool use_x, double tol, double bnorm_override) {
    if (A.dcol)
        k_bcg_init<T, TM, true><<<RGRID, RB, 0, E.s>>>(A, b, V.x, use_x, V.r, V.r0, V.p, V.v, E.S, E.P, tol,
                                                       bnorm_override);
    else
        k_bcg_init<T, TM, false><<<RGRID, RB, 0, E.s>>>(A, b, V.x, use_x, V.r, V.r0, V.p, V.v, E.S, E.P, tol,
                                                        bnorm_override);
    LSMPS_CHECK_LAUNCH();
}

// the mixed solver's FP64 residual replacement
void launch_replace(cudaStream_t s, const Sell<double>& As, const double* b, const Vecs<double>& V, Engine& E) {
    if (As.dcol) k_replace_residual<true><<<RGRID, RB, 0, s>>>(As, b, V.x, V.r, V.r0, E.S, E.P);
    else k_replace_residual<false><<<RGRID, RB, 0, s>>>(As, b, V.x, V.r, V.r0, E.S, E.P);
    LSMPS_CHECK_LAUNCH();
}

void residual64(Engine& E, const Sell<double>& A, const double* b, const double* x, double* r, double* out2) {
    if (A.dcol) k_residual64<true><<<RGRID, RB, 0, E.s>>>(A, b, x, r, out2, E.P, &E.S->counter[5]);
    else k_residual64<false><<<RGRID, RB, 0, E.s>>>(A, b, x, r, out2, E.P, &E.S->counter[5]);
    LSMPS_CHECK_LAUNCH();
}

void set_scalar_caps(Engine& E, int max_iter, int stall_window) {
    BcgScalars init{};
    init.max_iter = max_iter;
    init.stall_window = stall_window;
    LSMPS_CUDA(cudaMemcpyAsync(E.S, &init, sizeof(init), cudaMemcpyHostToDevice, E.s));
}

// Entries of a slice that k_sell_build stages: a third more than the mean slice has, so that only
// slices of unusually long rows are read in place and the others leave room for more blocks (half
// as much again: 207 against 196 us at 911k unknowns).
static int sell_stage_cap(lsmps_ctx* ctx) {
    const long long mean = 32 * (ctx->nnz / std::max(ctx->U, 1LL) + 1);
    return (int)std::min<long long>(SB_MAX, (mean + mean / 3 + 127) / 128 * 128);
}

}  // namespace

// ---------------------------------------------------------------------------------------
// ---- SELL-32 copies of the assembled matrix (built on first use after an assembly) ----
static void sell_raw(lsmps_ctx* ctx);
// kind 0: A (FP64), 1: A D^-1 (FP64), 2: A D^-1 (FP32)
static void sell_structure(lsmps_ctx* ctx) {
    if (ctx->have_sell) return;
    cudaStream_t s = ctx->stream;
    const long long U = ctx->U;
    const long long ns = (U + 31) / 32;
    int* slen = ctx->S_len.ensure<int>(ns + 1);
    int* ssize = ctx->vtmp.ensure<int>(ns + 1);
    int* sptr = ctx->S_ptr.ensure<int>(ns + 1);
    if (ns) {
        k_sell_len<<<blocks_for(ns * 32, 256), 256, 0, s>>>(U, ns, ctx->A_row.get<int>(), slen, ssize);
        LSMPS_CHECK_LAUNCH();
    }
    scan_exclusive<int>(ssize, sptr, ns, s, ctx->scan_tmp, ctx->dflags.get<int>());
    int total = 0;
    read_back(ctx, {{sptr + ns, &total, sizeof(int)}}, "SELL layout");
    ctx->sell_nslices = ns;
    ctx->sell_entries = total;
    int* col = ctx->S_col.ensure<int>((size_t)total + 8);
    double* val = ctx->S_val.ensure<double>((size_t)total + 8);
    double* vals = ctx->S_vals.ensure<double>((size_t)total + 8);
    float* valf = ctx->S_valf.ensure<float>((size_t)total + 8);
    unsigned short* dcol = ctx->S_dcol.ensure<unsigned short>((size_t)total + 8);
    int* rbase = ctx->S_rbase.ensure<int>(ns * 32 + 1);
    ctx->have_steps = false;
    if (ns) {
        int* bad = ctx->scratch.get<int>() + 46;
        const int cap = sell_stage_cap(ctx);
        LSMPS_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), s));
        k_sell_build<<<(unsigned)ns, 32 * SB_WARPS, cap * 12, s>>>(U, ctx->A_row.get<int>(), ctx->A_col.get<int>(),
                                                              ctx->A_val.get<double>(), ctx->A_dinv.get<double>(), sptr,
                                                              slen, col, val, dcol, rbase, vals, valf, bad, 0, cap);
        LSMPS_CHECK_LAUNCH();
        int hbad = 1;
        read_back(ctx, {{bad, &hbad, sizeof(int)}}, nullptr);
        ctx->have_steps = hbad == 0 && ctx->sell_steps_enabled;
    }
    ctx->have_sell_s = ctx->have_sell_f = true;  // the scaled copies come with the structure
    ctx->have_sell = true;
    ctx->have_sell_raw = ns == 0;
    if (!ctx->have_steps) sell_raw(ctx);  // every view then reads the 32-bit columns
}

// The unscaled FP64 values and 32-bit columns (the plain FP64 solver's matrix, and the columns
// of every view when the copies have no 16-bit steps): the same build again, writing them too.
static void sell_raw(lsmps_ctx* ctx) {
    if (ctx->have_sell_raw) return;
    const long long U = ctx->U, ns = ctx->sell_nslices;
    if (ns) {
        int* bad = ctx->scratch.get<int>() + 46;
        const int cap = sell_stage_cap(ctx);
        k_sell_build<<<(unsigned)ns, 32 * SB_WARPS, cap * 12, ctx->stream>>>(
            U, ctx->A_row.get<int>(), ctx->A_col.get<int>(), ctx->A_val.get<double>(), ctx->A_dinv.get<double>(),
            ctx->S_ptr.get<int>(), ctx->S_len.get<int>(), ctx->S_col.get<int>(), ctx->S_val.get<double>(),
            ctx->S_dcol.get<unsigned short>(), ctx->S_rbase.get<int>(), ctx->S_vals.get<double>(),
            ctx->S_valf.get<float>(), bad, 1, cap);
        LSMPS_CHECK_LAUNCH();
    }
    ctx->have_sell_raw = true;
}

template <class T>
static const int* sell_cuts(lsmps_ctx* ctx, const Sell<T>& A) {
    const unsigned blocks = krylov_blocks(ctx, A.nslices);
    int* cut = ctx->S_cut.ensure<int>(blocks + 1);
    k_sell_cuts<<<1, 256, 0, ctx->stream>>>(A, blocks, cut);
    LSMPS_CHECK_LAUNCH();
    return cut;
}

template <class T>
static Sell<T> sell_view(lsmps_ctx* ctx, const T* val) {
    Sell<T> A{ctx->U, ctx->sell_nslices, ctx->S_ptr.get<int>(), ctx->S_len.get<int>(), ctx->S_col.get<int>(), val};
    if (ctx->have_steps) {
        A.dcol = ctx->S_dcol.get<unsigned short>();
        A.rbase = ctx->S_rbase.get<int>();
    }
    return A;
}

static Sell<double> sell_a64(lsmps_ctx* ctx) {
    sell_structure(ctx);
    sell_raw(ctx);
    return sell_view<double>(ctx, ctx->S_val.get<double>());
}

Sell<double> sell_a64_view(lsmps_ctx* ctx) { return sell_a64(ctx); }

static Sell<double> sell_scaled64(lsmps_ctx* ctx) {  // A D^-1 in FP64 (built with the structure)
    sell_structure(ctx);
    return sell_view<double>(ctx, ctx->S_vals.get<double>());
}

static Sell<float> sell_scaled32(lsmps_ctx* ctx) {  // A D^-1 in FP32 (built with the structure)
    sell_structure(ctx);
    return sell_view<float>(ctx, ctx->S_valf.get<float>());
}

Sell<float> sell_scaled32_view(lsmps_ctx* ctx) { return sell_scaled32(ctx); }

static KrylovVecs krylov_vecs(lsmps_ctx* ctx) {
    const long long U = ctx->U;
    KrylovVecs V{ctx->vx.ensure<double>(U + 2), ctx->vr.ensure<double>(U + 2), ctx->vr0.ensure<double>(U + 2),
                 ctx->vp.ensure<double>(U + 2), ctx->vv.ensure<double>(U + 2), ctx->vs.ensure<double>(U + 2),
                 ctx->vt.ensure<double>(U + 2)};
    V.b = ctx->A_b.get<double>();
    return V;
}

static void krylov_stats(lsmps_ctx* ctx, const KrylovResult& h, lsmps_ppe_stats* ps) {
    double mx;
    std::memcpy(&mx, &h.maxbits, sizeof(mx));
    ps->iterations = h.iterations;
    ps->outer_iterations = h.outer;
    ps->converged = h.converged && !h.nonfinite;
    ps->fallback = h.fallback;
    ps->max_error = mx;
    ps->relative_l2_error = std::sqrt(h.err2 / std::max(h.ref2, 1e-30));
    ps->solve_ms = ev_elapsed(ctx, 10, 11);
}

// Fast FP64 / Jacobi: BiCGStab on A (or A D^-1) in FP64.
static void solve_fast64(lsmps_ctx* ctx, const lsmps_solver_opts* o, lsmps_ppe_stats* ps, bool jacobi) {
    const long long U = ctx->U;
    const bool warm = o->warm_start && ctx->have_solution;
    ev_record(ctx, 10);
    const KrylovVecs V = krylov_vecs(ctx);
    const Sell<double> A = jacobi ? sell_scaled64(ctx) : sell_a64(ctx);
    const double* dinv = ctx->A_dinv.get<double>();
    ctx->have_solution = false;  // until the solve has succeeded: x is overwritten from here on
    if (warm && jacobi) {  // the iteration works on y = D x
        k_scale_by_diag<<<1184, 256, 0, ctx->stream>>>(U, V.x, dinv);
        LSMPS_CHECK_LAUNCH();
    }
    KrylovOpts k;
    k.tol = o->tol;
    k.chunk = std::max(1, o->check_every > 0 ? o->check_every : 8);
    k.max_iter = o->max_iter;
    k.use_x = warm;
    k.dinv = jacobi ? dinv : nullptr;
    k.xe = ctx->A_xexact.get<double>();
    krylov_stats(ctx, krylov_solve(ctx, nullptr, A, V, k), ps);
}

// Mixed precision with FP32 vectors (MIXED_F32). One FP32 Jacobi-BiCGStab on A D^-1 y = r0 / sigma (sigma =
// |r0|, so FP32 values start at O(1)) accumulates y_lo; whenever its recursive residual has
// dropped by a factor `inner_tol` since the last update (checked every `check_every`
// iterations), a reliable update folds y_lo into the FP64 solution x_hi, recomputes the
// true residual b - A x_hi with the FP64 matrix, and replaces the FP32 residual with it,
// keeping the search direction. Convergence is always decided on the FP64 residual. A
// breakdown, a stall (LEARNED: no 1 % progress in `stall_window` iterations) or an FP32
// residual that claims convergence the FP64 one does not confirm restarts the Krylov space
// from the true residual; LEARNED starts the first run from the network's guess and, after
// a stall, continues as plain Jacobi-BiCGStab (fallback).
static void solve_mixed_f32(lsmps_ctx* ctx, const lsmps_solver_opts* o, lsmps_ppe_stats* ps, bool learned) {
    cudaStream_t s = ctx->stream;
    long long U = ctx->U;
    Engine E = make_engine(ctx);
    double* scal = engine_scalars(ctx);  // [0] |r|^2, [1] |b|^2, [6] sigma
    double* sigma = scal + 6;
    const double* dinv = ctx->A_dinv.get<double>();
    double* x = ctx->vx.ensure<double>(U + 2);
    double* r64 = ctx->vr.ensure<double>(U + 1);
    float* rhs = ctx->fph.ensure<float>(U + 1);
    Vecs<float> V{ctx->fx.ensure<float>(U + 1), ctx->fr.ensure<float>(U + 1), ctx->fr0.ensure<float>(U + 1),
                  ctx->fp.ensure<float>(U + 1), ctx->fv.ensure<float>(U + 1), ctx->fs.ensure<float>(U + 1),
                  ctx->ft.ensure<float>(U + 1)};
    const bool use_nn = learned && mpnn_ready(ctx);
    const bool warm = o->warm_start && ctx->have_solution;
    const double delta = o->inner_tol > 0 ? o->inner_tol : 0.1;  // residual drop between updates
    const int chunk = std::max(1, o->check_every > 0 ? o->check_every : 8);
    const int stall = o->stall_window > 0 ? o->stall_window : 20;
    ev_record(ctx, 10);
    Sell<double> A = sell_a64(ctx);
    Sell<float> Af = sell_scaled32(ctx);
    set_scalar_caps(E, 0, 0);  // zero the reduction tickets
    ctx->have_solution = false;  // until the solve has succeeded: x is overwritten from here on
    if (!warm) LSMPS_CUDA(cudaMemsetAsync(x, 0, U * sizeof(double), s));
    auto true_residual = [&]() {
        residual64(E, A, ctx->A_b.get<double>(), x, r64, scal);
        double h2[2];
        LSMPS_CUDA(cudaMemcpyAsync(h2, scal, sizeof(h2), cudaMemcpyDeviceToHost, s));
        LSMPS_CUDA(cudaStreamSynchronize(s));
        return std::make_pair(std::sqrt(h2[0]), std::sqrt(h2[1]));
    };
    auto [rnorm, bnorm] = true_residual();
    const double thresh = o->tol * std::max(1.0, bnorm);
    int total = 0, runs = 0, updates = 0, fallback = 0;
    bool converged = rnorm <= thresh;
    bool nonfinite = !std::isfinite(rnorm);
    cudaGraphExec_t exec = nullptr;
    auto read_scalars = [&](BcgScalars& h) {
        LSMPS_CUDA(cudaMemcpyAsync(&h, E.S, sizeof(h), cudaMemcpyDeviceToHost, s));
        LSMPS_CUDA(cudaStreamSynchronize(s));
    };
    while (!converged && !nonfinite && total < o->max_iter) {
        // ---- an FP32 run from the true residual: sigma = |r|, rhs = r / sigma ----
        k_start_rhs<<<1184, 256, 0, s>>>(U, r64, scal, sigma, rhs, V.x);
        LSMPS_CHECK_LAUNCH();
        const bool nn_now = use_nn && !fallback && runs == 0;
        if (nn_now) mpnn_warm_start(ctx, rhs, V.x);
        set_scalar_caps(E, o->max_iter - total, nn_now ? stall : 0);
        // FP32 threshold in the scaled system's units: |r| / sigma <= thresh / sigma
        init<float>(E, Af, rhs, V, nn_now, thresh / std::max(rnorm, 1e-300), 1.0);
        ++runs;
        if (!exec && o->use_graph) {
            cudaGraph_t graph;
            LSMPS_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
            for (int c = 0; c < chunk; ++c) iteration<float>(E, Af, V);
            note_launches(0 - (uint64_t)(5 * chunk));  // captured, not launched
            cudaError_t e = cudaStreamEndCapture(s, &graph);
            LSMPS_CUDA(e);
            LSMPS_CUDA(cudaGraphInstantiate(&exec, graph, 0));
            cudaGraphDestroy(graph);
        }
        BcgScalars h{};
        read_scalars(h);
        double rn_upd = h.rn;  // FP32 residual at the last update of this run
        int run_base = 0;      // iterations of this run already counted
        while (true) {
            if (!h.done) {
                if (exec) {
                    LSMPS_CUDA(cudaGraphLaunch(exec, s));
                    note_launches(5 * (uint64_t)chunk);
                } else {
                    for (int k = 0; k < chunk; ++k) iteration<float>(E, Af, V);
                    LSMPS_CHECK_LAUNCH();
                }
                read_scalars(h);
            }
            total += h.iters - run_base;
            run_base = h.iters;
            if (!h.done && h.rn > delta * rn_upd) continue;
            // ---- reliable update: fold y_lo into x_hi, true FP64 residual ----
            k_reliable_x<<<1184, 256, 0, s>>>(U, x, V.x, dinv, sigma);
            LSMPS_CHECK_LAUNCH();
            std::tie(rnorm, bnorm) = true_residual();
            ++updates;
            if (!std::isfinite(rnorm)) { nonfinite = true; break; }
            if (rnorm <= thresh) { converged = true; break; }
            if (total >= o->max_iter || h.done == 3) break;
            if (h.done) {  // breakdown, stall, or an FP32 convergence the FP64 residual denies
                if (h.done == 4 && nn_now) fallback = 1;
                break;     // restart from the true residual
            }
            k_reliable_r<<<RGRID, RB, 0, s>>>(U, r64, sigma, V.r, V.r0, E.S, E.P);
            LSMPS_CHECK_LAUNCH();
            read_scalars(h);
            rn_upd = h.rn;
            if (h.done) break;  // rho breakdown after the replacement: restart
        }
        if (h.done == 3) break;
    }
    if (exec) cudaGraphExecDestroy(exec);
    ev_record(ctx, 11);
    LSMPS_CUDA(cudaStreamSynchronize(s));
    ps->iterations = total;
    ps->outer_iterations = updates;
    ps->converged = converged && !nonfinite;
    ps->fallback = fallback;
    ps->solve_ms = ev_elapsed(ctx, 10, 11);
}

// The multigrid hierarchy set-up on the context's side stream (created at first use with the
// device's highest priority), ordered after everything the context stream held when `fork`
// was recorded; the context stream then waits for it. The set-up reads each level's size back
// to the host, so work queued on the context stream meanwhile (the network's inference) fills
// the GPU during those round trips, and the set-up's kernels take the SMs first when both wait.
static void mg_setup_on_side(lsmps_ctx* ctx) {
    cudaStream_t main = ctx->stream;
    LSMPS_CUDA(cudaStreamWaitEvent(ctx->side_stream, ctx->side_fork, 0));
    ctx->stream = ctx->side_stream;
    try {
        mg_setup(ctx);
    } catch (...) {
        ctx->stream = main;
        cudaStreamSynchronize(ctx->side_stream);
        throw;
    }
    ctx->stream = main;
    LSMPS_CUDA(cudaEventRecord(ctx->side_join, ctx->side_stream));
    LSMPS_CUDA(cudaStreamWaitEvent(main, ctx->side_join, 0));
}

static void side_stream_fork(lsmps_ctx* ctx) {
    if (!ctx->side_stream) {
        int least = 0, greatest = 0;
        LSMPS_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
        LSMPS_CUDA(cudaStreamCreateWithPriority(&ctx->side_stream, cudaStreamNonBlocking, greatest));
        LSMPS_CUDA(cudaEventCreateWithFlags(&ctx->side_fork, cudaEventDisableTiming));
        LSMPS_CUDA(cudaEventCreateWithFlags(&ctx->side_join, cudaEventDisableTiming));
    }
    LSMPS_CUDA(cudaEventRecord(ctx->side_fork, ctx->stream));
}

// Mixed precision (MIXED, and LEARNED): Jacobi-BiCGStab with FP64 vectors and recurrences
// whose two SpMVs per iteration read the FP32 copy of A D^-1 (8 bytes per entry instead
// of 12: the matrix is the bandwidth). The FP32 matrix perturbs each product at ~6e-8
// relative, so the recursive residual drifts from the true one; whenever it has fallen by
// `inner_tol` (default 0.01: measured best on the 1M WLS system) since the last replacement, or the iteration stops, the true
// residual b - A D^-1 y is recomputed with the FP64 matrix and replaces it, keeping the
// search direction. Convergence is decided on that FP64 residual only. A breakdown, a
// stall (LEARNED: no 1 % progress in `stall_window` iterations) or an FP32-driven
// convergence claim the FP64 residual denies restarts the Krylov space from the current
// iterate; LEARNED starts from the network's guess and, after a stall, continues as plain
// Jacobi-BiCGStab (fallback). With the multigrid preconditioner a stall (no 1 % progress in
// `stall_window` iterations) or a breakdown ends the multigrid phase, and the solve continues
// as Jacobi MIXED from the current iterate (from zero when it is no longer finite; fallback).
// exit_res: {|b - A D^-1 y|, |b|} of the returned iterate when the solve converged (the
// convergence test's own FP64 residual), else {-1, -1}. Returns whether ps holds the error
// against p*. The Jacobi solves run in krylov.cu's one launch; the multigrid's launch the
// iteration's kernels from the host (2 x 9 + 5 of them with four coarse levels), each under programmatic dependent launch
// (the same steps between the grid barriers of one launch measured 370-400 against 303 us per
// iteration at 1M: one block of 1,024 threads per SM hides less of the V-cycle's dependent
// loads than the kernels' 2,048 threads, and its shared memory takes the L1 from the row products).
static bool solve_mixed(lsmps_ctx* ctx, const lsmps_solver_opts* o, lsmps_ppe_stats* ps, bool learned,
                        double* exit_res) {
    cudaStream_t s = ctx->stream;
    const long long U = ctx->U;
    const double* dinv = ctx->A_dinv.get<double>();
    const double* b = ctx->A_b.get<double>();
    const bool use_nn = learned && mpnn_ready(ctx);
    const bool warm = o->warm_start && ctx->have_solution;
    const bool mg = o->precond == LSMPS_PRECOND_MULTIGRID;
    const int stall = o->stall_window > 0 ? o->stall_window : 20;
    ev_record(ctx, 10);
    const KrylovVecs K = krylov_vecs(ctx);
    Vecs<double> V{K.x, K.r, K.r0, K.p, K.v, K.s, K.t};
    Engine E = make_engine(ctx);
    double* scal = engine_scalars(ctx);
    if (use_nn) set_scalar_caps(E, 0, 0);  // zeroes the reduction tickets of the kernels below
    // y0 = |b| net(b / |b|): launches only (no host round trip)
    auto net_guess = [&] {
        float* rhs = ctx->fph.ensure<float>(U + 1);
        float* yf = ctx->fx.ensure<float>(U + 1);
        k_norm2<<<RGRID, RB, 0, s>>>(U, b, scal, E.P, &E.S->counter[5]);
        k_rhs_unit<<<1184, 256, 0, s>>>(U, b, rhs, scal);  // network input: b / |b| in FP32
        LSMPS_CHECK_LAUNCH();
        mpnn_warm_start(ctx, rhs, yf);
        k_y_from_net<<<1184, 256, 0, s>>>(U, yf, scal, V.x);
        LSMPS_CHECK_LAUNCH();
    };
    // LEARNED with the multigrid from a cold start: the network's guess (context stream) and
    // the hierarchy set-up (side stream) run at the same time; they read the assembled system
    // and write disjoint buffers
    const bool overlap = mg && use_nn && !warm;
    if (mg) {
        if (overlap) {
            side_stream_fork(ctx);
            ctx->have_solution = false;  // as below
            net_guess();
            mg_setup_on_side(ctx);
        } else {
            mg_setup(ctx);
        }
        V.ph = ctx->vph.ensure<double>(U + 1);
        V.sh = ctx->vsh.ensure<double>(U + 1);
    }
    const Sell<double> As = sell_scaled64(ctx);
    const Sell<float> Af = sell_scaled32(ctx);
    KrylovOpts ko;
    ko.tol = o->tol;
    ko.delta = o->inner_tol > 0 ? o->inner_tol : 0.01;
    ko.chunk = std::max(1, o->check_every > 0 ? o->check_every : 8);
    ko.max_iter = o->max_iter;
    ko.max_chunks = (long long)o->max_iter / ko.chunk + 4 + o->max_iter;
    ko.stall = stall;
    ko.use_x = warm || use_nn;
    ko.use_nn = use_nn;
    ko.dinv = dinv;
    ko.xe = ctx->A_xexact.get<double>();
    ctx->have_solution = false;  // until the solve has succeeded: x is overwritten from here on
    if (warm) {  // the iteration works on y = D x
        k_scale_by_diag<<<1184, 256, 0, s>>>(U, V.x, dinv);
        LSMPS_CHECK_LAUNCH();
        if (use_nn) {  // the network corrects the warm start: y += |r0| net(r0 / |r0|), r0 = b - A D^-1 y
            float* rhs = ctx->fph.ensure<float>(U + 1);
            float* yf = ctx->fx.ensure<float>(U + 1);
            residual64(E, As, b, V.x, V.r, scal);
            k_rhs_unit<<<1184, 256, 0, s>>>(U, V.r, rhs, scal);
            LSMPS_CHECK_LAUNCH();
            mpnn_warm_start(ctx, rhs, yf);
            k_y_add_net<<<1184, 256, 0, s>>>(U, yf, scal, V.x, V.s);  // the warm start kept in s
            LSMPS_CHECK_LAUNCH();
            ko.warm_rn2 = scal;
        }
    } else if (use_nn && !overlap) {
        net_guess();
    }
    exit_res[0] = exit_res[1] = -1.0;
    auto finish = [&](const KrylovResult& h) {
        krylov_stats(ctx, h, ps);
        // convergence is only declared right after a residual replacement or a (re)start, whose
        // FP64 residual b - A D^-1 y of the final iterate h holds
        if (h.converged && std::isfinite(h.rn)) {
            exit_res[0] = h.rn;
            exit_res[1] = h.bnorm;
        }
        return true;
    };
    if (!mg) {
        KrylovVecs W = K;
        W.keep = V.s;
        return finish(krylov_solve(ctx, &Af, As, W, ko));
    }
    set_scalar_caps(E, o->max_iter, stall);
    if (!ko.use_x) LSMPS_CUDA(cudaMemsetAsync(V.x, 0, U * sizeof(double), s));
    init<double, double>(E, As, b, V, ko.use_x != 0, o->tol, -1.0);
    BcgScalars h{};
    double warm_rn2 = 0;  // |b - A x0|^2 of a warm start the network corrected
    auto read = [&] { read_back(ctx, {{E.S, &h, sizeof(h)}}, nullptr); };
    read_back(ctx, {{E.S, &h, sizeof(h)}, {scal, &warm_rn2, sizeof(warm_rn2)}}, nullptr);
    int total = 0, replacements = 0, restarts = 0, fallback = 0;
    if (use_nn && (!std::isfinite(h.rn) || h.rn >= (warm ? std::sqrt(warm_rn2) : h.bnorm))) {
        // the network's guess is worse than zero (its correction than the warm start): discard it
        fallback = 1;
        if (warm) LSMPS_CUDA(cudaMemcpyAsync(V.x, V.s, U * sizeof(double), cudaMemcpyDeviceToDevice, s));
        else LSMPS_CUDA(cudaMemsetAsync(V.x, 0, U * sizeof(double), s));
        set_scalar_caps(E, o->max_iter, stall);
        init<double, double>(E, As, b, V, warm, o->tol, -1.0);
        read();
    }
    // iterates until converged, failed or the iteration cap, or until the multigrid breaks down
    // or stalls (give_up)
    bool converged = h.done == 1, failed = h.done == 2 && h.nonfinite, give_up = false;
    double rn_upd = h.rn;
    int base = h.iters;
    for (long long guard = 0; !converged && !failed && guard < ko.max_chunks; ++guard) {
        if (!h.done) {
            for (int k = 0; k < ko.chunk; ++k) iteration_mg(E, Af, V);
            LSMPS_CHECK_LAUNCH();
            read();
        }
        total += h.iters - base;
        base = h.iters;
        if (!h.done && h.rn > ko.delta * rn_upd) continue;
        const int why = h.done;  // 0: drop by delta; else the iteration stopped
        if (why == 3 || total >= o->max_iter) {
            // iteration cap: report the true residual of the last iterate
            launch_replace(s, As, b, V, E);
            read();
            converged = h.done == 1;
            break;
        }
        if (why == 0) {
            launch_replace(s, As, b, V, E);
            ++replacements;
            read();
            rn_upd = h.rn;
            if (h.done == 1) { converged = true; break; }
            if (h.done == 0) continue;
            // rho breakdown after the replacement: fall through
        }
        if (h.done == 2 || h.done == 4) { give_up = true; break; }
        if (h.nonfinite) { failed = true; break; }
        // restart from the current iterate with the FP64 matrix (true residual)
        set_scalar_caps(E, o->max_iter - total, stall);
        init<double, double>(E, As, b, V, true, o->tol, -1.0);
        ++restarts;
        read();
        base = 0;
        rn_upd = h.rn;
        if (h.done == 1) { converged = true; break; }
        if (h.done) { failed = true; break; }
    }
    if (give_up) {
        // The multigrid broke down or stalled (near-singular aggregates can do this): continue
        // as Jacobi MIXED from the current iterate, or from zero if it is no longer finite.
        ko.use_nn = 0;
        ko.warm_rn2 = nullptr;
        ko.use_x = !h.nonfinite;
        ko.max_iter = o->max_iter - total;
        KrylovResult k = krylov_solve(ctx, &Af, As, K, ko);
        k.iterations += total;
        k.outer += replacements + restarts + 1;
        k.fallback = 1;
        return finish(k);
    }
    k_unscale<<<1184, 256, 0, s>>>(U, V.x, dinv);
    LSMPS_CHECK_LAUNCH();
    ev_record(ctx, 11);
    ps->iterations = total;
    ps->outer_iterations = replacements + restarts;
    ps->converged = converged;
    ps->fallback = fallback;
    ps->solve_ms = ev_elapsed(ctx, 10, 11);
    if (converged && std::isfinite(h.rn)) {
        exit_res[0] = h.rn;
        exit_res[1] = h.bnorm;
    }
    return false;
}

void ppe_set_initial_particles(lsmps_ctx* ctx, const double* pp, size_t n, bool device) {
    LSMPS_REQUIRE(ctx->have_ppe && !ctx->ppe_loaded, LSMPS_ERR_STATE,
                  "per-particle initial guesses need an assembled particle system");
    LSMPS_REQUIRE(n == ctx->n && (n == 0 || pp), LSMPS_ERR_ARG, "initial guess must hold one value per particle");
    cudaStream_t s = ctx->stream;
    const long long U = ctx->U;
    double* x = ctx->vx.ensure<double>(U + 2);
    const double* src = pp;
    if (!device && n) {
        double* tmp = ctx->vtmp.ensure<double>(n + 1);
        LSMPS_CUDA(cudaMemcpyAsync(tmp, pp, n * sizeof(double), cudaMemcpyHostToDevice, s));
        src = tmp;
    }
    if (U) {
        k_guess_from_particles<<<1184, 256, 0, s>>>(U, ctx->sorted_of_u.get<int>(), ctx->perm.get<int>(), src, x);
        LSMPS_CHECK_LAUNCH();
    }
    LSMPS_CUDA(cudaStreamSynchronize(s));
    ctx->have_solution = true;
}

void ppe_pressure_particles(lsmps_ctx* ctx, double* pp, size_t n, double fill, bool device) {
    LSMPS_REQUIRE(ctx->have_solution, LSMPS_ERR_STATE, "no solution: lsmps_ppe_solve first");
    LSMPS_REQUIRE(!ctx->ppe_loaded, LSMPS_ERR_STATE, "per-particle pressure needs an assembled particle system");
    LSMPS_REQUIRE(n == ctx->n && (n == 0 || pp), LSMPS_ERR_ARG, "output must hold one value per particle");
    cudaStream_t s = ctx->stream;
    const long long U = ctx->U;
    double* dst = device ? pp : ctx->vtmp.ensure<double>(n + 1);
    if (n && std::isnan(fill)) {  // keep the other particles' values
        if (!device) LSMPS_CUDA(cudaMemcpyAsync(dst, pp, n * sizeof(double), cudaMemcpyHostToDevice, s));
    } else if (n) {
        k_fill_value<<<std::min<unsigned>(blocks_for(n, 256), 1184), 256, 0, s>>>(n, fill, dst);
        LSMPS_CHECK_LAUNCH();
    }
    if (U) {
        k_solution_to_particles<<<1184, 256, 0, s>>>(U, ctx->sorted_of_u.get<int>(), ctx->perm.get<int>(),
                                                     ctx->vx.get<double>(), dst);
        LSMPS_CHECK_LAUNCH();
    }
    if (!device && n) LSMPS_CUDA(cudaMemcpyAsync(pp, dst, n * sizeof(double), cudaMemcpyDeviceToHost, s));
    LSMPS_CUDA(cudaStreamSynchronize(s));
}

void ppe_solve(lsmps_ctx* ctx, const lsmps_solver_opts* o, lsmps_ppe_stats* out) {
    LSMPS_REQUIRE(ctx->have_ppe, LSMPS_ERR_STATE, "PPE solve needs lsmps_ppe_assemble first");
    LSMPS_REQUIRE(o && o->solver >= 0 && o->solver <= 5, LSMPS_ERR_ARG, "unknown solver");
    LSMPS_REQUIRE(o->solver != LSMPS_SOLVER_LEARNED || mpnn_ready(ctx), LSMPS_ERR_STATE,
                  "learned solver needs lsmps_mpnn_init / lsmps_mpnn_load first");
    LSMPS_REQUIRE(o->solver != LSMPS_SOLVER_LEARNED || !ctx->ppe_loaded, LSMPS_ERR_STATE,
                  "the learned solver needs an assembled particle system (its features are per particle)");
    LSMPS_REQUIRE(o->precond == LSMPS_PRECOND_JACOBI ||
                      (o->precond == LSMPS_PRECOND_MULTIGRID &&
                       (o->solver == LSMPS_SOLVER_MIXED || o->solver == LSMPS_SOLVER_LEARNED)),
                  LSMPS_ERR_ARG, "the multigrid preconditioner is for the MIXED and LEARNED solvers");
    LSMPS_REQUIRE(o->precond != LSMPS_PRECOND_MULTIGRID || !ctx->ppe_loaded, LSMPS_ERR_STATE,
                  "the multigrid preconditioner aggregates particle cells: a loaded CSR system has none");
    lsmps_ppe_stats ps = ctx->ppe_assembly;
    ps.iterations = 0;
    ps.converged = 0;
    long long U = ctx->U;
    if (U == 0) {  // src/lsmps.cpp:67: if(!n) return st;
        if (out) *out = ps;
        return;
    }
    if (o->solver == LSMPS_SOLVER_REFERENCE) {
        solve_exact(ctx, o, &ps);
    } else {
        double exit_res[2] = {-1.0, -1.0};
        bool have_error = true;
        if (o->solver == LSMPS_SOLVER_FP64) solve_fast64(ctx, o, &ps, false);
        else if (o->solver == LSMPS_SOLVER_JACOBI) solve_fast64(ctx, o, &ps, true);
        else if (o->solver == LSMPS_SOLVER_MIXED_F32) solve_mixed_f32(ctx, o, &ps, have_error = false);
        else have_error = solve_mixed(ctx, o, &ps, o->solver == LSMPS_SOLVER_LEARNED, exit_res);
        // final statistics in FP64: |Ax - b|, |b| (for a converged MIXED / LEARNED solve the
        // convergence test's own FP64 residual of the final iterate, |b - A D^-1 y| with
        // y = D x), error against p* (krylov.cu's solves bring their own)
        if (exit_res[0] < 0 || !have_error) {
            cudaStream_t s = ctx->stream;
            Engine E = make_engine(ctx);
            double* scal = engine_scalars(ctx);
            double* x = ctx->vx.get<double>();
            double* tmp = ctx->vt.ensure<double>(U + 2);
            auto* maxbits = reinterpret_cast<unsigned long long*>(scal + 4);
            set_scalar_caps(E, 0, 0);  // zeroes the reduction tickets
            if (exit_res[0] < 0) residual64(E, sell_a64(ctx), ctx->A_b.get<double>(), x, tmp, scal);
            LSMPS_CUDA(cudaMemsetAsync(maxbits, 0, sizeof(unsigned long long), s));
            if (!have_error) {
                k_error_stats<<<RGRID, RB, 0, s>>>(U, x, ctx->A_xexact.get<double>(), scal + 2, E.P, &E.S->counter[6],
                                                    maxbits);
                LSMPS_CHECK_LAUNCH();
            }
            double h[5];
            read_back(ctx, {{scal, h, sizeof(h)}}, nullptr);
            if (exit_res[0] < 0) {
                exit_res[0] = std::sqrt(h[0]);
                exit_res[1] = std::sqrt(h[1]);
            }
            if (!have_error) {
                ps.relative_l2_error = std::sqrt(h[2] / std::max(h[3], 1e-30));
                std::memcpy(&ps.max_error, &h[4], sizeof(double));
            }
        }
        ps.initial_residual = exit_res[1];
        ps.final_residual = exit_res[0];
        ps.relative_residual = ps.final_residual / std::max(ps.initial_residual, 1e-300);
        if (!std::isfinite(ps.final_residual)) ps.converged = 0;
    }
    ctx->have_solution = true;
    ctx->timings[5] = ps.solve_ms;
    if (out) *out = ps;
}

// The solver's SpMV as the iterations run it: LSMPS_KB_SPMV32 is the MIXED solver's kernel
// (FP32 A D^-1 values, FP64 vectors), LSMPS_KB_SPMV64 the plain FP64 solver's (FP64 A).
void solver_kernel_bench(lsmps_ctx* ctx, int kernel, int reps, double* ms, double* bytes) {
    LSMPS_REQUIRE(ctx->have_ppe, LSMPS_ERR_STATE, "SpMV bench needs an assembled PPE");
    cudaStream_t s = ctx->stream;
    const long long U = ctx->U;
    const bool f32 = kernel == LSMPS_KB_SPMV32;
    double* x = ctx->vp.ensure<double>(U + 1);
    double* r0 = ctx->vr0.ensure<double>(U + 1);
    double* y = ctx->vv.ensure<double>(U + 1);
    k_fill<double><<<1184, 256, 0, s>>>(U, x, 1.0);
    k_fill<double><<<1184, 256, 0, s>>>(U, r0, 1.0);
    LSMPS_CHECK_LAUNCH();
    Sell<float> Af{};
    Sell<double> Ad{};
    if (f32) Af = sell_scaled32(ctx);
    else Ad = sell_a64(ctx);
    const int* cut = f32 ? sell_cuts(ctx, Af) : sell_cuts(ctx, Ad);
    auto launch = [&] {
        if (f32) krylov_row_product(ctx, Af, cut, x, y, r0);
        else krylov_row_product(ctx, Ad, cut, x, y, r0);
    };
    launch();
    ev_record(ctx, 14);
    for (int r = 0; r < reps; ++r) launch();
    ev_record(ctx, 15);
    *ms = ev_elapsed(ctx, 14, 15) / reps;
    // algorithmic bytes: values + columns of the nonzeros (not the padding), the x gathers
    // counted once, y written, r0 read (FP64 vectors), slice pointers and lengths
    const double nnz = (double)ctx->nnz;
    // values + columns (2 bytes as steps, plus a 4-byte first column per row) per entry
    *bytes = ((f32 ? 4.0 : 8.0) + (ctx->have_steps ? 2.0 : 4.0)) * nnz + (ctx->have_steps ? 28.25 : 24.25) * U;
    // the bench overwrote solver vectors: a warm start from them is no longer valid
    ctx->have_solution = false;
}

__global__ void k_to_ref(const double* __restrict__ x, const int* __restrict__ u_of_ref, long long U,
                         double* __restrict__ out) {
    long long rr = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (rr < U) out[rr] = x[u_of_ref[rr]];
}

void ppe_download_pressure(lsmps_ctx* ctx, double* p, size_t u) {
    LSMPS_REQUIRE(ctx->have_solution, LSMPS_ERR_STATE, "no PPE solution");
    LSMPS_REQUIRE((long long)u == ctx->U, LSMPS_ERR_ARG, "pressure buffer size differs from the unknown count");
    if (!u) return;
    double* tmp = ctx->vtmp.ensure<double>(u + 1);
    k_to_ref<<<blocks_for(u, 256), 256, 0, ctx->stream>>>(ctx->vx.get<double>(), ctx->u_of_ref.get<int>(),
                                                          (long long)u, tmp);
    LSMPS_CHECK_LAUNCH();
    LSMPS_CUDA(cudaMemcpyAsync(p, tmp, u * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    LSMPS_CUDA(cudaStreamSynchronize(ctx->stream));
}

// The same values without waiting: reordered into a staging buffer on the context stream,
// then copied to the host on the context's copy stream, so the next step's kernels run while
// the copy is in flight. The staging buffer is reused by the next call, which therefore first
// orders the context stream after the previous copy.
void ppe_download_pressure_async(lsmps_ctx* ctx, double* p, size_t u) {
    LSMPS_REQUIRE(ctx->have_solution, LSMPS_ERR_STATE, "no PPE solution");
    LSMPS_REQUIRE((long long)u == ctx->U, LSMPS_ERR_ARG, "pressure buffer size differs from the unknown count");
    if (!u) return;
    if (!ctx->copy_stream) LSMPS_CUDA(cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
    if (!ctx->dl_ready) {
        LSMPS_CUDA(cudaEventCreateWithFlags(&ctx->dl_ready, cudaEventDisableTiming));
        LSMPS_CUDA(cudaEventCreateWithFlags(&ctx->dl_done, cudaEventDisableTiming));
    }
    if (ctx->dl_pending) {
        if (ctx->dl_stage.bytes < (u + 1) * sizeof(double)) {  // growing frees the copy's source
            LSMPS_CUDA(cudaEventSynchronize(ctx->dl_done));
            ctx->dl_pending = false;
        } else {
            LSMPS_CUDA(cudaStreamWaitEvent(ctx->stream, ctx->dl_done, 0));
        }
    }
    double* st = ctx->dl_stage.ensure<double>(u + 1);
    k_to_ref<<<blocks_for(u, 256), 256, 0, ctx->stream>>>(ctx->vx.get<double>(), ctx->u_of_ref.get<int>(),
                                                          (long long)u, st);
    LSMPS_CHECK_LAUNCH();
    LSMPS_CUDA(cudaEventRecord(ctx->dl_ready, ctx->stream));
    LSMPS_CUDA(cudaStreamWaitEvent(ctx->copy_stream, ctx->dl_ready, 0));
    LSMPS_CUDA(cudaMemcpyAsync(p, st, u * sizeof(double), cudaMemcpyDeviceToHost, ctx->copy_stream));
    LSMPS_CUDA(cudaEventRecord(ctx->dl_done, ctx->copy_stream));
    ctx->dl_pending = true;
}

void ppe_download_wait(lsmps_ctx* ctx) {
    if (!ctx->dl_pending) return;
    LSMPS_CUDA(cudaEventSynchronize(ctx->dl_done));
    ctx->dl_pending = false;
}

}  // namespace lsmps_gpu
