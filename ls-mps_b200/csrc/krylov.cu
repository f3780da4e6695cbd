// The BiCGStab engine of the FP64, JACOBI, MIXED and LEARNED solvers: a whole solve is one
// cooperative launch. Every block owns a contiguous range of rows (whole 32-row slices of the
// SELL copy, balanced by stored entries) in every vector update and row product, and the
// blocks meet at grid barriers, which also carry the dot products: each block leaves its
// partial sums before it arrives, and after the barrier every block adds all partials in block
// order, takes the iteration's scalar step and makes the loop's decisions (convergence,
// residual replacement, restart, fallback) for itself, from the same bits. So an iteration has
// no launches, no last-block serial step and no host round trip.
//
// What bounds it: the row products' matrix stream for large systems (2 x 41 us of a 911k-unknown
// iteration's 102), their gathers' latency at ~180k (2 x 13 of 38 us), and for small systems the
// barriers: 1.5 us each, 2.4 us with sums, five per iteration. As five kernels per iteration with a
// last-block sum in each, host-launched, an iteration took 35.0 us at 6,000 unknowns (17.5 now),
// 52 us at 181k (37.9) and 117 us at 911k (102).
//
// Waits are bounded: a block that polls a barrier more often than the context's wait limit raises
// DFLAG_TIMEOUT and ends, and so does every block that waits for it.
#include <algorithm>
#include <cmath>

#include "krylov.cuh"
#include "ops.cuh"
#include "sell.cuh"
#include "solver.cuh"

namespace lsmps_gpu {
namespace {

constexpr int KT = 1024;             // threads per block, one block per SM
constexpr int KW = KT / 32;
constexpr int KMAXB = 256;           // blocks of a launch at most

// ---- grid barrier and sums ----------------------------------------------------------------
struct Shared {
    double wa[KW], wb[KW];  // warps' partial sums
    double ga, gb;          // the grid's sums
    // the iteration's scalars (thread 0 updates them, every block the same)
    double rho, rho0, alpha, omega, beta, thresh, rn, best_rn, bnorm, rn_upd, first_rn;
    int done;    // 0 running, 1 converged, 2 breakdown, 3 iteration cap, 4 stalled
    int s_conv, it, iters, max_iter, stall, since_best, nonfinite;
    int act, in_chunk, total, base, replacements, restarts, fallback, tried, use_x;
    int converged, dead;
    long long guard;
};

struct Comm {
    double* part;   // two copies of (2 x KMAXB) partial sums
    unsigned* ctr;  // arrivals since the launch
    int* dflag;
    int limit;  // polls of a barrier; 0: every wait gives up
    unsigned epoch = 0;
    // (warp index shuffled so that the compiler knows it to be the same in all lanes)
    int warp, lane;

    // thread 0 of every block: arrive, wait for all blocks
    __device__ __forceinline__ void arrive_and_wait(Shared& sh) {
        if (sh.dead) return;
        const unsigned target = (epoch + 1) * gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
        unsigned v;
        int polls = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
        } while ((int)(v - target) < 0 && ++polls < limit);
        if (polls >= limit) {
            atomicOr(dflag, DFLAG_TIMEOUT);
            sh.dead = 1;
            sh.done = 5;
        }
    }
    // all blocks' earlier writes are visible after it
    __device__ __forceinline__ void barrier(Shared& sh) {
        __syncthreads();
        if (threadIdx.x == 0) arrive_and_wait(sh);
        ++epoch;
        __syncthreads();
    }
    // the barrier with the grid's sums of a and b in sh.ga, sh.gb (block order, then a fixed
    // tree), followed by step() in thread 0
    template <class F>
    __device__ __forceinline__ void sums(double a, double b, Shared& sh, F&& step) {
        a = warp_sum(a);
        b = warp_sum(b);
        if (lane == 0) {
            sh.wa[warp] = a;
            sh.wb[warp] = b;
        }
        __syncthreads();
        if (warp == 0) {
            double* p = part + (epoch & 1) * 2 * KMAXB;
            const double x = warp_sum(lane < KW ? sh.wa[lane] : 0.0), y = warp_sum(lane < KW ? sh.wb[lane] : 0.0);
            if (lane == 0) {
                __stcg(p + blockIdx.x, x);
                __stcg(p + KMAXB + blockIdx.x, y);
                arrive_and_wait(sh);
            }
            __syncwarp();
            double s = 0, t = 0;
            for (int k = lane; k < (int)gridDim.x; k += 32) {
                s += __ldcg(p + k);
                t += __ldcg(p + KMAXB + k);
            }
            s = warp_sum(s);
            t = warp_sum(t);
            if (lane == 0) {
                sh.ga = s;
                sh.gb = t;
                if (!sh.dead) step();
            }
        }
        ++epoch;
        __syncthreads();
    }
};

enum Act { ACT_INIT, ACT_ITER, ACT_REPLACE, ACT_END };

// Thread 0, after the iteration stopped (or broke down after a replacement): the Krylov space
// restarts from the current iterate and its true residual.
__device__ void restart_or_stop(Shared& sh, const KrylovOpts& o) {
    if (sh.done == 4 && o.use_nn) sh.fallback = 1;
    if (sh.nonfinite) {
        sh.act = ACT_END;
        return;
    }
    sh.use_x = 1;
    sh.stall = 0;
    sh.max_iter = o.max_iter - sh.total;
    sh.restarts += 1;
    sh.act = ++sh.guard < o.max_chunks ? ACT_INIT : ACT_END;
}

__device__ __forceinline__ double2 ld2(const double* p) { return *reinterpret_cast<const double2*>(p); }
__device__ __forceinline__ void st2(double* p, double a, double b) {
    *reinterpret_cast<double2*>(p) = make_double2(a, b);
}

// MIXED: iterate with the FP32 copy A, take residuals with the FP64 copy As; else A throughout.
template <class TM, bool MIXED, bool C16>
__global__ void __launch_bounds__(KT, 1) k_bicgstab(const Sell<TM> A, const Sell<double> As, const KrylovVecs V,
                                                    const KrylovOpts o, Comm C0, KrylovResult* out) {
    __shared__ Shared sh;
    Comm C = C0;
    C.warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    C.lane = threadIdx.x & 31;
    const long long sl0 = sell_cut(A, blockIdx.x, gridDim.x), sl1 = sell_cut(A, blockIdx.x + 1, gridDim.x);
    const long long r0 = sl0 << 5, r1 = min(sl1 << 5, A.n);
    const int tid = threadIdx.x;
    auto rows = [&](auto&& f) {
        for (long long i = r0 + tid; i < r1; i += KT) f(i);
    };
    // two rows per thread with 16-byte accesses (vectors hold one element past the last row)
    auto pairs = [&](auto&& f) {
        for (long long i = r0 + 2 * tid; i < r1; i += 2 * KT) f(i);
    };
    auto product = [&](const auto& S, const double* x, auto&& f) {
        for (long long s = sl0 + C.warp; s < sl1; s += KW) {
            const double y = sell_product<C16>(S, s, C.lane, x);
            const long long i = (s << 5) + C.lane;
            if (i < A.n) f(i, y);
        }
    };
    if (tid == 0) {
        sh.act = ACT_INIT;
        sh.use_x = o.use_x;
        sh.max_iter = o.max_iter;
        sh.stall = o.use_nn ? o.stall : 0;
        sh.total = sh.base = sh.replacements = sh.restarts = sh.fallback = sh.tried = 0;
        sh.converged = sh.dead = sh.done = 0;
        sh.guard = 0;
    }
    __syncthreads();
    for (;;) {
        const int act = sh.act;
        if (act == ACT_END || sh.dead) break;
        double a = 0, b = 0;
        if (act == ACT_INIT) {
            // r = b - A x (or b), r0 = r, p = v = 0
            const bool use_x = sh.use_x != 0;
            auto start = [&](long long i, double ax) {
                const double bi = V.b[i], ri = use_x ? bi - ax : bi;
                V.r[i] = ri;
                V.r0[i] = ri;
                V.p[i] = 0;
                V.v[i] = 0;
                a += bi * bi;
                b += ri * ri;
            };
            if (use_x) {
                if constexpr (MIXED) product(As, V.x, start);
                else product(A, V.x, start);
            } else {
                rows([&](long long i) {
                    V.x[i] = 0;
                    start(i, 0.0);
                });
            }
            C.sums(a, b, sh, [&] {
                sh.bnorm = sqrt(sh.ga);
                sh.thresh = o.tol * fmax(1.0, sh.bnorm);
                sh.rho0 = sh.alpha = sh.omega = 1.0;
                sh.rho = sh.beta = sh.gb;  // beta: (rho / rho0) (alpha / omega)
                sh.rn = sh.best_rn = sqrt(sh.gb);
                sh.since_best = sh.it = sh.iters = sh.s_conv = 0;
                sh.nonfinite = !isfinite(sh.gb);
                sh.done = sh.nonfinite ? 2 : sh.rn <= sh.thresh ? 1 : fabs(sh.gb) < 1e-30 ? 2 : sh.max_iter <= 0 ? 3 : 0;
                sh.base = sh.in_chunk = 0;
                sh.rn_upd = sh.rn;
                if (sh.tried == 0) {  // the first start: a network guess worse than none goes
                    sh.tried = 1;
                    sh.first_rn = sh.rn;
                    if (o.use_nn && (!isfinite(sh.rn) || sh.rn >= (o.warm_rn2 ? sqrt(*o.warm_rn2) : sh.bnorm))) {
                        sh.fallback = 1;
                        sh.tried = 2;
                        sh.stall = 0;
                        sh.use_x = o.warm_rn2 ? 2 : 0;
                        sh.act = ACT_INIT;
                        return;
                    }
                }
                if (sh.done == 1) {
                    sh.converged = 1;
                    sh.act = ACT_END;
                } else if (sh.done == 2) {
                    sh.act = ACT_END;
                } else if (sh.done == 3) {  // no iterations asked for: the start's true residual decides
                    sh.act = MIXED && sh.restarts == 0 ? ACT_REPLACE : ACT_END;
                } else {
                    sh.act = ACT_ITER;
                }
            });
            if (sh.act == ACT_INIT && sh.use_x == 2) {  // back to the warm start, kept in s
                rows([&](long long i) { V.x[i] = V.keep[i]; });
                C.barrier(sh);
            }
        } else if (act == ACT_ITER) {
            // p = r + beta (p - omega v)
            {
                const double beta = sh.beta, omega = sh.omega;
                    pairs([&](long long i) {
                        const double2 ri = ld2(V.r + i), pi = ld2(V.p + i), vi = ld2(V.v + i);
                        st2(V.p + i, ri.x + beta * (pi.x - omega * vi.x), ri.y + beta * (pi.y - omega * vi.y));
                    });
            }
            C.barrier(sh);
            product(A, V.p, [&](long long i, double y) {  // v = A p, r0.v
                V.v[i] = y;
                a += V.r0[i] * y;
            });
            C.sums(a, 0.0, sh, [&] {
                const double den = sh.ga;
                if (!isfinite(den)) { sh.nonfinite = 1; sh.done = 2; }
                else if (fabs(den) < 1e-30) sh.done = 2;
                else sh.alpha = sh.rho / den;
            });
            if (!sh.done) {
                // s = r - alpha v, |s|
                const double alpha = sh.alpha;
                double ss = 0;
                    pairs([&](long long i) {
                        const double2 ri = ld2(V.r + i), vi = ld2(V.v + i);
                        const double s0 = ri.x - alpha * vi.x, s1 = ri.y - alpha * vi.y;
                        st2(V.s + i, s0, s1);
                        ss += s0 * s0;
                        if (i + 1 < r1) ss += s1 * s1;
                    });
                C.sums(ss, 0.0, sh, [&] {
                    const double sn = sqrt(sh.ga);
                    if (sn <= sh.thresh) {
                        sh.s_conv = 1;
                        sh.iters = sh.it + 1;
                        sh.rn = sn;
                        sh.done = 1;
                    }
                });
                if (sh.s_conv) {
                    rows([&](long long i) {
                        V.x[i] += alpha * V.p[i];
                        V.r[i] = V.s[i];
                    });
                    C.barrier(sh);  // the next product gathers x
                } else if (!sh.done) {
                    double ts = 0, tt = 0;
                    product(A, V.s, [&](long long i, double y) {  // t = A s, t.s, t.t
                        V.t[i] = y;
                        ts += y * V.s[i];
                        tt += y * y;
                    });
                    C.sums(ts, tt, sh, [&] {
                        if (!isfinite(sh.ga) || !isfinite(sh.gb)) { sh.nonfinite = 1; sh.done = 2; }
                        else if (sh.gb < 1e-30) sh.done = 2;
                        else sh.omega = sh.ga / sh.gb;
                    });
                    if (!sh.done) {
                        // x += alpha p + omega s, r = s - omega t, |r|, r0.r
                        const double omega = sh.omega;
                        double rr = 0, r0r = 0;
                        pairs([&](long long i) {
                            const double2 xi = ld2(V.x + i), pi = ld2(V.p + i), si = ld2(V.s + i),
                                          ti = ld2(V.t + i), zi = ld2(V.r0 + i);
                            st2(V.x + i, xi.x + (alpha * pi.x + omega * si.x), xi.y + (alpha * pi.y + omega * si.y));
                            const double ra = si.x - omega * ti.x, rb = si.y - omega * ti.y;
                            st2(V.r + i, ra, rb);
                            rr += ra * ra;
                            r0r += zi.x * ra;
                            if (i + 1 < r1) {
                                rr += rb * rb;
                                r0r += zi.y * rb;
                            }
                        });
                        C.sums(rr, r0r, sh, [&] {
                            sh.it += 1;
                            sh.iters = sh.it;
                            const double rn = sqrt(sh.ga), rho = sh.gb;
                            sh.rn = rn;
                            if (!isfinite(rn)) { sh.nonfinite = 1; sh.done = 2; return; }
                            if (rn <= sh.thresh) { sh.done = 1; return; }
                            if (rn < 0.99 * sh.best_rn) { sh.best_rn = rn; sh.since_best = 0; }
                            else if (++sh.since_best >= sh.stall && sh.stall > 0) { sh.done = 4; return; }
                            if (fabs(sh.omega) < 1e-30) { sh.done = 2; return; }
                            if (sh.it >= sh.max_iter) { sh.done = 3; return; }
                            if (fabs(rho) < 1e-30) { sh.done = 2; return; }
                            sh.beta = (rho / sh.rho) * (sh.alpha / sh.omega);
                            sh.rho0 = sh.rho;
                            sh.rho = rho;
                        });
                    }
                }
            }
            // the decision after a chunk of iterations (or at a stop)
            __syncthreads();
            if (tid == 0) {
                if (!sh.done && ++sh.in_chunk < o.chunk) {
                    sh.act = ACT_ITER;
                } else if (!MIXED) {
                    sh.in_chunk = 0;
                    if (sh.done) {
                        sh.converged = sh.done == 1;
                        sh.act = ACT_END;
                    }
                } else {
                    sh.in_chunk = 0;
                    sh.total += sh.iters - sh.base;
                    sh.base = sh.iters;
                    if (!sh.done && sh.rn > o.delta * sh.rn_upd) sh.act = ACT_ITER;
                    else if (sh.done == 0 || sh.done == 3 || sh.total >= o.max_iter) sh.act = ACT_REPLACE;
                    else restart_or_stop(sh, o);
                }
            }
            __syncthreads();
        } else {
            // ACT_REPLACE: r = b - (A D^-1) y with the FP64 matrix replaces the recursive residual,
            // keeping the search direction (van der Vorst & Ye)
            if constexpr (MIXED) {
                product(As, V.x, [&](long long i, double ay) {
                    const double ri = V.b[i] - ay;
                    V.r[i] = ri;
                    a += ri * ri;
                    b += V.r0[i] * ri;
                });
                C.sums(a, b, sh, [&] {
                    const bool last = sh.done == 3 || sh.total >= o.max_iter;  // iteration cap
                    sh.rn = sqrt(sh.ga);
                    if (sh.rn < sh.best_rn) sh.best_rn = sh.rn;
                    sh.beta = (sh.gb / sh.rho0) * (sh.alpha / sh.omega);
                    sh.rho = sh.gb;
                    sh.done = 0;
                    sh.s_conv = 0;
                    if (!isfinite(sh.ga)) { sh.nonfinite = 1; sh.done = 2; }
                    else if (sh.rn <= sh.thresh) sh.done = 1;
                    else if (!isfinite(sh.gb) || fabs(sh.gb) < 1e-30) sh.done = 2;
                    if (last) {
                        sh.converged = sh.done == 1;
                        sh.act = ACT_END;
                        return;
                    }
                    sh.replacements += 1;
                    sh.rn_upd = sh.rn;
                    if (sh.done == 1) {
                        sh.converged = 1;
                        sh.act = ACT_END;
                    } else if (sh.done == 0) {
                        sh.act = ACT_ITER;
                    } else {
                        restart_or_stop(sh, o);
                    }
                });
            }
        }
    }
    if (sh.dead) return;
    // x = D^-1 y, then the error against p*
    if (o.dinv) rows([&](long long i) { V.x[i] *= o.dinv[i]; });
    __syncthreads();
    double se = 0, ee = 0, mx = 0;
    rows([&](long long i) {
        const double e = V.x[i] - o.xe[i];
        se += e * e;
        ee += o.xe[i] * o.xe[i];
        mx = fmax(mx, fabs(e));
    });
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, k));
    if (C.lane == 0 && mx > 0) atomicMax(&out->maxbits, (unsigned long long)__double_as_longlong(mx));
    C.sums(se, ee, sh, [] {});
    if (blockIdx.x == 0 && tid == 0) {
        out->rn = sh.rn;
        out->bnorm = sh.bnorm;
        out->iterations = MIXED ? sh.total : sh.iters;
        out->outer = sh.replacements + sh.restarts;
        out->converged = sh.converged;
        out->fallback = sh.fallback;
        out->nonfinite = sh.nonfinite;
        out->err2 = sh.ga;
        out->ref2 = sh.gb;
    }
}

// The row product of an iteration on its own, for the kernel bench (a solve forms it inside
// k_bicgstab): v = A p and the partials of r0.v
template <class TM, bool C16>
__global__ void __launch_bounds__(KT, 1) k_row_product(const Sell<TM> A, const int* cut, const double* p, double* v,
                                                       const double* r0, double* part) {
    __shared__ double ws[KW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long sl0 = cut[blockIdx.x], sl1 = cut[blockIdx.x + 1];
    double acc = 0;
    for (long long s = sl0 + warp; s < sl1; s += KW) {
        const double y = sell_product<C16>(A, s, lane, p);
        const long long i = (s << 5) + lane;
        if (i < A.n) {
            v[i] = y;
            acc += r0[i] * y;
        }
    }
    acc = warp_sum(acc);
    if (lane == 0) ws[warp] = acc;
    __syncthreads();
    if (warp == 0) {
        acc = warp_sum(lane < KW ? ws[lane] : 0.0);
        if (lane == 0) part[blockIdx.x] = acc;
    }
}

// zeroed barrier state behind the partial sums (all in ctx->red)
Comm make_comm(lsmps_ctx* ctx, KrylovResult** out) {
    double* red = ctx->red.ensure<double>(4 * KMAXB + 64);
    LSMPS_CUDA(cudaMemsetAsync(red + 4 * KMAXB, 0, 64 * sizeof(double), ctx->stream));
    if (out) *out = reinterpret_cast<KrylovResult*>(red + 4 * KMAXB + 8);
    static_assert(sizeof(KrylovResult) <= 48 * sizeof(double), "result layout");
    Comm c;
    c.part = red;
    c.ctr = reinterpret_cast<unsigned*>(red + 4 * KMAXB);
    c.dflag = ctx->dflags.get<int>();
    c.limit = ctx->wait_limit;
    return c;
}

template <class TM, bool MIXED, bool C16>
void launch(lsmps_ctx* ctx, Sell<TM> A, Sell<double> As, KrylovVecs V, KrylovOpts o, Comm C, KrylovResult* out) {
    auto k = k_bicgstab<TM, MIXED, C16>;
    void* args[] = {&A, &As, &V, &o, &C, &out};
    LSMPS_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(k), dim3(krylov_blocks(ctx, A.nslices)), dim3(KT), args, 0,
                                           ctx->stream));
    note_launches(1);
}

}  // namespace

// blocks of a launch: one per SM, less those the context leaves free; fewer for small systems (at
// least eight slices each). A block fills its SM's register file for the whole solve
// (milliseconds), so the kernels of other contexts and streams wait for its end unless SMs are left
// to them: a 20,000-particle list build on another context took 35 ms beside FP64 solves at 1M and
// 20 ms beside MIXED ones, 1.1 ms with two SMs left, 0.65 with four. Two cost 102.2 -> 104.4 us per
// MIXED iteration at 911k unknowns (106.6 four) and other bits (the sums' order goes by blocks), so
// none is the default.
unsigned krylov_blocks(lsmps_ctx* ctx, long long nslices) {
    int sms = 0;
    LSMPS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
    const int most = std::max(1, std::min(sms - ctx->free_sms, KMAXB));
    return (unsigned)std::max<long long>(1, std::min<long long>(most, (nslices + 7) / 8));
}

KrylovResult krylov_solve(lsmps_ctx* ctx, const Sell<float>* Af, const Sell<double>& A, const KrylovVecs& V,
                          const KrylovOpts& o) {
    KrylovResult* out = nullptr;
    const Comm C = make_comm(ctx, &out);
    const bool c16 = A.dcol != nullptr;
    if (!Af) {
        if (c16) launch<double, false, true>(ctx, A, A, V, o, C, out);
        else launch<double, false, false>(ctx, A, A, V, o, C, out);
    } else {
        if (c16) launch<float, true, true>(ctx, *Af, A, V, o, C, out);
        else launch<float, true, false>(ctx, *Af, A, V, o, C, out);
    }
    ev_record(ctx, 11);
    KrylovResult h{};
    read_back(ctx, {{out, &h, sizeof(h)}}, "PPE solve");
    return h;
}

template <class TM>
void krylov_row_product(lsmps_ctx* ctx, const Sell<TM>& A, const int* cut, const double* p, double* v,
                        const double* r0) {
    double* part = ctx->red.ensure<double>(4 * KMAXB + 64);
    const unsigned nb = krylov_blocks(ctx, A.nslices);
    if (A.dcol) k_row_product<TM, true><<<nb, KT, 0, ctx->stream>>>(A, cut, p, v, r0, part);
    else k_row_product<TM, false><<<nb, KT, 0, ctx->stream>>>(A, cut, p, v, r0, part);
    LSMPS_CHECK_LAUNCH();
}
template void krylov_row_product<float>(lsmps_ctx*, const Sell<float>&, const int*, const double*, double*, const double*);
template void krylov_row_product<double>(lsmps_ctx*, const Sell<double>&, const int*, const double*, double*,
                                         const double*);

}  // namespace lsmps_gpu
