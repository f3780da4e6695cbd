// Sums with the rounding of a sequential loop, formed in parallel by one block.
//
// s <- fl(s + a) for a in order. While |s| stays in one binade [2^e, 2^(e+1)), write
// |s| = m u with u = 2^(e-52) and m an integer of 53 bits; then fl(s + a) = (m + q) u with q
// the integer nearest to a / u (signs folded into a), unless a / u lies half-way between two
// integers. So a run of elements that stays inside the binade and has no such tie is one
// integer addition to the mantissa of s. Elements at which the running value reaches the
// binade's ends, or ties, are added by ordinary rounded additions, after which the binade is
// taken anew: the result is the sequential sum's for any input.
#pragma once
#include "common.cuh"

namespace lsmps_gpu {

struct SeqRun {
    long long d = 0;           // increment of m over the run
    long long lo = 0, hi = 0;  // its smallest and largest value on the way (0 included)
};
constexpr long long SEQ_NEVER = 1LL << 61;  // hi of a run that has to be added one by one

// first a, then b
__device__ __forceinline__ SeqRun seq_then(const SeqRun& a, const SeqRun& b) {
    return SeqRun{a.d + b.d, min(a.lo, a.d + b.lo), min(max(a.hi, a.d + b.hi), SEQ_NEVER)};
}

__device__ __forceinline__ unsigned seq_key(double s) {  // sign and exponent field
    return (unsigned)((unsigned long long)__double_as_longlong(s) >> 52);
}
// 1 / u is a normal number and s is finite and not zero
__device__ __forceinline__ bool seq_key_ok(unsigned key) { return (key & 0x7ffu) >= 60u && (key & 0x7ffu) < 2047u; }

// Adds element a to the run. scale: 1 / u with the sign of s. |a| >= 2^51 u, NaN and ties make
// the run SEQ_NEVER.
__device__ __forceinline__ void seq_element(SeqRun& r, double a, double scale) {
    const double magic = 6755399441055744.0;  // 1.5 * 2^52: t + magic rounds t to an integer
    const double t = xmul(a, scale);
    const double tm = xadd(t, magic);
    const double rem = xsub(t, xsub(tm, magic));  // exact for |t| <= 2^51
    r.d += __double_as_longlong(tm) - __double_as_longlong(magic);
    r.lo = min(r.lo, r.d);
    r.hi = max(r.hi, r.d);
    if (!(fabs(t) < 2251799813685248.0) || fabs(rem) == 0.5) {
        r.d = 0;
        r.hi = SEQ_NEVER;
    }
}

constexpr int SEQ_THREADS = 1024;
constexpr int SEQ_L = 7;                       // elements per thread (odd: no bank conflicts)
constexpr int SEQ_PASS = SEQ_THREADS * SEQ_L;  // elements per pass, staged in shared memory
constexpr size_t SEQ_SMEM = (SEQ_PASS + 16) * sizeof(double);

// The lanes' runs of a pass: the increment up to and including the lane's run within its warp
// (wrapping arithmetic: only differences over lanes whose runs hold are used), the run's bounds
// and the key of the binade it is for; and the same of the warps' runs.
struct SeqShared {
    unsigned long long upto[SEQ_THREADS];
    long long d[SEQ_THREADS], lo[SEQ_THREADS], hi[SEQ_THREADS];
    unsigned key[SEQ_THREADS];
    SeqRun warp[32];
    unsigned wkey[32];
    double wsum[32];
    double sum;
};

// e[0..n) added to s one by one; the next eight elements are read during eight additions, so the
// chain is the additions' own latency (reads go up to 16 past the end).
__device__ __forceinline__ double seq_add_run(const double* e, int n, double s) {
    double cur[8], nxt[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) cur[k] = e[k];
    int b = 0;
    for (; b + 8 <= n; b += 8) {
#pragma unroll
        for (int k = 0; k < 8; ++k) nxt[k] = e[b + 8 + k];
#pragma unroll
        for (int k = 0; k < 8; ++k) s = xadd(s, cur[k]);
#pragma unroll
        for (int k = 0; k < 8; ++k) cur[k] = nxt[k];
    }
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        if (b + k >= n) break;
        s = xadd(s, cur[k]);
    }
    return s;
}

// One warp: adds runs `pos`, pos + 1, ... (lane l holds run l: upto, r, key) to s for as long as
// each starts and stays in the binade of s; returns the first that does not, or n.
__device__ __forceinline__ int seq_skip(double& s, int pos, int n, unsigned long long upto, const SeqRun& r,
                                        unsigned key) {
    const int lane = threadIdx.x & 31;
    const long long bits = __double_as_longlong(s);
    // (upto up to, not including, lane pos: of lane pos itself less its own run)
    const unsigned long long before = __shfl_sync(0xffffffffu, upto - (unsigned long long)r.d, pos);
    const long long m = (bits & 0xfffffffffffffLL) + (long long)(upto - (unsigned long long)r.d - before);
    const bool in = (lane < n) & (key == seq_key(s)) & (m + r.lo > 0) & (m + r.hi < (1LL << 52));
    const unsigned out = ~(__ballot_sync(0xffffffffu, in) >> pos);
    const int q = min(pos + (int)__clz(__brev(out)), 32);
    const unsigned long long after = __shfl_sync(0xffffffffu, upto, max(q - 1, 0));
    s = __longlong_as_double(q > pos ? bits + (long long)(after - before) : bits);
    return q;
}

// The sequential sum of prod[0..n) from 0, by one block of SEQ_THREADS threads; the result in
// warp 0. Per pass of up to SEQ_PASS elements, each lane guesses the sum at its first element
// from plain partial sums (right to ~1e-13, so its binade is almost always the true one) and
// makes its L elements a run of that binade; a warp whose lanes agree on the binade has a run
// of all of them. Warp 0 then skips over the warps' runs as far as they stay in the binade of
// the sum, goes through the lanes' runs of a warp that does not, and adds a lane's elements one
// by one where the sum leaves its binade among them. Sums of squares leave it ~9 times at
// U = 6,000; r0.v and r0.r, which BiCGStab drives towards zero, up to 800 times.
__device__ inline double block_seq_sum(const double* __restrict__ prod, long long n, double* el, SeqShared& sh) {
    // (a shuffled warp index, so that the compiler knows `warp == 0` below to be the same in all
    // lanes: with threadIdx.x >> 5 the walk's shuffles took ~1,300 cycles each step instead of 230)
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    double s = 0.0;
    if (threadIdx.x == 0) sh.sum = 0.0;
    for (long long base = 0; base < n; base += SEQ_PASS) {
        const int cnt = (int)min((long long)SEQ_PASS, n - base);
        const int L = ((cnt + SEQ_THREADS - 1) / SEQ_THREADS) | 1;
#pragma unroll
        for (int k = 0; k < SEQ_L; ++k) {  // past the end -0.0, which changes no sum
            const int i = threadIdx.x + k * SEQ_THREADS;
            if (k < L) el[i] = i < cnt ? prod[base + i] : -0.0;
        }
        __syncthreads();
        // (loops kept rolled: a launch runs this code once, and cold code costs ~10 cycles per
        // instruction)
        double incl = 0.0;
#pragma unroll 1
        for (int k = 0; k < L; ++k) incl += el[threadIdx.x * L + k];
        const double own = incl;
#pragma unroll 1
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) sh.wsum[warp] = incl;
        __syncthreads();
        const unsigned key = seq_key(sh.sum + warp_sum(lane < warp ? sh.wsum[lane] : 0.0) + (incl - own));
        SeqRun r;
        if (seq_key_ok(key)) {
            const double scale = __longlong_as_double(((long long)(2098u - (key & 0x7ffu)) << 52) |
                                                      ((long long)(key & 0x800u) << 52));
#pragma unroll 1
            for (int k = 0; k < L; ++k) seq_element(r, el[threadIdx.x * L + k], scale);
        } else {
            r.hi = SEQ_NEVER;
        }
        sh.d[threadIdx.x] = r.d;
        sh.lo[threadIdx.x] = r.lo;
        sh.hi[threadIdx.x] = r.hi;
        sh.key[threadIdx.x] = key;
#pragma unroll 1
        for (int o = 1; o < 32; o <<= 1) {  // lane l: the run of lanes 0 .. l
            SeqRun before;
            before.d = __shfl_up_sync(0xffffffffu, r.d, o);
            before.lo = __shfl_up_sync(0xffffffffu, r.lo, o);
            before.hi = __shfl_up_sync(0xffffffffu, r.hi, o);
            if (lane >= o) r = seq_then(before, r);
        }
        sh.upto[threadIdx.x] = (unsigned long long)r.d;
        const bool agree = __all_sync(0xffffffffu, key == __shfl_sync(0xffffffffu, key, 0));
        if (lane == 31) {
            if (!agree) r.hi = SEQ_NEVER;
            sh.warp[warp] = r;
            sh.wkey[warp] = key;
        }
        __syncthreads();
        if (warp == 0) {
            s = sh.sum;
            const int nw = (cnt + 32 * L - 1) / (32 * L);
            const SeqRun wr = sh.warp[lane];
            const unsigned wk = sh.wkey[lane];
            unsigned long long wupto = (unsigned long long)wr.d;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xffffffffu, wupto, o);
                if (lane >= o) wupto += y;
            }
            // a skip takes ~230 cycles, a lane's seven additions ~60: while skipping passes fewer
            // than four lanes, twice as many lanes (up to four warps' lanes) are added one by
            // one before it is tried again
            int alone = 1;
            for (int t = 0; t < 32 * nw;) {  // t: the next lane of the pass
                const int w = t >> 5;
                if ((t & 31) == 0) {
                    t = 32 * seq_skip(s, w, nw, wupto, wr, wk);
                    if (t > 32 * w) continue;
                }
                const SeqRun lr{sh.d[32 * w + lane], sh.lo[32 * w + lane], sh.hi[32 * w + lane]};
                const unsigned lk = sh.key[32 * w + lane];
                const unsigned long long lupto = sh.upto[32 * w + lane];
                while (t < 32 * (w + 1)) {
                    const int from = t;
                    t = 32 * w + seq_skip(s, t & 31, 32, lupto, lr, lk);
                    if (t == 32 * (w + 1)) break;
                    alone = t - from >= 4 ? max(alone >> 1, 1) : min(2 * alone, 128);
                    const int to = min(t + alone, 32 * nw);
                    s = seq_add_run(el + t * L, (to - t) * L, s);
                    t = to;
                }
            }
            if (lane == 0) sh.sum = s;
        }
        __syncthreads();  // the next pass overwrites the elements
    }
    return s;
}

}  // namespace lsmps_gpu
