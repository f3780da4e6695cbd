// Row products of the SELL-32x4 copies.
#pragma once
#include "solver.cuh"

namespace lsmps_gpu {

// Row i of a SELL-32x4 matrix: slice s = i / 32 stores its 32 rows in chunks of four
// consecutive entries per row (entries 4c..4c+3 of lane l at sptr[s] + 128 c + 4 l), zero-
// padded to the slice's longest row rounded up to a multiple of four. One thread per row,
// one warp per slice: each thread reads its next four values and four columns with two
// 16-byte loads (a warp covers 512 contiguous bytes per load), and two chunks are issued
// before their eight x gathers, so each thread keeps 64-96 bytes of matrix loads and eight
// gathers in flight. Matrix loads stream past L1/L2 (__ldcs) so the vectors, re-read every
// iteration, stay in the 126 MB L2.
__device__ __forceinline__ void ld4(const float* p, float v[4]) {
    float4 q = __ldcs(reinterpret_cast<const float4*>(p));
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void ld4(const double* p, double v[4]) {
    double2 a = __ldcs(reinterpret_cast<const double2*>(p));
    double2 b = __ldcs(reinterpret_cast<const double2*>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void ld4(const int* p, int v[4]) {
    int4 q = __ldcs(reinterpret_cast<const int4*>(p));
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
// four 16-bit column steps (8 bytes) -> four columns continuing from c
__device__ __forceinline__ void ld4_steps(const unsigned short* p, int& c, int out[4]) {
    uint2 q = __ldcs(reinterpret_cast<const uint2*>(p));
    c += (int)(q.x & 0xffffu);
    out[0] = c;
    c += (int)(q.x >> 16);
    out[1] = c;
    c += (int)(q.y & 0xffffu);
    out[2] = c;
    c += (int)(q.y >> 16);
    out[3] = c;
}

// The row product with 16-bit column steps (2 bytes per entry instead of 4).
template <class TM, class T>
__device__ __forceinline__ double sell_row16(const Sell<TM>& A, long long s, int lane, const T* x) {
    const long long base = (long long)A.sptr[s] + 4 * lane;
    const TM* __restrict__ val = A.val + base;
    const unsigned short* __restrict__ dc = A.dcol + base;
    int cur = A.rbase[(s << 5) + lane];
    const int chunks = A.slen[s] >> 2;
    double a0 = 0, a1 = 0;
    int c = 0;
    for (; c + 2 <= chunks; c += 2) {
        TM v0[4], v1[4];
        int c0[4], c1[4];
        ld4(val + 128 * c, v0);
        ld4(val + 128 * (c + 1), v1);
        ld4_steps(dc + 128 * c, cur, c0);
        ld4_steps(dc + 128 * (c + 1), cur, c1);
        T x0[4], x1[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            x0[j] = x[c0[j]];
            x1[j] = x[c1[j]];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            a0 += (double)v0[j] * (double)x0[j];
            a1 += (double)v1[j] * (double)x1[j];
        }
    }
    if (c < chunks) {
        TM v0[4];
        int c0[4];
        ld4(val + 128 * c, v0);
        ld4_steps(dc + 128 * c, cur, c0);
#pragma unroll
        for (int j = 0; j < 4; ++j) a0 += (double)v0[j] * (double)x[c0[j]];
    }
    return a0 + a1;
}

// The same row product, software-pipelined: the next pair of chunks' values and column steps
// are loaded while the current pair's gathers are in flight, so a pair of chunks waits for one
// round trip instead of two. The sums are added in the same order as sell_row16 (same bits);
// it needs ~64 registers, so its kernels run 4 blocks of RB threads per SM instead of 6.
__device__ __forceinline__ void steps_to_cols(uint2 q, int& c, int out[4]) {
    c += (int)(q.x & 0xffffu);
    out[0] = c;
    c += (int)(q.x >> 16);
    out[1] = c;
    c += (int)(q.y & 0xffffu);
    out[2] = c;
    c += (int)(q.y >> 16);
    out[3] = c;
}
template <class TM, class T>
__device__ __forceinline__ double sell_row16_pipe(const Sell<TM>& A, long long s, int lane,
                                                  const T* x) {
    const long long base = (long long)A.sptr[s] + 4 * lane;
    const TM* __restrict__ val = A.val + base;
    const unsigned short* __restrict__ dc = A.dcol + base;
    int cur = A.rbase[(s << 5) + lane];
    const int chunks = A.slen[s] >> 2;
    double a0 = 0, a1 = 0;
    int c = 0;
    TM v0[4], v1[4];
    uint2 s0 = make_uint2(0, 0), s1 = make_uint2(0, 0);
    if (chunks >= 2) {
        ld4(val, v0);
        ld4(val + 128, v1);
        s0 = __ldcs(reinterpret_cast<const uint2*>(dc));
        s1 = __ldcs(reinterpret_cast<const uint2*>(dc + 128));
    }
    for (; c + 2 <= chunks; c += 2) {
        int c0[4], c1[4];
        steps_to_cols(s0, cur, c0);
        steps_to_cols(s1, cur, c1);
        T x0[4], x1[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            x0[j] = x[c0[j]];
            x1[j] = x[c1[j]];
        }
        if (c + 4 <= chunks) {  // the next pair, in flight with the gathers above
            TM w0[4], w1[4];
            ld4(val + 128 * (c + 2), w0);
            ld4(val + 128 * (c + 3), w1);
            const uint2 t0 = __ldcs(reinterpret_cast<const uint2*>(dc + 128 * (c + 2)));
            const uint2 t1 = __ldcs(reinterpret_cast<const uint2*>(dc + 128 * (c + 3)));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                a0 += (double)v0[j] * (double)x0[j];
                a1 += (double)v1[j] * (double)x1[j];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v0[j] = w0[j];
                v1[j] = w1[j];
            }
            s0 = t0;
            s1 = t1;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                a0 += (double)v0[j] * (double)x0[j];
                a1 += (double)v1[j] * (double)x1[j];
            }
        }
    }
    if (c < chunks) {
        TM u0[4];
        int c0[4];
        ld4(val + 128 * c, u0);
        ld4_steps(dc + 128 * c, cur, c0);
#pragma unroll
        for (int j = 0; j < 4; ++j) a0 += (double)u0[j] * (double)x[c0[j]];
    }
    return a0 + a1;
}

// C16: the view's columns are 16-bit steps (a compile-time choice: one code path per kernel)
template <bool C16, class TM, class T>
__device__ __forceinline__ double sell_row(const Sell<TM>& A, long long s, int lane, const T* x) {
    if constexpr (C16) return sell_row16(A, s, lane, x);
    const long long base = (long long)A.sptr[s] + 4 * lane;
    const TM* __restrict__ val = A.val + base;
    const int* __restrict__ col = A.col + base;
    const int chunks = A.slen[s] >> 2;
    double a0 = 0, a1 = 0;
    int c = 0;
    for (; c + 2 <= chunks; c += 2) {
        TM v0[4], v1[4];
        int c0[4], c1[4];
        ld4(val + 128 * c, v0);
        ld4(col + 128 * c, c0);
        ld4(val + 128 * (c + 1), v1);
        ld4(col + 128 * (c + 1), c1);
        T x0[4], x1[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            x0[j] = x[c0[j]];
            x1[j] = x[c1[j]];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            a0 += (double)v0[j] * (double)x0[j];
            a1 += (double)v1[j] * (double)x1[j];
        }
    }
    if (c < chunks) {
        TM v0[4];
        int c0[4];
        ld4(val + 128 * c, v0);
        ld4(col + 128 * c, c0);
#pragma unroll
        for (int j = 0; j < 4; ++j) a0 += (double)v0[j] * (double)x[c0[j]];
    }
    return a0 + a1;
}

// The first slice of part b of `parts`, which hold about the same number of stored entries
template <class T>
__device__ __forceinline__ long long sell_cut(const Sell<T>& A, unsigned b, unsigned parts) {
    if (b == 0) return 0;
    if (b >= parts) return A.nslices;
    const long long total = A.sptr[A.nslices - 1] + 32LL * A.slen[A.nslices - 1];
    const long long want = total * b / parts;
    long long lo = 0, hi = A.nslices;  // first slice that starts at or after want
    while (lo < hi) {
        const long long mid = (lo + hi) >> 1;
        if (A.sptr[mid] < want) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// The row product of the solvers' iterations: FP32 values with 16-bit steps are software-pipelined.
// (x is read with ordinary loads: kernels that hold several iterations write it in between.)
template <bool C16, class TM, class T>
__device__ __forceinline__ double sell_product(const Sell<TM>& A, long long s, int lane, const T* x) {
    if constexpr (C16 && sizeof(TM) == 4) return sell_row16_pipe(A, s, lane, x);
    else return sell_row<C16>(A, s, lane, x);
}

}  // namespace lsmps_gpu
