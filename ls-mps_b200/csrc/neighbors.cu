// Uniform-grid neighbor build and 14-direction classification on sm_100a.
//
// Semantics follow the reference's neighbors() and classify() (src/lsmps.cpp:16-18,26-27)
// bit for bit; the data flow is the GPU's own:
//   1. cell coordinates floor(r / re) (IEEE division) and their bounding box;
//   2. a counting sort of particles into a dense cell grid (atomic slots, scan), then
//      each cell's members sorted by particle index, so that every 3-cell x-row of the grid
//      is one contiguous, index-ascending range of the sorted arrays;
//   3. a scan of every cell's 9 contiguous candidate rows by one warp (FP32 with a guard band,
//      exact FP64 near the cutoff) into per-particle slot rows, packed into the CSR once the
//      counts are scanned; or, where the slot rows would not fit, a count pass and a fill pass.
//      Taking the 9 rows in (dz, dy) order with candidates in sorted order is exactly the
//      reference's order (27 cells dz, dy, dx; ascending index in a cell), so the sorted column
//      indices of a row ascend and the first max_neighbors are the ones the reference keeps.
//      The scan (or the fill pass) fuses the classification over the kept list.
// Distances use __dadd_rn/__dmul_rn: the reference evaluates (dx*dx + dy*dy) + dz*dz
// without fused multiply-adds, and the acceptance test d^2 < re^2 must match at the ulp.
#include <algorithm>
#include <cmath>
#include <climits>
#include <vector>

#include "ops.cuh"
#include "scan.cuh"

namespace lsmps_gpu {
namespace {

constexpr long long MAX_CELLS = 1ll << 29;   // 2 GiB of int32 cell starts
constexpr int SMALL_CELL = 64;                // in-place insertion sort up to this occupancy
constexpr int BIG_CELL_MAX = 8192;            // shared-memory bitonic sort up to this occupancy
constexpr int NB_WARPS = 8;                   // warps (= particles) per block in the passes
constexpr double SLOT_BUDGET_BYTES = 4e9;     // slot rows of the single-pass build (n x maxn x 4 B)

// ---- 1. cell coordinates --------------------------------------------------------------
__global__ void k_cell_coords(const double* __restrict__ pos, size_t n, double re,
                              int3* __restrict__ cell, int* bounds, int* dflag) {
    int mn[3] = {INT_MAX, INT_MAX, INT_MAX}, mx[3] = {INT_MIN, INT_MIN, INT_MIN};
    bool bad = false;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        double c[3];
        int ci[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            double v = pos[3 * i + a];
            c[a] = floor(xdiv(v, re));
            if (!isfinite(c[a]) || fabs(c[a]) > (double)(1 << 30)) { bad = true; c[a] = 0; }
            ci[a] = (int)c[a];
            mn[a] = min(mn[a], ci[a]);
            mx[a] = max(mx[a], ci[a]);
        }
        cell[i] = make_int3(ci[0], ci[1], ci[2]);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mn[a] = min(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
            mx[a] = max(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
        }
    }
    // the block's bounds, then six atomics per block (per-warp atomics on the same six words
    // serialise in L2: ~9.5k per word at 1M particles)
    __shared__ int sb[6][32];
    const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            sb[a][warp] = mn[a];
            sb[3 + a][warp] = mx[a];
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int a = threadIdx.x;
        int v = sb[a][0];
        for (int w = 1; w < nwarps; ++w) v = a < 3 ? min(v, sb[a][w]) : max(v, sb[a][w]);
        if (a < 3 ? v != INT_MAX : v != INT_MIN) {
            if (a < 3) atomicMin(&bounds[a], v);
            else atomicMax(&bounds[a], v);
        }
    }
    if (bad) atomicOr(dflag, DFLAG_NONFINITE);
}

// ---- 2. counting sort -------------------------------------------------------------------
__global__ void k_cell_count(const int3* __restrict__ cell, size_t n, int3 g0, int3 gd,
                             int* __restrict__ lin_out, int* __restrict__ slot, int* __restrict__ count) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    int3 c = cell[i];
    int lin = ((c.z - g0.z) * gd.y + (c.y - g0.y)) * gd.x + (c.x - g0.x);
    lin_out[i] = lin;
    slot[i] = atomicAdd(&count[lin], 1);
}

__global__ void k_scatter(const int* __restrict__ lin, const int* __restrict__ slot, size_t n,
                          const int* __restrict__ cell_start, int* __restrict__ perm) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    perm[cell_start[lin[i]] + slot[i]] = (int)i;
}

// Atomic slots leave a cell's members in arbitrary order; restore ascending index (cells of up
// to 32 members sorted in registers, up to SMALL_CELL in place).
// Ascending bitonic sort of N (a power of two) values held in registers (the loops unroll to
// fixed indices).
template <int N>
__device__ __forceinline__ void bitonic_sort_regs(int (&v)[N]) {
#pragma unroll
    for (int k = 2; k <= N; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const int l = i ^ j;
                if (l > i) {
                    const int a = v[i], c = v[l];
                    const bool asc = (i & k) == 0;
                    v[i] = asc ? min(a, c) : max(a, c);
                    v[l] = asc ? max(a, c) : min(a, c);
                }
            }
}

// A cell's members (occ <= N, distinct indices) sorted ascending in registers: all loads in
// flight at once, padding INT_MAX sorts last.
template <int N>
__device__ __forceinline__ void sort_cell_regs(int* __restrict__ perm, int b, int occ) {
    int v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = i < occ ? perm[b + i] : INT_MAX;
    bitonic_sort_regs<N>(v);
#pragma unroll
    for (int i = 0; i < N; ++i)
        if (i < occ) perm[b + i] = v[i];
}

__global__ void k_sort_small_cells(const int* __restrict__ cell_start, long long ncells,
                                   int* __restrict__ perm, int* big_list, int* big_count,
                                   int* max_occ) {
    long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    int occ = 0;
    if (c < ncells) {
        int b = cell_start[c], e = cell_start[c + 1];
        occ = e - b;
        if (occ > SMALL_CELL) {
            int slot = atomicAdd(big_count, 1);
            big_list[slot] = (int)c;
        } else if (occ > 1 && occ <= 16) {
            sort_cell_regs<16>(perm, b, occ);
        } else if (occ > 1 && occ <= 32) {
            sort_cell_regs<32>(perm, b, occ);
        } else if (occ > 1) {
            for (int a = b + 1; a < e; ++a) {
                int v = perm[a];
                int t = a - 1;
                while (t >= b && perm[t] > v) {
                    perm[t + 1] = perm[t];
                    --t;
                }
                perm[t + 1] = v;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) occ = max(occ, __shfl_xor_sync(0xffffffffu, occ, o));
    // one atomic per block (per-warp atomics on one word serialise in L2)
    __shared__ int socc[32];
    if ((threadIdx.x & 31) == 0) socc[threadIdx.x >> 5] = occ;
    __syncthreads();
    if (threadIdx.x == 0) {
        int m = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = max(m, socc[w]);
        if (m > 0) atomicMax(max_occ, m);
    }
}

// One block per crowded cell: bitonic sort in shared memory (padding with INT_MAX).
__global__ void __launch_bounds__(1024) k_sort_big_cells(const int* __restrict__ cell_start,
                                                         int* __restrict__ perm,
                                                         const int* __restrict__ big_list,
                                                         const int* big_count, int* dflag) {
    __shared__ int s[BIG_CELL_MAX];
    int nbig = *big_count;
    for (int bi = blockIdx.x; bi < nbig; bi += gridDim.x) {
        int c = big_list[bi];
        int b = cell_start[c], e = cell_start[c + 1], occ = e - b;
        if (occ > BIG_CELL_MAX) {
            if (threadIdx.x == 0) atomicOr(dflag, DFLAG_CELL_OVERFLOW);
            continue;
        }
        int len = 1;
        while (len < occ) len <<= 1;
        for (int t = threadIdx.x; t < len; t += blockDim.x) s[t] = t < occ ? perm[b + t] : INT_MAX;
        __syncthreads();
        for (int k = 2; k <= len; k <<= 1) {
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int t = threadIdx.x; t < len; t += blockDim.x) {
                    int p = t ^ j;
                    if (p > t) {
                        bool up = (t & k) == 0;
                        int a = s[t], d = s[p];
                        if ((a > d) == up) { s[t] = d; s[p] = a; }
                    }
                }
                __syncthreads();
            }
        }
        for (int t = threadIdx.x; t < occ; t += blockDim.x) perm[b + t] = s[t];
        __syncthreads();
    }
}

__global__ void k_gather_sorted(const int* __restrict__ perm, size_t n, const double* __restrict__ pos,
                                const uint8_t* __restrict__ type_in, const int* __restrict__ lin,
                                double* __restrict__ sx, double* __restrict__ sy, double* __restrict__ sz,
                                uint8_t* __restrict__ stype, int* __restrict__ scell, int* __restrict__ iperm) {
    size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    int i = perm[k];
    sx[k] = pos[3 * (size_t)i];
    sy[k] = pos[3 * (size_t)i + 1];
    sz[k] = pos[3 * (size_t)i + 2];
    stype[k] = type_in[i];
    scell[k] = lin[i];
    iperm[i] = (int)k;
}

// ---- 3. count / fill passes ---------------------------------------------------------------
struct GridView {
    const int* cell_start;
    int nx, ny, nz;
};

// Candidate range of row (dz, dy) around cell (cx, cy, cz): cells x-1..x+1 of that row.
__device__ __forceinline__ bool row_range(const GridView& g, int cx, int cy, int cz, int dy, int dz,
                                          int& beg, int& end) {
    int y = cy + dy, z = cz + dz;
    if (y < 0 || y >= g.ny || z < 0 || z >= g.nz) return false;
    int xlo = max(cx - 1, 0), xhi = min(cx + 1, g.nx - 1);
    int base = (z * g.ny + y) * g.nx;
    beg = g.cell_start[base + xlo];
    end = g.cell_start[base + xhi + 1];
    return beg < end;
}

__device__ __forceinline__ unsigned sector_bits(double dx, double dy, double dz) {
    double ax = fabs(dx), ay = fabs(dy), az = fabs(dz);
    int s = (ax >= ay && ax >= az) ? (dx >= 0 ? 0 : 1)
                                   : ((ay >= ax && ay >= az) ? (dy >= 0 ? 2 : 3) : (dz >= 0 ? 4 : 5));
    int o = 6 + (dx >= 0) + 2 * (dy >= 0) + 4 * (dz >= 0);
    return (1u << s) | (1u << o);
}

// The reference's decision (src/lsmps.cpp:27) from the kept count and sector mask.
__device__ __forceinline__ uint8_t classify_rule(uint8_t tin, int kept, unsigned sectors_mask, double z,
                                                 double l0) {
    if (tin == LSMPS_WALL) return LSMPS_WALL;
    if (kept < 10) return LSMPS_SPLASH;
    int sectors = __popc(sectors_mask);
    if (z < xmul(1.5, l0)) return LSMPS_NEAR_WALL;
    if (sectors < 11) return LSMPS_FREE_SURFACE;
    return LSMPS_INTERIOR;
}

// Global-memory form of one query (one warp): count / fill the accepted candidates of
// sorted particle k; used by the staged kernels when a segment's neighborhood does not fit
// in shared memory.
__device__ __forceinline__ int count_query_global(const GridView& g, const double* __restrict__ sx,
                                                  const double* __restrict__ sy, const double* __restrict__ sz,
                                                  const int* __restrict__ scell, int k, double re2, int lane) {
    int lin = scell[k];
    int cx = lin % g.nx, t = lin / g.nx, cy = t % g.ny, cz = t / g.ny;
    double xi = sx[k], yi = sy[k], zi = sz[k];
    int count = 0;
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy) {
            int beg, end;
            if (!row_range(g, cx, cy, cz, dy, dz, beg, end)) continue;
            for (int mb = beg; mb < end; mb += 32) {
                int m = mb + lane;
                bool ok = false;
                if (m < end && m != k) ok = xnorm2(xsub(sx[m], xi), xsub(sy[m], yi), xsub(sz[m], zi)) < re2;
                count += __popc(__ballot_sync(0xffffffffu, ok));
            }
        }
    return count;
}

__device__ __forceinline__ void fill_query_global(const GridView& g, const double* __restrict__ sx,
                                                  const double* __restrict__ sy, const double* __restrict__ sz,
                                                  const int* __restrict__ scell, const uint8_t* __restrict__ stype,
                                                  int k, double re2, int maxn, double l0, int classify,
                                                  const int* __restrict__ row, int* __restrict__ col,
                                                  uint8_t* __restrict__ cls, int lane) {
    unsigned lt = (1u << lane) - 1u;
    int lin = scell[k];
    int cx = lin % g.nx, t = lin / g.nx, cy = t % g.ny, cz = t / g.ny;
    double xi = sx[k], yi = sy[k], zi = sz[k];
    int out0 = row[k];
    const int room = row[k + 1] - out0;  // = min(count, maxn) from the count pass
    int written = 0;
    unsigned sec = 0;
    for (int dz = -1; dz <= 1 && written < maxn; ++dz)
        for (int dy = -1; dy <= 1 && written < maxn; ++dy) {
            int beg, end;
            if (!row_range(g, cx, cy, cz, dy, dz, beg, end)) continue;
            for (int mb = beg; mb < end && written < maxn; mb += 32) {
                int m = mb + lane;
                bool ok = false;
                double dx = 0, dyv = 0, dzv = 0;
                if (m < end && m != k) {
                    dx = xsub(sx[m], xi);
                    dyv = xsub(sy[m], yi);
                    dzv = xsub(sz[m], zi);
                    ok = xnorm2(dx, dyv, dzv) < re2;
                }
                unsigned bal = __ballot_sync(0xffffffffu, ok);
                if (ok) {
                    int p = written + __popc(bal & lt);
                    if (p < maxn && p < room) {
                        col[out0 + p] = m;
                        if (classify) sec |= sector_bits(dx, dyv, dzv);
                    }
                }
                written += __popc(bal);
            }
        }
    if (classify) {
        sec = __reduce_or_sync(0xffffffffu, sec);
        if (lane == 0) cls[k] = classify_rule(stype[k], min(written, maxn), sec, zi, l0);
    }
}

// ---- staged passes: one block per segment of SEG cells along x, one thread per particle -----
// The block copies the candidates of its 9 cell rows (cells cx0-1 .. cx1+1 of rows (cy+dy,
// cz+dz)) into shared memory once, as FP32 positions relative to the segment's corner, plus
// the row pointers of its own particles (a contiguous range of the sorted arrays). Each
// thread then walks one particle's 9 row ranges (cells cx-1 .. cx+1 of each row, contiguous
// in the sorted order) candidate by candidate, so its kept list comes out in the reference's
// order without any cross-lane bookkeeping. Cells whose box is farther than re (plus a 1e-4
// relative margin) are skipped. A candidate is accepted when its FP32 distance^2 is below
// re^2 (1 - 2e-5) and rejected above re^2 (1 + 2e-5); in between the exact FP64 test on the
// global positions decides. Coordinates lie within (SEG + 2) re of the corner, so the FP32
// distance^2 is within 1e-5 re^2 of the exact one and the kept lists are the reference's bit
// for bit. The sector bits of the classification use the FP32 differences when every sign
// and |d| comparison they need is separated by more than 4e-6 re, else the exact FP64 ones.
constexpr int SEG = 12;
constexpr int SEG_THREADS = 128;
constexpr int SEG_MAXC = 1536;  // staged candidates (24 KB)
constexpr int SEG_MAXQ = 512;   // queries per segment

struct SegGrid {
    GridView g;
    int3 g0;   // grid origin cell
    double re;
    int nsegx;
};

// The decisions are safe when no component is within `margin` of zero and the largest is that far
// above the other two (not so when two of them are beyond the FP32 range).
__device__ __forceinline__ bool sector_bits_f32(float dx, float dy, float dz, float margin, unsigned& bits) {
    const float ax = fabsf(dx), ay = fabsf(dy), az = fabsf(dz);
    const float lo = fminf(ax, ay), hi = fmaxf(ax, ay), top = fmaxf(hi, az);
    if (!(fminf(lo, az) > margin) || !(top - fmaxf(lo, fminf(hi, az)) > margin)) {
        bits = 0;
        return false;
    }
    const unsigned sx = __float_as_uint(dx) >> 31, sy = __float_as_uint(dy) >> 31, sz = __float_as_uint(dz) >> 31;
    const unsigned s = az == top ? 4 + sz : (ay == top ? 2 + sy : sx);
    bits = (1u << s) | ((1u << 13) >> (sx + 2 * sy + 4 * sz));
    return true;
}

// Non-empty segments of the grid, listed in any order (each segment's outputs are addressed
// by its own particles, so the order does not affect the result).
__global__ void k_list_segments(SegGrid G, long long nseg, int* __restrict__ list, int* __restrict__ count) {
    const long long seg = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    bool nonempty = false;
    if (seg < nseg) {
        const int sxi = (int)(seg % G.nsegx);
        const long long tt = seg / G.nsegx;
        const int cy = (int)(tt % G.g.ny), cz = (int)(tt / G.g.ny);
        const int cx0 = sxi * SEG, cx1 = min(cx0 + SEG, G.g.nx) - 1;
        const int rowlin = (cz * G.g.ny + cy) * G.g.nx;
        nonempty = G.g.cell_start[rowlin + cx0] != G.g.cell_start[rowlin + cx1 + 1];
    }
    const unsigned bal = __ballot_sync(0xffffffffu, nonempty);
    int base = 0;
    if ((threadIdx.x & 31) == 0 && bal) base = atomicAdd(count, __popc(bal));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (nonempty) list[base + __popc(bal & ((1u << (threadIdx.x & 31)) - 1u))] = (int)seg;
}

// One accepted-or-band candidate of the thread's query (the rare path of the scan).
template <bool FILL>
__device__ __forceinline__ void seg_accept(float d2, float lo_th, float dx, float dy, float dz, int m, int k,
                                           const double* __restrict__ sx, const double* __restrict__ sy,
                                           const double* __restrict__ sz, double re2, int maxn, int room, int out0,
                                           int classify, float margin, int* __restrict__ col, int& written,
                                           unsigned& sec) {
    if (m == k) return;
    if (d2 >= lo_th && !(xnorm2(xsub(sx[m], sx[k]), xsub(sy[m], sy[k]), xsub(sz[m], sz[k])) < re2)) return;
    if (FILL && written < maxn && written < room) {
        col[out0 + written] = m;
        if (classify) {
            unsigned bb;
            if (!sector_bits_f32(dx, dy, dz, margin, bb))
                bb = sector_bits(xsub(sx[m], sx[k]), xsub(sy[m], sy[k]), xsub(sz[m], sz[k]));
            sec |= bb;
        }
    }
    ++written;
}

template <bool FILL>
__global__ void __launch_bounds__(SEG_THREADS, 8) k_seg_pass(SegGrid G, const int* __restrict__ seg_list,
                                                            const double* __restrict__ sx,
                                                            const double* __restrict__ sy,
                                                            const double* __restrict__ sz,
                                                            const int* __restrict__ scell,
                                                            const uint8_t* __restrict__ stype, double re2,
                                                            int maxn, double l0, int classify,
                                                            int* __restrict__ cnt,
                                                            unsigned long long* trunc_total,
                                                            const int* __restrict__ row, int* __restrict__ col,
                                                            uint8_t* __restrict__ cls) {
    __shared__ float4 cf[SEG_MAXC];
    __shared__ int qrow[SEG_MAXQ + 1];
    __shared__ int rbase[10], rfirst[9], rcs[9][SEG + 3];
    const float re_f = (float)G.re;
    const float re2f = (float)re2;
    const float lo_th = re2f * (1.f - 2e-5f), hi_th = re2f * (1.f + 2e-5f);
    const float cull = re2f * (1.f + 1e-4f);
    const float margin = 4e-6f * re_f;
    const int seg = seg_list[blockIdx.x];
    const int sxi = seg % G.nsegx, tt = seg / G.nsegx, cy = tt % G.g.ny, cz = tt / G.g.ny;
    const int cx0 = sxi * SEG, cx1 = min(cx0 + SEG, G.g.nx) - 1;
    const int lo = max(cx0 - 1, 0), hi = min(cx1 + 1, G.g.nx - 1);
    const int rowlin = (cz * G.g.ny + cy) * G.g.nx;
    const int q0 = G.g.cell_start[rowlin + cx0], q1 = G.g.cell_start[rowlin + cx1 + 1];
    for (int t = threadIdx.x; t < 9 * (SEG + 3); t += blockDim.x) {
        const int r = t / (SEG + 3), c = lo + t % (SEG + 3);
        const int y = cy + (r % 3 - 1), z = cz + (r / 3 - 1);
        int v = 0;
        if (y >= 0 && y < G.g.ny && z >= 0 && z < G.g.nz && c <= hi + 1) v = G.g.cell_start[(z * G.g.ny + y) * G.g.nx + c];
        rcs[r][c - lo] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        rbase[0] = 0;
        for (int r = 0; r < 9; ++r) {
            rfirst[r] = rcs[r][0];
            rbase[r + 1] = rbase[r] + (rcs[r][hi + 1 - lo] - rcs[r][0]);
        }
    }
    __syncthreads();
    const int total = rbase[9];
    if (total > SEG_MAXC || q1 - q0 > SEG_MAXQ) {
        // crowded neighborhood: the global-memory form, one query per warp
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        for (int k = q0 + warp; k < q1; k += SEG_THREADS / 32) {
            if (FILL) {
                fill_query_global(G.g, sx, sy, sz, scell, stype, k, re2, maxn, l0, classify, row, col, cls, lane);
            } else {
                int c = count_query_global(G.g, sx, sy, sz, scell, k, re2, lane);
                if (lane == 0) {
                    cnt[k] = min(c, maxn);
                    if (c > maxn) atomicAdd(trunc_total, (unsigned long long)(c - maxn));
                }
            }
        }
        return;
    }
    const double ox = (G.g0.x + cx0) * G.re, oy = (G.g0.y + cy) * G.re, oz = (G.g0.z + cz) * G.re;
    for (int r = 0; r < 9; ++r) {  // row by row: consecutive threads load consecutive particles
        const int n_r = rbase[r + 1] - rbase[r], f = rfirst[r], b = rbase[r];
        for (int i = threadIdx.x; i < n_r; i += blockDim.x)
            cf[b + i] = make_float4((float)(sx[f + i] - ox), (float)(sy[f + i] - oy), (float)(sz[f + i] - oz), 0.f);
    }
    if (FILL)
        for (int i = threadIdx.x; i <= q1 - q0; i += blockDim.x) qrow[i] = row[q0 + i];
    __syncthreads();
    for (int k = q0 + threadIdx.x; k < q1; k += blockDim.x) {
        int ck = cx0;
        while (ck < cx1 && k >= rcs[4][ck + 1 - lo]) ++ck;
        const float4 qf = cf[rbase[4] + (k - rfirst[4])];  // the query is staged in the centre row
        const float qx = qf.x - (ck - cx0) * re_f;          // position inside its own cell (x)
        int written = 0, out0 = 0, room = 0;
        unsigned sec = 0;
        if (FILL) {
            out0 = qrow[k - q0];
            room = qrow[k - q0 + 1] - out0;
        }
        for (int r = 0; r < 9; ++r) {
            const int dy = r % 3 - 1, dz = r / 3 - 1;
            const float gy = dy < 0 ? qf.y : (dy > 0 ? re_f - qf.y : 0.f);
            const float gz = dz < 0 ? qf.z : (dz > 0 ? re_f - qf.z : 0.f);
            const float gyz = gy * gy + gz * gz;
            if (gyz > cull) continue;
            // cells ck-1 .. ck+1 of this row, each kept when its box is within re
            int clo = max(ck - 1, lo), chi = min(ck + 1, hi);
            if (clo < ck && gyz + qx * qx > cull) clo = ck;
            if (chi > ck && gyz + (re_f - qx) * (re_f - qx) > cull) chi = ck;
            const int gb = rcs[r][clo - lo], ge = rcs[r][chi + 1 - lo];
            const int sb = rbase[r] + (gb - rfirst[r]);
            const int se = sb + (ge - gb);
            const int mshift = rfirst[r] - rbase[r];  // global index = staged index + mshift
            int si = sb;
            for (; si + 4 <= se; si += 4) {
                float d2[4], ddx[4], ddy[4], ddz[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float4 cj = cf[si + u];
                    ddx[u] = cj.x - qf.x;
                    ddy[u] = cj.y - qf.y;
                    ddz[u] = cj.z - qf.z;
                    d2[u] = ddx[u] * ddx[u] + ddy[u] * ddy[u] + ddz[u] * ddz[u];
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (d2[u] <= hi_th)
                        seg_accept<FILL>(d2[u], lo_th, ddx[u], ddy[u], ddz[u], si + u + mshift, k, sx, sy, sz, re2,
                                         maxn, room, out0, classify, margin, col, written, sec);
            }
            for (; si < se; ++si) {
                const float4 cj = cf[si];
                const float dx = cj.x - qf.x, dyf = cj.y - qf.y, dzf = cj.z - qf.z;
                const float d2 = dx * dx + dyf * dyf + dzf * dzf;
                if (d2 <= hi_th)
                    seg_accept<FILL>(d2, lo_th, dx, dyf, dzf, si + mshift, k, sx, sy, sz, re2, maxn, room, out0,
                                     classify, margin, col, written, sec);
            }
        }
        if (FILL) {
            if (classify) cls[k] = classify_rule(stype[k], min(written, maxn), sec, sz[k], l0);
        } else {
            cnt[k] = min(written, maxn);
            if (written > maxn) atomicAdd(trunc_total, (unsigned long long)(written - maxn));
        }
    }
}

// ---- single pass: each query's kept list straight into its slot row ------------------------
// One warp per cell and 32 of its particles (the queries). The cell's candidates, the particles
// of its 27 cells in the reference's order (9 rows of three cells, contiguous in the sorted
// order), go into registers, one per lane and chunk of 32, as FP32 positions relative to the
// cell's corner in units of re (so that neither they nor their squares leave the FP32 range, and an
// empty lane's marker lies far outside the radius, whatever re is). The warp then takes the queries
// one by one: every lane tests its candidates with packed FP32x2 arithmetic, the ballots of a
// chunk are the hits in order, the hits are packed into shared memory and from there, a lane each,
// written to slots[k * maxn + p] for p < maxn, with their sector bits for the classification. A
// query with a candidate in the guard band of k_seg_pass (|d^2 - re^2| <= 2.1e-5 re^2; the FP32
// distance^2 is within 3e-6 re^2 of the exact one, out to 2^31 cells from the origin) has its hits
// there decided exactly in FP64, so the kept lists are the reference's bit for bit. Cells of more
// than SCAN_CH chunks take them in turns. Counting continues past maxn for the truncation
// statistic. k_slots_compact then packs the slot rows into the CSR once the kept counts are scanned.
// What bounds it: issue slots (70 % busy) and the latency of a query's chain (ballots, packing,
// sector bits) at 16 warps per SM; two queries at a time hide half of the latter (one at a time took
// 518 us at 1M when two took 479). It took the place of a block per 12-cell segment with a thread
// per query, which was bound by shared memory (24 bytes per candidate pair and lane) and by the
// divergent walk over each thread's hits, with 23 (mixed set) to 39 % (rain) of its warps' lanes
// idle: 532 us for 1M particles of a mixed set (470 now), 172 us for 200k of a rain set (107) and
// 890 for 1M at radius 2.3 (490). Five blocks per SM (102
// registers, spilled) took 499 us, three 565. The sector bits are left out where the rule does not
// read them (walls, a third of a rain set: 513 -> 496 us).
constexpr int SCAN_CH = 10;     // chunks of 32 candidates in registers (a cell of side 2.1 has 250 candidates)
constexpr int SCAN_WARPS = 4;   // per block

// The scan's FP32 limits on d^2 / re^2: above hi no neighbor, below lo one, between them the exact
// test; queries with a candidate within `band` of 1 look.
struct ScanBand {
    float lo, hi, band;
};

// Items of the scan (cell x, y, z and first query), in any order (an item's outputs are addressed by
// its own particles): every 32nd particle of a cell makes one. items[0].x is their number,
// items[0].y how many the scan has drawn. rel: each particle's position relative to its cell's
// corner in units of re, and the cell's x index. (One thread per particle: with one per cell of the
// dense grid a build of 100k particles over 512M cells took 7.4 ms, now 5.9. One addition to the
// count per block: per warp it cost a 1M build 12 us.)
__global__ void __launch_bounds__(256) k_scan_prep(GridView g, int3 g0, double re, int n, const int* __restrict__ scell,
                            const double* __restrict__ sx, const double* __restrict__ sy,
                            const double* __restrict__ sz, int4* __restrict__ items, float4* __restrict__ rel) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    int cx = 0, cy = 0, cz = 0;
    bool first = false;
    if (t < n) {
        const int lin = scell[t], u = lin / g.nx;
        cx = lin % g.nx, cy = u % g.ny, cz = u / g.ny;
        rel[t] = make_float4((float)((sx[t] - (g0.x + cx) * re) / re), (float)((sy[t] - (g0.y + cy) * re) / re),
                             (float)((sz[t] - (g0.z + cz) * re) / re), __int_as_float(cx));
        first = (((int)t - g.cell_start[lin]) & 31) == 0;
    }
    __shared__ int before[9];  // items of the block's warps in front, then the block's first place
    const unsigned m = __ballot_sync(0xffffffffu, first);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) before[warp] = __popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
        int sum = 0;
        for (int w = 0; w < 8; ++w) {
            const int c = before[w];
            before[w] = sum;
            sum += c;
        }
        before[8] = sum ? atomicAdd(&items[0].x, sum) + 1 : 0;
    }
    __syncthreads();
    if (first) items[before[8] + before[warp] + __popc(m & ((1u << lane) - 1u))] = make_int4(cx, cy, cz, (int)t);
}

__global__ void __launch_bounds__(32 * SCAN_WARPS, 4) k_cell_scan(
    GridView g, int n, int4* __restrict__ items, const float4* __restrict__ rel, const double* __restrict__ sx,
    const double* __restrict__ sy, const double* __restrict__ sz, const uint8_t* __restrict__ stype, ScanBand lim,
    double re2, int maxn, double l0, int classify, int* __restrict__ cnt, unsigned long long* trunc_total,
    int* __restrict__ slots, uint8_t* __restrict__ cls) {
    __shared__ float4 packed[SCAN_WARPS][2 * 32 * SCAN_CH];  // two queries' hits: position and index
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    float4* hits = packed[warp];
    constexpr float margin = 4e-6f;  // units of re, as lim
    const int nitems = items[0].x;
    // An item's number, cell, row ranges and candidates are four dependent loads: the first three
    // are made one to three items ahead. The first items go by the warp's number, the others are
    // drawn from a counter.
    const int first = blockIdx.x * SCAN_WARPS + warp;
    int drawn = 0;  // in lane 0
    auto draw = [&] {
        if (lane == 0) drawn = gridDim.x * SCAN_WARPS + atomicAdd(&items[0].y, 1);
    };
    auto after = [&] {
        const int it = __shfl_sync(0xffffffffu, drawn, 0);
        draw();
        return it;
    };
    draw();
    auto cell_of = [&](int it) { return it < nitems ? items[it + 1] : make_int4(-1, 0, 0, 0); };
    struct Head {
        int cx, qb, nq, beg, len;  // beg, len: row r of the candidates in lane r < 9
        float4 me;                 // lane q < nq: query qb + q
        double z;
        uint8_t type;
    };
    auto head_of = [&](int4 item) {
        Head h{item.x, item.w, 0, 0, 0, {}, 0.0, LSMPS_WALL};
        if (item.x < 0) return h;
        h.nq = min(32, g.cell_start[(item.z * g.ny + item.y) * g.nx + item.x + 1] - item.w);
        if (lane < 9) {
            int end = 0;
            if (row_range(g, item.x, item.y, item.z, lane % 3 - 1, lane / 3 - 1, h.beg, end)) h.len = end - h.beg;
        }
        const int k = min(item.w + lane, n - 1);  // (lanes past nq load another particle's)
        h.me = rel[k];
        if (classify) h.type = stype[k], h.z = sz[k];
        return h;
    };
    Head next = head_of(cell_of(first));
    int4 item1 = cell_of(after());
    while (next.nq > 0) {
        const Head H = next;
        next = head_of(item1);
        item1 = cell_of(after());
        const int cx = H.cx, qb = H.qb, nq = H.nq;
        int pre = H.len;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += v;
        }
        const int total = __shfl_sync(0xffffffffu, pre, 8);
        const int shift = H.beg - (pre - H.len);  // candidate index to particle
        int start[9];                             // where the rows start among the candidates
#pragma unroll
        for (int r = 1; r < 9; ++r) start[r] = __shfl_sync(0xffffffffu, pre, r - 1);
        // the rule reads the sectors of fluid particles above the wall layer only
        const unsigned need = __ballot_sync(0xffffffffu, H.type != LSMPS_WALL && !(H.z < xmul(1.5, l0)));
        int written = 0;
        unsigned sec = 0;
        for (int c0 = 0; c0 < total; c0 += 32 * SCAN_CH) {
            float x[SCAN_CH], y[SCAN_CH], z[SCAN_CH];
            int m[SCAN_CH];
#pragma unroll
            for (int c = 0; c < SCAN_CH; ++c) {
                const int b = c0 + 32 * c, j = b + lane;
                x[c] = y[c] = z[c] = 1e18f;  // no candidate: far away
                m[c] = -1;
                if (b < total) {
                    int r = 0;
#pragma unroll
                    for (int t = 1; t < 9; ++t) r += j >= start[t] ? 1 : 0;
                    const int mm = j + __shfl_sync(0xffffffffu, shift, r);
                    if (j < total) {
                        const float4 p = rel[mm];
                        m[c] = mm;
                        x[c] = p.x + (float)(__float_as_int(p.w) - cx);
                        y[c] = p.y + (float)(r % 3 - 1);
                        z[c] = p.z + (float)(r / 3 - 1);
                    }
                }
            }
            // two queries at a time, so that one's chain of ballot, packing and sector bits fills the
            // other's waits (an odd last query goes twice, the second time without results)
            for (int q = 0; q < nq; q += 2) {
                float qx[2], qy[2], qz[2], near = 1.f;
                unsigned bal[2][SCAN_CH];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int from = min(q + h, nq - 1);
                    qx[h] = __shfl_sync(0xffffffffu, H.me.x, from);
                    qy[h] = __shfl_sync(0xffffffffu, H.me.y, from);
                    qz[h] = __shfl_sync(0xffffffffu, H.me.z, from);
                }
#pragma unroll
                for (int c = 0; c < SCAN_CH; c += 2) {
                    bal[0][c] = bal[0][c + 1] = bal[1][c] = bal[1][c + 1] = 0;
                    if (c0 + 32 * c < total) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float2 dx = __fadd2_rn(make_float2(x[c], x[c + 1]), make_float2(-qx[h], -qx[h]));
                            const float2 dy = __fadd2_rn(make_float2(y[c], y[c + 1]), make_float2(-qy[h], -qy[h]));
                            const float2 dz = __fadd2_rn(make_float2(z[c], z[c + 1]), make_float2(-qz[h], -qz[h]));
                            float2 d2 = __fmul2_rn(dx, dx);
                            d2 = __ffma2_rn(dy, dy, d2);
                            d2 = __ffma2_rn(dz, dz, d2);
                            const float2 o = __fadd2_rn(d2, make_float2(-1.f, -1.f));
                            near = fminf(near, fminf(fabsf(o.x), fabsf(o.y)));
                            bal[h][c] = __ballot_sync(0xffffffffu, d2.x <= lim.hi && m[c] != qb + q + h);
                            bal[h][c + 1] = __ballot_sync(0xffffffffu, d2.y <= lim.hi && m[c + 1] != qb + q + h);
                        }
                    }
                }
                if (__any_sync(0xffffffffu, near <= lim.band)) {
#pragma unroll 1
                    for (int h = 0; h < 2; ++h) {
                        const int kq = qb + min(q + h, nq - 1);
#pragma unroll
                        for (int c = 0; c < SCAN_CH; ++c) {
                            const unsigned old = h ? bal[1][c] : bal[0][c];
                            bool ok = (old >> lane) & 1u;
                            if (ok) {
                                const float dx = x[c] - (h ? qx[1] : qx[0]), dy = y[c] - (h ? qy[1] : qy[0]),
                                            dz = z[c] - (h ? qz[1] : qz[0]);
                                if (dx * dx + dy * dy + dz * dz >= lim.lo)
                                    ok = xnorm2(xsub(sx[m[c]], sx[kq]), xsub(sy[m[c]], sy[kq]),
                                                xsub(sz[m[c]], sz[kq])) < re2;
                            }
                            const unsigned now = __ballot_sync(0xffffffffu, ok);
                            if (h) bal[1][c] = now;
                            else bal[0][c] = now;
                        }
                    }
                }
                int w[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    w[h] = 0;
#pragma unroll
                    for (int c = 0; c < SCAN_CH; ++c) {
                        if ((bal[h][c] >> lane) & 1u)
                            hits[h * 32 * SCAN_CH + w[h] + __popc(bal[h][c] & lt)] =
                                make_float4(x[c], y[c], z[c], __int_as_float(m[c]));
                        w[h] += __popc(bal[h][c]);
                    }
                }
                __syncwarp();
                const bool two = q + 1 < nq;
                unsigned sb[2] = {0, 0};
                int w0[2];
                w0[0] = __shfl_sync(0xffffffffu, written, q);
                w0[1] = __shfl_sync(0xffffffffu, written, min(q + 1, 31));
                const int most = max(w[0], two ? w[1] : 0);
                for (int e = lane; e < most; e += 32) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (e < w[h] && e < maxn - w0[h] && (h == 0 || two)) {
                            const int kq = qb + q + h;
                            const float4 f = hits[h * 32 * SCAN_CH + e];
                            const int mh = __float_as_int(f.w);
                            slots[(size_t)kq * maxn + w0[h] + e] = mh;
                            if ((need >> (q + h)) & 1u) {
                                unsigned bb;
                                if (!sector_bits_f32(f.x - qx[h], f.y - qy[h], f.z - qz[h], margin, bb))
                                    bb = sector_bits(xsub(sx[mh], sx[kq]), xsub(sy[mh], sy[kq]), xsub(sz[mh], sz[kq]));
                                sb[h] |= bb;
                            }
                        }
                    }
                }
                const unsigned s0 = __reduce_or_sync(0xffffffffu, sb[0]), s1 = __reduce_or_sync(0xffffffffu, sb[1]);
                if (lane == q) {
                    written += w[0];
                    sec |= s0;
                }
                if (lane == q + 1 && two) {
                    written += w[1];
                    sec |= s1;
                }
                __syncwarp();
            }
        }
        if (lane < nq) {
            const int k = qb + lane;
            cnt[k] = min(written, maxn);
            if (written > maxn) atomicAdd(trunc_total, (unsigned long long)(written - maxn));
            if (classify) cls[k] = classify_rule(H.type, min(written, maxn), sec, H.z, l0);
        }
    }
}

// Packs the slot rows into the CSR: eight lanes per row, row k's kept list from
// slots[k * maxn] to col[row[k]].
__global__ void __launch_bounds__(256) k_slots_compact(int n, int maxn, const int* __restrict__ slots,
                                                       const int* __restrict__ row, int* __restrict__ col) {
    const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int k = (int)(g >> 3), sub = (int)(g & 7);
    if (k >= n) return;
    const int b = row[k], c = row[k + 1] - b;
    const int* src = slots + (size_t)k * maxn;
    for (int p = sub; p < c; p += 8) col[b + p] = __ldcs(src + p);
}

// Refresh of skin lists in one pass (eight lanes per particle): the candidates j != i of the
// candidate CSR (radius re + skin, ascending sorted index) that pass the build's exact FP64 test
// |r_j - r_i|^2 < re^2, in candidate order, go to the particle's slot row (the first maxn),
// with the sector bits of the kept ones for the classification; counting continues past maxn.
// The sector bits come from the FP32 rounding of the FP64 differences when every comparison
// they need is separated by more than `margin` (1e-6 re, the differences being below re and
// rounded to 6e-8 of themselves), else from the FP64 ones.
// Bound by instruction issue (70 % of the slots): with a warp per particle and every kept
// candidate's sector bits in FP64 it took 1,665 us for 3M particles (997 now; 1,100 with the bits
// of walls, which the rule does not read).
__global__ void __launch_bounds__(256) k_filter_slots(int n, const int* __restrict__ crow,
                                                      const int* __restrict__ ccol, const double* __restrict__ sx,
                                                      const double* __restrict__ sy, const double* __restrict__ sz,
                                                      const uint8_t* __restrict__ stype, double re2, float margin,
                                                      int maxn, double l0, int classify, int* __restrict__ slots,
                                                      int* __restrict__ cnt, unsigned long long* trunc,
                                                      uint8_t* __restrict__ cls) {
    const int lane = threadIdx.x & 31, sub = lane & 7;
    const long long step = (gridDim.x * (long long)blockDim.x) >> 3;
    // (the four particles of a warp go round together)
    for (long long i0 = (blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31)) >> 3; i0 < n; i0 += step) {
        const bool live = i0 + (lane >> 3) < n;
        const int i = live ? (int)(i0 + (lane >> 3)) : n - 1;
        const double xi = sx[i], yi = sy[i], zi = sz[i];
        const uint8_t ti = classify ? stype[i] : LSMPS_WALL;
        // the rule reads the sectors of fluid particles above the wall layer only
        const bool need = ti != LSMPS_WALL && !(zi < xmul(1.5, l0));
        const int c0 = crow[i], c1 = live ? crow[i + 1] : c0;
        int* out = slots + (size_t)i * maxn;
        int kept = 0;
        unsigned sec = 0;
        const int steps = __reduce_max_sync(0xffffffffu, (c1 - c0 + 7) >> 3);
        int jnext = c0 + sub < c1 ? ccol[c0 + sub] : 0;  // loaded one step ahead of its position
        for (int t = 0, e = c0 + sub; t < steps; ++t, e += 8) {
            const int j = jnext;
            jnext = e + 8 < c1 ? ccol[e + 8] : 0;
            bool ok = e < c1 && j != i;
            double dx = 0, dy = 0, dz = 0;
            if (ok) {
                dx = xsub(sx[j], xi);
                dy = xsub(sy[j], yi);
                dz = xsub(sz[j], zi);
                ok = xnorm2(dx, dy, dz) < re2;
            }
            const unsigned m = (__ballot_sync(0xffffffffu, ok) >> (lane & 24)) & 0xffu;
            const int p = kept + __popc(m & ((1u << sub) - 1u));
            if (ok && p < maxn) {
                out[p] = j;
                if (need) {
                    unsigned bb;
                    if (!sector_bits_f32((float)dx, (float)dy, (float)dz, margin, bb)) bb = sector_bits(dx, dy, dz);
                    sec |= bb;
                }
            }
            kept += __popc(m);
        }
        if (classify)
            for (int o = 4; o; o >>= 1) sec |= __shfl_xor_sync(0xffffffffu, sec, o);
        if (live && sub == 0) {
            cnt[i] = min(kept, maxn);
            if (kept > maxn) atomicAdd(trunc, (unsigned long long)(kept - maxn));
            if (classify) cls[i] = classify_rule(ti, min(kept, maxn), sec, zi, l0);
        }
    }
}

// Standalone classification over an existing CSR (warp per particle).
__global__ void __launch_bounds__(NB_WARPS * 32) k_classify(const double* __restrict__ sx,
                                                          const double* __restrict__ sy,
                                                          const double* __restrict__ sz,
                                                          const uint8_t* __restrict__ stype, int n,
                                                          double l0, const int* __restrict__ row,
                                                          const int* __restrict__ col,
                                                          uint8_t* __restrict__ cls) {
    int k = blockIdx.x * NB_WARPS + (threadIdx.x >> 5);
    if (k >= n) return;
    int lane = threadIdx.x & 31;
    double xi = sx[k], yi = sy[k], zi = sz[k];
    int b = row[k], e = row[k + 1];
    unsigned sec = 0;
    for (int p = b + lane; p < e; p += 32) {
        int m = col[p];
        sec |= sector_bits(xsub(sx[m], xi), xsub(sy[m], yi), xsub(sz[m], zi));
    }
    sec = __reduce_or_sync(0xffffffffu, sec);
    if (lane == 0) cls[k] = classify_rule(stype[k], e - b, sec, zi, l0);
}

// Histogram of kept counts and class counts (block-private in shared memory).
// stats layout (u64): [0..4] class counts, [5] truncated pairs, [6] max count,
// [8 .. 8+maxn] count histogram.
__global__ void k_nbr_stats(const int* __restrict__ cnt, const uint8_t* __restrict__ cls, int n, int maxn,
                            int have_cls, unsigned long long* stats) {
    extern __shared__ unsigned int sh[];
    unsigned int* hist = sh;              // maxn + 1
    unsigned int* tc = sh + maxn + 1;     // 5
    unsigned int* mxc = tc + 5;           // 1
    for (int t = threadIdx.x; t < maxn + 7; t += blockDim.x) sh[t] = 0;
    __syncthreads();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        int c = cnt[k];
        atomicAdd(&hist[c], 1u);
        atomicMax(mxc, (unsigned)c);
        if (have_cls) atomicAdd(&tc[cls[k] < 5 ? cls[k] : 0], 1u);
    }
    __syncthreads();
    for (int t = threadIdx.x; t <= maxn; t += blockDim.x)
        if (hist[t]) atomicAdd(&stats[8 + t], (unsigned long long)hist[t]);
    if (threadIdx.x < 5 && tc[threadIdx.x]) atomicAdd(&stats[threadIdx.x], (unsigned long long)tc[threadIdx.x]);
    if (threadIdx.x == 0) atomicMax(&stats[6], (unsigned long long)*mxc);
}

// ---- downloads in caller order ------------------------------------------------------------
__global__ void k_orig_counts(const int* __restrict__ iperm, const int* __restrict__ row, size_t n,
                              int* __restrict__ ocnt) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    int k = iperm[i];
    ocnt[i] = row[k + 1] - row[k];
}

__global__ void k_orig_fill(const int* __restrict__ iperm, const int* __restrict__ perm,
                            const int* __restrict__ row, const int* __restrict__ col, int n,
                            const int* __restrict__ orow, int* __restrict__ ocol) {
    int i = blockIdx.x * NB_WARPS + (threadIdx.x >> 5);
    if (i >= n) return;
    int lane = threadIdx.x & 31;
    int k = iperm[i];
    int b = row[k], e = row[k + 1], o = orow[i];
    for (int p = b + lane; p < e; p += 32) ocol[o + (p - b)] = perm[col[p]];
}

__global__ void k_orig_types(const int* __restrict__ iperm, const uint8_t* __restrict__ cls, size_t n,
                             uint8_t* __restrict__ out) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = cls[iperm[i]];
}

}  // namespace

// Percentiles as the reference computes them (src/lsmps.cpp:73): sort the counts and take
// cnt[(size_t)(q * (N - 1))], here from the count histogram.
static void fill_stats(lsmps_ctx* ctx, const std::vector<unsigned long long>& st, lsmps_neighbor_stats* out) {
    size_t n = ctx->n;
    lsmps_neighbor_stats s{};
    for (int t = 0; t < 5; ++t) s.type_count[t] = st[t];
    s.truncated = st[5];
    s.max_count = (int32_t)st[6];
    s.pairs = ctx->pairs;
    s.mean = n ? (double)ctx->pairs / (double)n : 0.0;
    auto pct = [&](double q) -> int {
        if (!n) return 0;
        size_t idx = (size_t)(q * (double)(n - 1));
        unsigned long long cum = 0;
        for (int c = 0; c <= ctx->maxn; ++c) {
            cum += st[8 + c];
            if (cum > idx) return c;
        }
        return ctx->maxn;
    };
    s.p50 = pct(.5);
    s.p90 = pct(.9);
    s.p99 = pct(.99);
    s.grid_cells = ctx->ncells;
    s.max_cell_occupancy = (int32_t)st[7];
    if (out) *out = s;
}

void nb_stats(lsmps_ctx* ctx, lsmps_neighbor_stats* out, const char* where) {
    int n = (int)ctx->n;
    int maxn = ctx->maxn;
    auto* st = ctx->nbr_stats.ensure<unsigned long long>(8 + maxn + 1);
    LSMPS_CUDA(cudaMemsetAsync(st, 0, (8 + maxn + 1) * sizeof(unsigned long long), ctx->stream));
    if (n > 0) {
        size_t shm = (maxn + 7) * sizeof(unsigned int);
        k_nbr_stats<<<std::min(148 * 4, (int)blocks_for(n, 256)), 256, shm, ctx->stream>>>(
            ctx->nbr_cnt.get<int>(), ctx->cls.get<uint8_t>(), n, maxn, ctx->have_classes ? 1 : 0, st);
        LSMPS_CHECK_LAUNCH();
    }
    std::vector<unsigned long long> h(8 + maxn + 1);
    read_back(ctx, {{st, h.data(), h.size() * sizeof(unsigned long long)}}, where);
    h[5] = ctx->truncated;
    h[7] = (unsigned long long)ctx->max_cell_occupancy;
    fill_stats(ctx, h, out);
}

static GridView grid_view(lsmps_ctx* ctx) {
    return {ctx->cell_start.get<int>(), ctx->gdim[0], ctx->gdim[1], ctx->gdim[2]};
}

// The two passes' non-empty segments, listed in ctx->seg_list
static SegGrid list_segments(lsmps_ctx* ctx) {
    cudaStream_t s = ctx->stream;
    const SegGrid sg{grid_view(ctx), make_int3(ctx->gmin[0], ctx->gmin[1], ctx->gmin[2]), ctx->re,
                     (ctx->gdim[0] + SEG - 1) / SEG};
    const long long nseg = (long long)sg.nsegx * ctx->gdim[1] * ctx->gdim[2];
    int* list = ctx->seg_list.ensure<int>(nseg + 1);
    int* count = ctx->scratch.get<int>() + 40;
    LSMPS_CUDA(cudaMemsetAsync(count, 0, sizeof(int), s));
    k_list_segments<<<(unsigned)((nseg + 255) / 256), 256, 0, s>>>(sg, nseg, list, count);
    LSMPS_CHECK_LAUNCH();
    read_back(ctx, {{count, &ctx->nsegs, sizeof(int)}}, nullptr);
    return sg;
}

// The single pass's items and relative positions
static void scan_prep(lsmps_ctx* ctx) {
    cudaStream_t s = ctx->stream;
    const size_t n = ctx->n;
    const size_t most = std::min((size_t)ctx->ncells, n) + n / 32 + 1;  // non-empty cells, and their further blocks
    int4* items = ctx->scan_items.ensure<int4>(most + 1);
    float4* rel = ctx->scan_rel.ensure<float4>(n);
    LSMPS_CUDA(cudaMemsetAsync(items, 0, sizeof(int4), s));
    k_scan_prep<<<blocks_for(n, 256), 256, 0, s>>>(
        grid_view(ctx), make_int3(ctx->gmin[0], ctx->gmin[1], ctx->gmin[2]), ctx->re, (int)n, ctx->scell.get<int>(),
        ctx->sx.get<double>(), ctx->sy.get<double>(), ctx->sz.get<double>(), items, rel);
    LSMPS_CHECK_LAUNCH();
}

static void launch_cell_scan(lsmps_ctx* ctx, int maxn, double l0, int classify, int* cnt, unsigned long long* trunc,
                             int* slots, uint8_t* cls, bool again = false) {
    const size_t n = ctx->n, most = std::min((size_t)ctx->ncells, n) + n / 32 + 1;
    const unsigned grid = (unsigned)std::min<size_t>((most + SCAN_WARPS - 1) / SCAN_WARPS, 148 * 4);
    if (again) LSMPS_CUDA(cudaMemsetAsync(&ctx->scan_items.get<int4>()->y, 0, sizeof(int), ctx->stream));
    // where re^2 itself leaves the FP64 range every candidate (d^2 <= 12 re^2) is decided exactly
    const bool in_range = ctx->re2 > 1e-290 && ctx->re2 < 1e290;
    const ScanBand lim = in_range ? ScanBand{1.f - 2e-5f, 1.f + 2e-5f, 2.1e-5f} : ScanBand{0.f, 100.f, INFINITY};
    k_cell_scan<<<grid, 32 * SCAN_WARPS, 0, ctx->stream>>>(
        grid_view(ctx), (int)n, ctx->scan_items.get<int4>(), ctx->scan_rel.get<float4>(), ctx->sx.get<double>(),
        ctx->sy.get<double>(), ctx->sz.get<double>(), ctx->stype.get<uint8_t>(), lim, ctx->re2, maxn, l0,
        classify, cnt, trunc, slots, cls);
    LSMPS_CHECK_LAUNCH();
}

void nb_build(lsmps_ctx* ctx, double re, int maxn, double l0, int flags, lsmps_neighbor_stats* out) {
    LSMPS_REQUIRE(re > 0 && std::isfinite(re), LSMPS_ERR_ARG, "re must be positive and finite");
    LSMPS_REQUIRE(maxn >= 0 && maxn <= 8192, LSMPS_ERR_ARG, "max_neighbors must be in [0, 8192]");
    LSMPS_REQUIRE(ctx->n < (size_t)INT_MAX, LSMPS_ERR_OVERFLOW, "particle count beyond int32");
    cudaStream_t s = ctx->stream;
    const size_t n = ctx->n;
    ctx->re = re;
    ctx->re2 = re * re;
    ctx->l0 = l0;
    ctx->maxn = maxn;
    ctx->have_neighbors = ctx->have_classes = false;
    ctx->have_wls = ctx->have_ppe = ctx->have_solution = false;
    ctx->have_candidates = false;  // the sorted numbering changes
    int* dflag = ctx->dflags.get<int>();

    // 1. cell coordinates + bounds
    int3* cell = ctx->cell_of.ensure<int3>(n);
    int* bounds = ctx->scratch.ensure<int>(64);
    int init[6] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN};
    LSMPS_CUDA(cudaMemcpyAsync(bounds, init, sizeof(init), cudaMemcpyHostToDevice, s));
    if (n) {
        k_cell_coords<<<std::min<unsigned>(blocks_for(n, 256), 148 * 8), 256, 0, s>>>(
            ctx->pos.get<double>(), n, re, cell, bounds, dflag);
        LSMPS_CHECK_LAUNCH();
    }
    int hb[6];
    read_back(ctx, {{bounds, hb, sizeof(hb)}}, "cell coordinates");
    if (n == 0) { hb[0] = hb[1] = hb[2] = 0; hb[3] = hb[4] = hb[5] = 0; }
    for (int a = 0; a < 3; ++a) {
        ctx->gmin[a] = hb[a];
        ctx->gdim[a] = hb[3 + a] - hb[a] + 1;
    }
    long long ncells = (long long)ctx->gdim[0] * ctx->gdim[1] * ctx->gdim[2];
    LSMPS_REQUIRE(ncells > 0 && ncells <= MAX_CELLS, LSMPS_ERR_GRID,
                  "dense cell grid of " + std::to_string(ncells) + " cells exceeds the limit of " +
                      std::to_string(MAX_CELLS));
    ctx->ncells = ncells;

    // 2. counting sort
    int* lin = ctx->slot.ensure<int>(2 * n + 1);  // lin[0..n) and slot[n..2n)
    int* slot = lin + n;
    int* count = ctx->cell_count.ensure<int>(ncells + 1);
    int* cstart = ctx->cell_start.ensure<int>(ncells + 1);
    int* perm = ctx->perm.ensure<int>(n);
    LSMPS_CUDA(cudaMemsetAsync(count, 0, (ncells + 1) * sizeof(int), s));
    int3 g0 = make_int3(ctx->gmin[0], ctx->gmin[1], ctx->gmin[2]);
    int3 gd = make_int3(ctx->gdim[0], ctx->gdim[1], ctx->gdim[2]);
    if (n) {
        k_cell_count<<<blocks_for(n, 256), 256, 0, s>>>(cell, n, g0, gd, lin, slot, count);
        LSMPS_CHECK_LAUNCH();
    }
    scan_exclusive<int>(count, cstart, ncells, s, ctx->scan_tmp, dflag);
    if (n) {
        k_scatter<<<blocks_for(n, 256), 256, 0, s>>>(lin, slot, n, cstart, perm);
        LSMPS_CHECK_LAUNCH();
    }
    int* big = ctx->scratch.get<int>() + 8;  // [8] big count, [9] max occupancy
    LSMPS_CUDA(cudaMemsetAsync(big, 0, 2 * sizeof(int), s));
    int* big_list = count;  // counts are no longer needed: reuse as the crowded-cell list
    k_sort_small_cells<<<(unsigned)((ncells + 255) / 256), 256, 0, s>>>(cstart, ncells, perm, big_list, big,
                                                                       big + 1);
    LSMPS_CHECK_LAUNCH();
    k_sort_big_cells<<<148, 1024, 0, s>>>(cstart, perm, big_list, big, dflag);
    LSMPS_CHECK_LAUNCH();

    double* sx = ctx->sx.ensure<double>(n);
    double* sy = ctx->sy.ensure<double>(n);
    double* sz = ctx->sz.ensure<double>(n);
    uint8_t* stype = ctx->stype.ensure<uint8_t>(n);
    int* scell = ctx->scell.ensure<int>(n);
    int* iperm = ctx->iperm.ensure<int>(n);
    if (n) {
        k_gather_sorted<<<blocks_for(n, 256), 256, 0, s>>>(perm, n, ctx->pos.get<double>(),
                                                           ctx->type_in.get<uint8_t>(), lin, sx, sy, sz,
                                                           stype, scell, iperm);
        LSMPS_CHECK_LAUNCH();
    }

    // 3. count pass, row pointers, fill pass (+ classification)
    int* cnt = ctx->nbr_cnt.ensure<int>(n + 1);
    int* row = ctx->nbr_row.ensure<int>(n + 1);
    unsigned long long* trunc_d = reinterpret_cast<unsigned long long*>(ctx->scratch.get<int>() + 16);
    LSMPS_CUDA(cudaMemsetAsync(trunc_d, 0, sizeof(unsigned long long), s));
    const int do_cls = (flags & LSMPS_NBR_CLASSIFY) ? 1 : 0;
    uint8_t* cls = ctx->cls.ensure<uint8_t>(n);
    // one pass into maxn slots per particle while they fit (the usual case: 0.5 GB at 1M
    // particles and maxn 128), else the count and fill passes
    const bool single = !(flags & LSMPS_NBR_TWO_PASS) && (double)n * (double)maxn * 4.0 <= SLOT_BUDGET_BYTES;
    ctx->nbr_single = single;
    int* slots = single ? ctx->nbr_slots.ensure<int>((size_t)n * maxn + 1) : nullptr;
    SegGrid sg{};
    if (n && single) {
        scan_prep(ctx);
        launch_cell_scan(ctx, maxn, l0, do_cls, cnt, trunc_d, slots, cls);
    } else if (n) {
        sg = list_segments(ctx);
        k_seg_pass<false><<<(unsigned)ctx->nsegs, SEG_THREADS, 0, s>>>(sg, ctx->seg_list.get<int>(), sx, sy, sz, scell,
                                                                       stype, ctx->re2, maxn, l0, 0, cnt, trunc_d,
                                                                       nullptr, nullptr, nullptr);
        LSMPS_CHECK_LAUNCH();
    }
    scan_exclusive<int>(cnt, row, (long long)n, s, ctx->scan_tmp, dflag);
    int hpairs = 0, hocc = 0;
    unsigned long long htr = 0;
    read_back(ctx, {{row + n, &hpairs, sizeof(int)}, {big + 1, &hocc, sizeof(int)}, {trunc_d, &htr, sizeof(htr)}},
              "neighbor count");
    ctx->pairs = (uint64_t)hpairs;
    ctx->truncated = htr;
    ctx->max_cell_occupancy = hocc;
    int* col = ctx->nbr_col.ensure<int>((size_t)hpairs + 1);
    if (n) {
        if (single)
            k_slots_compact<<<(unsigned)((8ull * n + 255) / 256), 256, 0, s>>>((int)n, maxn, slots, row, col);
        else
            k_seg_pass<true><<<(unsigned)ctx->nsegs, SEG_THREADS, 0, s>>>(sg, ctx->seg_list.get<int>(), sx, sy, sz,
                                                                          scell, stype, ctx->re2, maxn, l0, do_cls,
                                                                          nullptr, nullptr, row, col, cls);
        LSMPS_CHECK_LAUNCH();
    }
    ctx->have_neighbors = true;
    ctx->have_classes = do_cls != 0;
    // without statistics nothing is read back here (no device flag is set after the count's
    // read-back), so the host does not wait for the compaction
    if (out) nb_stats(ctx, out, "neighbor fill");
}

bool nb_filter_single(lsmps_ctx* ctx, int classify) {
    const size_t n = ctx->n;
    const int maxn = ctx->maxn;
    if ((double)n * (double)maxn * 4.0 > SLOT_BUDGET_BYTES) return false;
    cudaStream_t s = ctx->stream;
    int* dflag = ctx->dflags.get<int>();
    int* cnt = ctx->nbr_cnt.ensure<int>(n + 1);
    int* row = ctx->nbr_row.ensure<int>(n + 1);
    int* slots = ctx->nbr_slots.ensure<int>(n * maxn + 1);
    uint8_t* cls = ctx->cls.ensure<uint8_t>(n + 1);
    auto* trunc_d = reinterpret_cast<unsigned long long*>(ctx->scratch.get<int>() + 16);
    LSMPS_CUDA(cudaMemsetAsync(trunc_d, 0, sizeof(unsigned long long), s));
    if (n) {
        const unsigned grid = std::max(1u, std::min<unsigned>(blocks_for(n * 8, 256), 148 * 64));
        k_filter_slots<<<grid, 256, 0, s>>>((int)n, ctx->cand_row.get<int>(), ctx->cand_col.get<int>(),
                                            ctx->sx.get<double>(), ctx->sy.get<double>(), ctx->sz.get<double>(),
                                            ctx->stype.get<uint8_t>(), ctx->re2, (float)(1e-6 * ctx->re), maxn, ctx->l0,
                                            classify, slots, cnt, trunc_d, cls);
        LSMPS_CHECK_LAUNCH();
    }
    scan_exclusive<int>(cnt, row, (long long)n, s, ctx->scan_tmp, dflag);
    int hpairs = 0;
    unsigned long long htr = 0;
    read_back(ctx, {{row + n, &hpairs, sizeof(int)}, {trunc_d, &htr, sizeof(htr)}}, "neighbor filter");
    ctx->pairs = (uint64_t)hpairs;
    ctx->truncated = htr;
    int* col = ctx->nbr_col.ensure<int>((size_t)hpairs + 1);
    if (n) {
        k_slots_compact<<<(unsigned)((8ull * n + 255) / 256), 256, 0, s>>>((int)n, maxn, slots, row, col);
        LSMPS_CHECK_LAUNCH();
    }
    return true;
}

void nb_kernel_bench(lsmps_ctx* ctx, int kernel, int reps, double* ms, double* bytes) {
    LSMPS_REQUIRE(ctx->have_neighbors, LSMPS_ERR_STATE, "kernel bench needs neighbor lists");
    cudaStream_t s = ctx->stream;
    int n = (int)ctx->n;
    auto* trunc_d = reinterpret_cast<unsigned long long*>(ctx->scratch.get<int>() + 16);
    if (n == 0) { *ms = 0; *bytes = 0; return; }
    SegGrid sg{};
    if (kernel == LSMPS_KB_NBR_SCAN) scan_prep(ctx);
    else if (kernel != LSMPS_KB_NBR_COMPACT) sg = list_segments(ctx);
    const int* seg_list = ctx->seg_list.get<int>();
    const unsigned seg_grid = (unsigned)ctx->nsegs;
    int* slots = nullptr;
    if (kernel == LSMPS_KB_NBR_SCAN || kernel == LSMPS_KB_NBR_COMPACT) {
        LSMPS_REQUIRE((double)n * (double)ctx->maxn * 4.0 <= SLOT_BUDGET_BYTES, LSMPS_ERR_STATE,
                      "single-pass neighbor bench: slot rows exceed the budget");
        LSMPS_REQUIRE(kernel == LSMPS_KB_NBR_SCAN || ctx->nbr_single, LSMPS_ERR_STATE,
                      "compaction bench needs a single-pass build");
        slots = ctx->nbr_slots.ensure<int>((size_t)n * ctx->maxn + 1);
    }
    auto launch = [&] {
        if (kernel == LSMPS_KB_NBR_SCAN)
            launch_cell_scan(ctx, ctx->maxn, ctx->l0, ctx->have_classes ? 1 : 0, ctx->nbr_cnt.get<int>(), trunc_d, slots,
                             ctx->cls.get<uint8_t>(), true);
        else if (kernel == LSMPS_KB_NBR_COMPACT)
            k_slots_compact<<<(unsigned)((8ull * n + 255) / 256), 256, 0, s>>>(n, ctx->maxn, slots,
                                                                               ctx->nbr_row.get<int>(),
                                                                               ctx->nbr_col.get<int>());
        else if (kernel == LSMPS_KB_NBR_COUNT)
            k_seg_pass<false><<<seg_grid, SEG_THREADS, 0, s>>>(
                sg, seg_list, ctx->sx.get<double>(), ctx->sy.get<double>(), ctx->sz.get<double>(), ctx->scell.get<int>(),
                ctx->stype.get<uint8_t>(), ctx->re2, ctx->maxn, ctx->l0, 0, ctx->nbr_cnt.get<int>(), trunc_d, nullptr,
                nullptr, nullptr);
        else
            k_seg_pass<true><<<seg_grid, SEG_THREADS, 0, s>>>(
                sg, seg_list, ctx->sx.get<double>(), ctx->sy.get<double>(), ctx->sz.get<double>(), ctx->scell.get<int>(),
                ctx->stype.get<uint8_t>(), ctx->re2, ctx->maxn, ctx->l0, ctx->have_classes ? 1 : 0, nullptr, nullptr,
                ctx->nbr_row.get<int>(), ctx->nbr_col.get<int>(), ctx->cls.get<uint8_t>());
        LSMPS_CHECK_LAUNCH();
    };
    launch();  // warm
    ev_record(ctx, 14);
    for (int r = 0; r < reps; ++r) launch();
    ev_record(ctx, 15);
    *ms = ev_elapsed(ctx, 14, 15) / reps;
    // algorithmic bytes: positions (24 B) and cell (4 B) of every particle once, cell starts;
    // the count pass writes 4 B per particle, the fill pass reads types and row pointers and
    // writes the columns and classes
    double N = (double)n, P = (double)ctx->pairs, cells = (double)ctx->ncells;
    if (kernel == LSMPS_KB_NBR_SCAN)  // + scell, types, counts, kept slots, classes
        *bytes = 24.0 * N + 4.0 * N + 1.0 * N + 4.0 * N + 4.0 * P + 1.0 * N + 4.0 * cells;
    else if (kernel == LSMPS_KB_NBR_COMPACT)  // row pointers, the kept slots read and the CSR written
        *bytes = 4.0 * (N + 1) + 8.0 * P;
    else
        *bytes = kernel == LSMPS_KB_NBR_COUNT ? 32.0 * N + 4.0 * cells : 34.0 * N + 4.0 * P + 4.0 * cells;
}

void nb_classify(lsmps_ctx* ctx, double l0, lsmps_neighbor_stats* out) {
    LSMPS_REQUIRE(ctx->have_neighbors, LSMPS_ERR_STATE, "classify needs lsmps_build_neighbors first");
    int n = (int)ctx->n;
    ctx->l0 = l0;
    uint8_t* cls = ctx->cls.ensure<uint8_t>(ctx->n);
    if (n) {
        k_classify<<<(unsigned)((n + NB_WARPS - 1) / NB_WARPS), NB_WARPS * 32, 0, ctx->stream>>>(
            ctx->sx.get<double>(), ctx->sy.get<double>(), ctx->sz.get<double>(), ctx->stype.get<uint8_t>(), n,
            l0, ctx->nbr_row.get<int>(), ctx->nbr_col.get<int>(), cls);
        LSMPS_CHECK_LAUNCH();
    }
    ctx->have_classes = true;
    ctx->have_wls = ctx->have_ppe = ctx->have_solution = false;
    nb_stats(ctx, out);
}

void nb_download(lsmps_ctx* ctx, int32_t* row_ptr, int32_t* col, size_t col_cap) {
    LSMPS_REQUIRE(ctx->have_neighbors, LSMPS_ERR_STATE, "no neighbor lists built");
    cudaStream_t s = ctx->stream;
    size_t n = ctx->n;
    int* ocnt = ctx->vtmp.ensure<int>(2 * n + 2);
    int* orow = ocnt + n + 1;
    if (n) {
        k_orig_counts<<<blocks_for(n, 256), 256, 0, s>>>(ctx->iperm.get<int>(), ctx->nbr_row.get<int>(), n, ocnt);
        LSMPS_CHECK_LAUNCH();
    }
    scan_exclusive<int>(ocnt, orow, (long long)n, s, ctx->scan_tmp, ctx->dflags.get<int>());
    if (row_ptr) LSMPS_CUDA(cudaMemcpyAsync(row_ptr, orow, (n + 1) * sizeof(int), cudaMemcpyDeviceToHost, s));
    if (col) {
        LSMPS_REQUIRE(col_cap >= ctx->pairs, LSMPS_ERR_ARG, "col buffer smaller than the pair count");
        int* ocol = ctx->vs.ensure<int>(ctx->pairs + 1);
        if (n) {
            k_orig_fill<<<(unsigned)((n + NB_WARPS - 1) / NB_WARPS), NB_WARPS * 32, 0, s>>>(
                ctx->iperm.get<int>(), ctx->perm.get<int>(), ctx->nbr_row.get<int>(), ctx->nbr_col.get<int>(),
                (int)n, orow, ocol);
            LSMPS_CHECK_LAUNCH();
        }
        LSMPS_CUDA(cudaMemcpyAsync(col, ocol, ctx->pairs * sizeof(int), cudaMemcpyDeviceToHost, s));
    }
    LSMPS_CUDA(cudaStreamSynchronize(s));
}

void nb_download_types(lsmps_ctx* ctx, uint8_t* type, size_t n) {
    LSMPS_REQUIRE(ctx->have_classes, LSMPS_ERR_STATE, "no classification computed");
    LSMPS_REQUIRE(n == ctx->n, LSMPS_ERR_ARG, "type buffer size differs from the particle count");
    uint8_t* tmp = ctx->vtmp.ensure<uint8_t>(n + 1);
    if (n) {
        k_orig_types<<<blocks_for(n, 256), 256, 0, ctx->stream>>>(ctx->iperm.get<int>(), ctx->cls.get<uint8_t>(),
                                                                  n, tmp);
        LSMPS_CHECK_LAUNCH();
        LSMPS_CUDA(cudaMemcpyAsync(type, tmp, n, cudaMemcpyDeviceToHost, ctx->stream));
    }
    LSMPS_CUDA(cudaStreamSynchronize(ctx->stream));
}

}  // namespace lsmps_gpu
