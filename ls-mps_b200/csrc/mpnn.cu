// Learned preconditioner: a message-passing network over the PPE graph, trained and
// evaluated on the GPU with BF16 weights / activations and FP32 accumulation on the
// tensor cores (mma.sync m16n8k16 BF16; the 64x128 layer transform of a 16-node tile is
// 64 MMAs, so the layer is bound by the neighbor gathers of the aggregation, not the MMA).
//
// Network (parameter order of lsmps_gpu.h): x_i = [r_i sqrt(U), a_ii / mean(a) - 1,
// NearWall, row length / 32 - 1]; h0 = ReLU(W_enc x + b_enc); for l = 0..2:
// m_i = sum_j w_ij h_j with w_ij = -a_ij / a_ii, h <- h + ReLU(W_l [h | m] + b_l);
// y_i = (w_dec . h3_i + b_dec) / sqrt(U). Loss |y - t|^2 / |t|^2 with t = D x / |b| for the
// input r = b / |b| (the Jacobi-scaled solution of the unit right-hand side).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <random>
#include <vector>

#include "ops.cuh"
#include "scan.cuh"

namespace lsmps_gpu {

namespace {
constexpr int H = 64, KIN = 128, NF = 4, NL = 3;
constexpr int LDA = KIN + 8;  // padded shared-memory row of a [h | m] tile (bf16): conflict-free ldmatrix
constexpr int LDG = H + 8;    // padded row of a 64-wide tile
constexpr size_t OFF_WE = 0, OFF_BE = 256, OFF_L0 = 320, LSTRIDE = 8192 + 64;
constexpr size_t OFF_WD = OFF_L0 + NL * LSTRIDE, OFF_BD = OFF_WD + 64, NPARAM = OFF_BD + 1;
constexpr int WG_BLOCKS = 296;  // weight-gradient partial blocks (2 per SM)
using bf16 = __nv_bfloat16;
}  // namespace

struct MpnnGraph {
    long long U = 0, nnz = 0;
    DevBuf row, col, ew, feat, dg;  // row/col copies (training store) or unused (inference view); dg: a_ii
    const int* prow = nullptr;
    const int* pcol = nullptr;
};

struct MpnnSample {
    int graph;
    DevBuf r, t;  // float U: input b / |b|, target D x / |b|
    double tnorm2;
};

struct MpnnState {
    std::vector<float> w;  // FP32 master weights (host copy)
    DevBuf dw, wbf, am, av, grad, gpart, red;
    int adam_t = 0;
    std::vector<std::unique_ptr<MpnnGraph>> graphs;
    std::vector<std::unique_ptr<MpnnSample>> samples;
    long long graph_gen = -1;  // assembly generation of graphs.back()
    MpnnGraph infer;           // graph of the current system (inference)
    long long infer_gen = -1;
    long long cap = 0;         // workspace capacity (nodes)
    int loss_kind = 0;         // 0 error, 1 residual, 2 both
    DevBuf h[NL + 1], a[NL], z[NL + 1], y, gy, ay, q, gh[2], gam, gz;
};

namespace {

// ---- tensor-core helpers (inline PTX) ------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void ldsm_x4(unsigned addr, unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(unsigned addr, unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x2(unsigned addr, unsigned& r0, unsigned& r1) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x2_t(unsigned addr, unsigned& r0, unsigned& r1) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(addr));
}
// D = A (16x16 bf16, row) * B (16x8 bf16, col) + D, FP32 accumulate
__device__ __forceinline__ void mma16816(float* d, unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                         unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A-operand address of a 16x16 tile at (row 0, col k0) of a row-major bf16 tile with row
// stride ld (lanes 0-15: rows 0-15 at k0; lanes 16-31: rows 0-15 at k0 + 8)
__device__ __forceinline__ unsigned a_addr(const bf16* tile, int ld, int k0, int lane) {
    return smem_u32(tile + (lane & 15) * ld + k0 + ((lane >> 4) << 3));
}

// ---- graph construction from the assembled PPE ---------------------------------------
// Four rows per warp step (grid-stride), eight lanes over each row's entries, so a warp has
// four rows' loads in flight
__global__ void k_graph_ew(long long U, const int* __restrict__ row, const double* __restrict__ val,
                           const double* __restrict__ dinv, float* __restrict__ ew) {
    const int lane = threadIdx.x & 31, g = lane >> 3, sub = lane & 7;
    const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long u0 = ((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5) * 4; u0 < U; u0 += 4 * nw) {
        const long long u = u0 + g;
        if (u >= U) continue;
        const int e0 = row[u], e1 = row[u + 1];
        const double di = dinv[u];
#pragma unroll 4
        for (int e = e0 + sub; e < e1; e += 8) ew[e] = e < e1 - 1 ? (float)(-val[e] * di) : 0.f;  // diagonal last
    }
}

constexpr int MEAN_BLOCKS = 592;

// mean of a_uu = 1 / dinv_u (1 where dinv is 0): per-block sums, then one block adds them
// in block order (deterministic)
__global__ void k_diag_partials(long long U, const double* __restrict__ dinv, double* part) {
    __shared__ double ws[8];
    double acc = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < U; i += (long long)gridDim.x * blockDim.x)
        acc += dinv[i] != 0 ? 1.0 / dinv[i] : 1.0;
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += ws[k];
        part[blockIdx.x] = t;
    }
}

__global__ void k_mean_finish(long long U, const double* __restrict__ part, int nparts, double* out) {
    __shared__ double ws[8];
    double acc = 0;
    for (int k = threadIdx.x; k < nparts; k += blockDim.x) acc += part[k];
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += ws[k];
        *out = U ? t / (double)U : 1.0;
    }
}

// feat[u] = [a_uu / mean - 1, NearWall, (row length - 1) / 32 - 1]
__global__ void k_graph_feat(long long U, const int* __restrict__ row, const double* __restrict__ dinv,
                             const uint8_t* __restrict__ cls, const int* __restrict__ sorted_of_u,
                             const double* mean, float* __restrict__ feat, float* __restrict__ dg) {
    long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (u >= U) return;
    const double d = dinv[u] != 0 ? 1.0 / dinv[u] : 1.0;
    dg[u] = (float)d;
    feat[3 * u + 0] = (float)(d / *mean - 1.0);
    feat[3 * u + 1] = cls[sorted_of_u[u]] == LSMPS_NEAR_WALL ? 1.f : 0.f;
    feat[3 * u + 2] = (float)(row[u + 1] - row[u] - 1) / 32.f - 1.f;
}

// ---- forward ---------------------------------------------------------------------------
struct GView {
    long long U;
    const int* row;
    const int* col;
    const float* ew;
    const float* feat;
    const float* dg;  // a_ii
    float sqrt_u;
};

__device__ __forceinline__ void features(const GView& G, const float* __restrict__ r, long long i, float x[NF]) {
    x[0] = r[i] * G.sqrt_u;
    x[1] = G.feat[3 * i];
    x[2] = G.feat[3 * i + 1];
    x[3] = G.feat[3 * i + 2];
}

// h0 = ReLU(W_enc x + b_enc) (CUDA cores: K = 4). Four nodes per warp step, eight lanes per
// node and eight features per lane (whose weights stay in registers), so each node's
// 128-byte row is one coalesced store; four steps' inputs are loaded before their sums.
__global__ void __launch_bounds__(256) k_enc(GView G, const float* __restrict__ r, const float* __restrict__ w,
                                             bf16* __restrict__ h0, float* __restrict__ z0) {
    const int lane = threadIdx.x & 31, g = lane >> 3, c8 = (lane & 7) * 8;
    float we[8][NF], be[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        be[q] = w[OFF_BE + c8 + q];
#pragma unroll
        for (int f = 0; f < NF; ++f) we[q][f] = w[OFF_WE + (c8 + q) * NF + f];
    }
    const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
    constexpr int STEPS = 4;
    for (long long i0 = ((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5) * 4; i0 < G.U;
         i0 += 4 * STEPS * nw) {
        float x[STEPS][NF];
#pragma unroll
        for (int k = 0; k < STEPS; ++k) {
            const long long i = i0 + 4 * k * nw + g;
            if (i < G.U) features(G, r, i, x[k]);
        }
#pragma unroll
        for (int k = 0; k < STEPS; ++k) {
            const long long i = i0 + 4 * k * nw + g;
            if (i >= G.U) continue;
            __align__(16) bf16 hv[8];
            __align__(16) float zv[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                float zz = be[q];
#pragma unroll
                for (int f = 0; f < NF; ++f) zz += we[q][f] * x[k][f];
                zv[q] = zz;
                hv[q] = __float2bfloat16(fmaxf(zz, 0.f));
            }
            if (z0) {
                *reinterpret_cast<float4*>(z0 + i * H + c8) = *reinterpret_cast<const float4*>(zv);
                *reinterpret_cast<float4*>(z0 + i * H + c8 + 4) = *reinterpret_cast<const float4*>(zv + 4);
            }
            *reinterpret_cast<uint4*>(h0 + i * H + c8) = *reinterpret_cast<const uint4*>(hv);
        }
    }
}

// One message-passing layer, one warp per 16-node tile:
//   1. aggregation m_i = sum_j w_ij h_j (8 lanes per neighbor row, 8 features per lane; FP32),
//      staged with h_i as the bf16 A tile [h | m] (16 x 128) in shared memory;
//   2. z = [h | m] W^T on the tensor cores (8 k-steps x 8 n-tiles of m16n8k16);
//   3. h_out = h + ReLU(z + b) (bf16), with [h | m] and z kept for the backward pass.
// Launch shape (the autotuner's choice; every shape gives the same bits, since each node's
// sums run in the same order and an MMA row depends only on its own A row):
//   NB     4 NB neighbor-row gathers in flight per warp, 16 bytes per lane;
//   WARPS  warps per block (dynamic shared memory: W, the bias and one A tile per warp);
//   LOCAL  false: warp w of block b takes the 16 consecutive nodes of tile 4 b + w (grid-
//          stride); true: the block takes WARPS * 16 consecutive nodes and warp w the nodes
//          w, w + WARPS, ..., so the block's warps gather the neighbors of a few consecutive
//          nodes at a time and those rows (shared by ~3 nodes each in the cell-sorted order)
//          are re-read from L1 instead of L2.
// At most 72 registers (80 uncapped): the tuned shapes hold 24 warps per SM, which then leave
// 10,240 registers free, so the multigrid set-up's kernels on the LEARNED solve's side stream
// (blocks of at most 256 threads at 40 registers) run on the SMs beside the layer instead of
// waiting for it (step 14.01 against 14.12-14.23 ms at 1M particles; the layer's own time is
// unchanged, 503-511 us).
template <int NB, int WARPS, bool LOCAL>
__global__ void __maxnreg__(72)
    k_layer_fwd(GView G, const bf16* __restrict__ h_in, bf16* __restrict__ h_out, const bf16* __restrict__ Wl,
                const float* __restrict__ bl, bf16* __restrict__ a_save, float* __restrict__ z_save) {
    extern __shared__ __align__(16) unsigned char layer_smem[];
    bf16* Ws = reinterpret_cast<bf16*>(layer_smem);          // H x LDA
    bf16* As = Ws + H * LDA;                                 // WARPS tiles of 16 x LDA
    float* bs = reinterpret_cast<float*>(As + WARPS * 16 * LDA);  // H
    for (int k = threadIdx.x; k < H * KIN / 8; k += blockDim.x) {
        const int n = k / (KIN / 8), c = (k % (KIN / 8)) * 8;
        *reinterpret_cast<uint4*>(Ws + n * LDA + c) = *reinterpret_cast<const uint4*>(Wl + n * KIN + c);
    }
    if (threadIdx.x < H) bs[threadIdx.x] = bl[threadIdx.x];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    bf16* A = As + warp * 16 * LDA;
    constexpr long long SPAN = LOCAL ? WARPS * 16 : 16;  // nodes per job
    const long long njobs = (G.U + SPAN - 1) / SPAN;
    const long long j0 = LOCAL ? (long long)blockIdx.x : blockIdx.x * (long long)WARPS + warp;
    const long long js = LOCAL ? (long long)gridDim.x : (long long)gridDim.x * WARPS;
    // node of row t of this warp's tile in job `job`
    auto node = [&](long long job, int t) -> long long {
        return LOCAL ? job * SPAN + warp + (long long)WARPS * t : job * SPAN + t;
    };
    for (long long job = j0; job < njobs; job += js) {
        // first and one-past-last entry of node t's row in lane t (rows have U + 1 pointers)
        int rs = 0, re = 0;
        if (lane < 16) {
            const long long i = node(job, lane);
            if (i < G.U) {
                rs = G.row[i];
                re = G.row[i + 1];
            }
        }
        // (col, weight) of up to 32 edges of node t, one per lane; the diagonal (the row's last
        // entry) has no edge
        auto fetch = [&](int t, int& cj, float& wj, int& ne, int& e0) {
            e0 = __shfl_sync(0xffffffffu, rs, t);
            ne = max(__shfl_sync(0xffffffffu, re, t) - 1 - e0, 0);
            cj = 0;
            wj = 0.f;
            if (lane < min(ne, 32)) {
                cj = G.col[e0 + lane];
                wj = G.ew[e0 + lane];
            }
        };
        const int quad = lane >> 3, sub = lane & 7;  // 8 lanes per neighbor row, 8 features (16 B) per lane
        int cj, ne, e0;
        float wj;
        fetch(0, cj, wj, ne, e0);
        for (int t = 0; t < 16; ++t) {
            const long long i = node(job, t);
            int cjn = 0, nen = 0, e0n = 0;
            float wjn = 0.f;
            if (t < 15) fetch(t + 1, cjn, wjn, nen, e0n);  // in flight during node t's gathers
            __nv_bfloat162 own = __floats2bfloat162_rn(0.f, 0.f);
            if (i < G.U) own = *reinterpret_cast<const __nv_bfloat162*>(h_in + i * H + 2 * lane);
            float2 m2[4] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};  // features (2c, 2c + 1)
            for (int eb = 0; eb < ne; eb += 32) {
                if (eb) {  // rows of more than 32 edges
                    cj = 0;
                    wj = 0.f;
                    if (lane < min(ne - eb, 32)) {
                        cj = G.col[e0 + eb + lane];
                        wj = G.ew[e0 + eb + lane];
                    }
                }
                const int nb = min(32, ne - eb);
                // each lane sums the edges quad, quad + 4, ... of the chunk in ascending order
                // (the same order for every NB); 4 NB rows in flight per warp
                for (int k = 0; k < nb; k += 4 * NB) {
                    uint4 a[NB];
                    float w[NB];
#pragma unroll
                    for (int q = 0; q < NB; ++q) {
                        const int edge = k + 4 * q + quad;
                        const int src = min(edge, nb - 1);
                        const int j = __shfl_sync(0xffffffffu, cj, src);
                        const float wq = __shfl_sync(0xffffffffu, wj, src);
                        w[q] = edge < nb ? wq : 0.f;
                        a[q] = *reinterpret_cast<const uint4*>(h_in + (long long)j * H + 8 * sub);
                    }
#pragma unroll
                    for (int q = 0; q < NB; ++q) {
                        // a bf16 is the upper half of the float it rounds: the low element of a
                        // pair is u << 16, the high one u with its low half cleared (exact)
                        const unsigned u[4] = {a[q].x, a[q].y, a[q].z, a[q].w};
                        const float2 ww = make_float2(w[q], w[q]);
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const float2 f = make_float2(__uint_as_float(u[c] << 16), __uint_as_float(u[c] & 0xffff0000u));
                            m2[c] = __ffma2_rn(ww, f, m2[c]);  // two FP32 FMAs in one instruction
                        }
                    }
                }
            }
            float m[8];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                m[2 * c] = m2[c].x;
                m[2 * c + 1] = m2[c].y;
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) {  // the four edge classes: (0 + 1) + (2 + 3)
                m[c] += __shfl_xor_sync(0xffffffffu, m[c], 8);
                m[c] += __shfl_xor_sync(0xffffffffu, m[c], 16);
            }
            *reinterpret_cast<__nv_bfloat162*>(A + t * LDA + 2 * lane) = own;
            if (quad == 0) {
                uint4 pk;
                unsigned* pw = reinterpret_cast<unsigned*>(&pk);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    __nv_bfloat162 b2 = __floats2bfloat162_rn(m[2 * c], m[2 * c + 1]);
                    pw[c] = *reinterpret_cast<unsigned*>(&b2);
                }
                *reinterpret_cast<uint4*>(A + t * LDA + H + 8 * sub) = pk;
            }
            cj = cjn;
            wj = wjn;
            ne = nen;
            e0 = e0n;
        }
        __syncwarp();
        float acc[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < KIN / 16; ++ks) {
            unsigned a0, a1, a2, a3;
            ldsm_x4(a_addr(A, LDA, ks * 16, lane), a0, a1, a2, a3);
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                unsigned b0, b1;
                // B (k x n) = W^T: rows n of Ws hold k contiguously -> non-transposed ldmatrix
                ldsm_x2(smem_u32(Ws + (nt * 8 + (lane & 7)) * LDA + ks * 16 + ((lane >> 3) & 1) * 8), b0, b1);
                mma16816(acc[nt], a0, a1, a2, a3, b0, b1);
            }
        }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = g + 8 * half;
                const long long i = node(job, t);
                if (i >= G.U) continue;
                const int c = nt * 8 + 2 * tq;
                const float z0 = acc[nt][2 * half] + bs[c], z1 = acc[nt][2 * half + 1] + bs[c + 1];
                const float2 hold = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(A + t * LDA + c));
                *reinterpret_cast<__nv_bfloat162*>(h_out + i * H + c) =
                    __floats2bfloat162_rn(hold.x + fmaxf(z0, 0.f), hold.y + fmaxf(z1, 0.f));
                if (z_save) *reinterpret_cast<float2*>(z_save + i * H + c) = make_float2(z0, z1);
            }
        }
        if (a_save) {
            for (int t = 0; t < 16; ++t) {
                const long long i = node(job, t);
                if (i < G.U)
                    *reinterpret_cast<uint2*>(a_save + i * KIN + 4 * lane) =
                        *reinterpret_cast<const uint2*>(A + t * LDA + 4 * lane);
            }
        }
        __syncwarp();
    }
}

// y_i = (w_dec . h3_i + b_dec) / sqrt(U)
__global__ void k_dec(GView G, const bf16* __restrict__ h3, const float* __restrict__ w, float* __restrict__ y) {
    __shared__ float sw[H + 1];
    if (threadIdx.x <= H) sw[threadIdx.x] = w[OFF_WD + threadIdx.x];
    __syncthreads();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < G.U; i += (long long)gridDim.x * blockDim.x) {
        float o = sw[H];
        for (int c8 = 0; c8 < H; c8 += 8) {
            uint4 q = *reinterpret_cast<const uint4*>(h3 + i * H + c8);
            const bf16* hv = reinterpret_cast<const bf16*>(&q);
#pragma unroll
            for (int k = 0; k < 8; ++k) o += sw[c8 + k] * __bfloat162float(hv[k]);
        }
        y[i] = o / G.sqrt_u;
    }
}

// ---- loss and backward -------------------------------------------------------------------
// Sums of squares over the nodes: LOSS_BLOCKS partials, then one warp adds them in block order
// (one block over all nodes took 23 us at 119k unknowns; 3.0 + 2.6 us)
constexpr int LOSS_BLOCKS = 148 * 2;
__device__ __forceinline__ void square_sum_partial(double acc, double* part) {
    __shared__ double ws[8];
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0;
        for (int k = 0; k < 8; ++k) s += ws[k];
        part[blockIdx.x] = s;
    }
}
// |y - t|^2 (t null: |y|^2)
__global__ void __launch_bounds__(256) k_loss(long long U, const float* __restrict__ y, const float* __restrict__ t,
                                              double* part) {
    double acc = 0;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < U; i += gridDim.x * 256LL) {
        const double d = (double)y[i] - (t ? (double)t[i] : 0.0);
        acc += d * d;
    }
    square_sum_partial(acc, part);
}
__global__ void k_sum_partials(const double* __restrict__ part, int n, double* out) {
    double acc = 0;
    for (int k = threadIdx.x; k < n; k += 32) acc += part[k];
    acc = warp_sum(acc);
    if (threadIdx.x == 0) *out = acc;
}

// (A D^-1 y)_i = y_i - a_ii sum_j w_ij y_j / a_jj, eight lanes per row
__global__ void __launch_bounds__(256) k_apply_scaled(GView G, const float* __restrict__ y, float* __restrict__ ay) {
    const long long i = (blockIdx.x * 256LL + threadIdx.x) >> 3;
    const int sub = threadIdx.x & 7;
    float s = 0.f;
    if (i < G.U)
        for (int e = G.row[i] + sub, e1 = G.row[i + 1] - 1; e < e1; e += 8) s += G.ew[e] * y[G.col[e]] / G.dg[G.col[e]];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (i < G.U && sub == 0) ay[i] = y[i] - G.dg[i] * s;
}

// dL/dy of the selected loss kind. Error: 2 (y - t) / |t|^2. Residual (|r| = 1):
// g = -2 (r - A D^-1 y); dL/dy_k = g_k - (1 / a_kk) sum_i a_ii w_ik g_i (q holds the sum,
// accumulated by k_scatter_res beforehand). Both: the sum.
__global__ void k_dldy(long long U, const float* __restrict__ y, const float* __restrict__ t, const float* __restrict__ r,
                       const float* __restrict__ ay, const float* __restrict__ q, const float* __restrict__ dg,
                       float err_scale, int kind, float* __restrict__ gy) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= U) return;
    float g = 0.f;
    if (kind != 1) g += err_scale * (y[i] - t[i]);
    if (kind != 0) g += -2.f * (r[i] - ay[i]) - q[i] / dg[i];
    gy[i] = g;
}

// q_k += a_ii w_ik g_i with g = -2 (r - A D^-1 y) (transposed product, eight lanes per row)
__global__ void __launch_bounds__(256) k_scatter_res(GView G, const float* __restrict__ r, const float* __restrict__ ay,
                                                     float* __restrict__ q) {
    const long long i = (blockIdx.x * 256LL + threadIdx.x) >> 3;
    if (i >= G.U) return;
    const float gi = -2.f * (r[i] - ay[i]) * G.dg[i];
    for (int e = G.row[i] + (threadIdx.x & 7), e1 = G.row[i + 1] - 1; e < e1; e += 8)
        atomicAdd(&q[G.col[e]], G.ew[e] * gi);
}

// Sum over the block's eight warps of each warp's n values (v: the warp's slot of n floats in
// shared memory, filled by its lanes) into out, in warp order.
template <int N>
__device__ __forceinline__ void add_warps(const float (*v)[N], int n, float* __restrict__ out) {
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += v[w][k];
        out[k] = s;
    }
}

// go_i = dL/dy_i / sqrt(U); gh3 = go w_dec; block partials of dw_dec (64) and db_dec (1). One
// warp per node, two features per lane summed in registers over the warp's nodes (bound by
// its 388 bytes per node; shared-memory atomics per node and feature took 317 us at 119k nodes,
// now 20 us).
__global__ void __launch_bounds__(256) k_dec_bwd(GView G, const float* __restrict__ gy, const bf16* __restrict__ h3,
                                                 const float* __restrict__ w, float* __restrict__ gh3,
                                                 float* __restrict__ part) {
    __shared__ float sg[8][H + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float w0 = w[OFF_WD + 2 * lane], w1 = w[OFF_WD + 2 * lane + 1];
    float a0 = 0.f, a1 = 0.f, ago = 0.f;
    const long long nw = gridDim.x * 8LL;
#pragma unroll 4
    for (long long i = blockIdx.x * 8LL + warp; i < G.U; i += nw) {
        const float go = gy[i] / G.sqrt_u;
        const float2 h = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(h3 + i * H + 2 * lane));
        *reinterpret_cast<float2*>(gh3 + i * H + 2 * lane) = make_float2(go * w0, go * w1);
        a0 += go * h.x;
        a1 += go * h.y;
        ago += go;
    }
    sg[warp][2 * lane] = a0;
    sg[warp][2 * lane + 1] = a1;
    if (lane == 0) sg[warp][H] = ago;
    add_warps<H + 1>(sg, H + 1, part + blockIdx.x * (H + 1));
}

// Layer backward, part a (one warp per 16-node tile):
//   gz = gh_next * (z > 0) (bf16, kept for the weight gradient), gA = gz W on the tensor
//   cores (16 x 128: 16 n-tiles x 4 k-steps), gh_cur = gh_next + gA[:, :64], gam = gA[:, 64:];
//   block partials of db.
__global__ void __launch_bounds__(128) k_layer_bwd_a(GView G, const float* __restrict__ gh_next,
                                                     const float* __restrict__ z, const bf16* __restrict__ Wl,
                                                     bf16* __restrict__ gz_out, float* __restrict__ gh_cur,
                                                     float* __restrict__ gam, float* __restrict__ bpart) {
    __shared__ __align__(16) bf16 Ws[H * LDA];
    __shared__ __align__(16) bf16 Gs[4][16 * LDG];
    __shared__ float sb[H];
    for (int k = threadIdx.x; k < H * KIN / 8; k += blockDim.x) {
        const int n = k / (KIN / 8), c = (k % (KIN / 8)) * 8;
        *reinterpret_cast<uint4*>(Ws + n * LDA + c) = *reinterpret_cast<const uint4*>(Wl + n * KIN + c);
    }
    if (threadIdx.x < H) sb[threadIdx.x] = 0.f;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    bf16* Gt = Gs[warp];
    float db0 = 0.f, db1 = 0.f;
    const long long ntiles = (G.U + 15) / 16;
    for (long long tile = blockIdx.x * 4LL + warp; tile < ntiles; tile += gridDim.x * 4LL) {
        const long long base = tile * 16;
        for (int t = 0; t < 16; ++t) {
            const long long i = base + t;
            float g0 = 0.f, g1 = 0.f;
            if (i < G.U) {
                const float2 gh = *reinterpret_cast<const float2*>(gh_next + i * H + 2 * lane);
                const float2 zz = *reinterpret_cast<const float2*>(z + i * H + 2 * lane);
                g0 = zz.x > 0.f ? gh.x : 0.f;
                g1 = zz.y > 0.f ? gh.y : 0.f;
            }
            const __nv_bfloat162 gb = __floats2bfloat162_rn(g0, g1);
            *reinterpret_cast<__nv_bfloat162*>(Gt + t * LDG + 2 * lane) = gb;
            if (i < G.U) *reinterpret_cast<__nv_bfloat162*>(gz_out + i * H + 2 * lane) = gb;
            db0 += g0;
            db1 += g1;
        }
        __syncwarp();
        float acc[16][4];
#pragma unroll
        for (int nt = 0; nt < 16; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < H / 16; ++ks) {
            unsigned a0, a1, a2, a3;
            ldsm_x4(a_addr(Gt, LDG, ks * 16, lane), a0, a1, a2, a3);
#pragma unroll
            for (int nt = 0; nt < 16; ++nt) {
                unsigned b0, b1;
                // B (k = out, n = in) = W (row-major [out][in]): transposed ldmatrix
                ldsm_x2_t(smem_u32(Ws + (ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LDA + nt * 8), b0, b1);
                mma16816(acc[nt], a0, a1, a2, a3, b0, b1);
            }
        }
#pragma unroll
        for (int nt = 0; nt < 16; ++nt) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const long long i = base + g + 8 * half;
                if (i >= G.U) continue;
                const int c = nt * 8 + 2 * tq;
                const float v0 = acc[nt][2 * half], v1 = acc[nt][2 * half + 1];
                if (c < H) {
                    const float2 gn = *reinterpret_cast<const float2*>(gh_next + i * H + c);
                    *reinterpret_cast<float2*>(gh_cur + i * H + c) = make_float2(gn.x + v0, gn.y + v1);
                } else {
                    *reinterpret_cast<float2*>(gam + i * H + (c - H)) = make_float2(v0, v1);
                }
            }
        }
        __syncwarp();
    }
    atomicAdd(&sb[2 * lane], db0);
    atomicAdd(&sb[2 * lane + 1], db1);
    __syncthreads();
    if (threadIdx.x < H) bpart[blockIdx.x * H + threadIdx.x] = sb[threadIdx.x];
}

// Layer backward, part b: transposed aggregation gh[j] += w_ij gam[i]. Half a warp per edge,
// four features per lane, so an edge is one 256-byte row of 16-byte vector reductions (202 us
// per layer at 119k nodes with one reduction per float, now 121 us).
__global__ void k_layer_bwd_agg(GView G, const float* __restrict__ gam, float* __restrict__ gh_cur) {
    const int lane = threadIdx.x & 31, half = lane >> 4, sub = lane & 15;
    for (long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; i < G.U;
         i += ((long long)gridDim.x * blockDim.x) >> 5) {
        const float4 gm = *reinterpret_cast<const float4*>(gam + i * H + 4 * sub);
        const int e1 = G.row[i + 1] - 1;
        for (int e = G.row[i] + half; e < e1; e += 2) {
            const float w = G.ew[e];
            float* dst = gh_cur + (long long)G.col[e] * H + 4 * sub;
            asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(w * gm.x),
                         "f"(w * gm.y), "f"(w * gm.z), "f"(w * gm.w)
                         : "memory");
        }
    }
}

__device__ __forceinline__ void copy16_async(unsigned dst, const void* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}

// Layer backward, part c: dW = gz^T [h | m] on the tensor cores. A block walks a range of
// 64-node tiles, the next one copied into shared memory while the current one is multiplied
// (16-node tiles without overlap took 55 us at 119k nodes, now 13 us); warp w owns output rows
// 16w..16w+15 (A operand = gz^T via a transposed ldmatrix of the [node][out] tile) and all
// 128 inputs (B operand = [node][in] tile, a transposed ldmatrix); 16 n-tiles x 4
// accumulators per thread, written as a block partial.
constexpr int BW_NODES = 64;
constexpr size_t BW_SMEM = 2 * BW_NODES * (LDG + LDA) * sizeof(bf16);
__global__ void __launch_bounds__(128) k_layer_bwd_w(GView G, const bf16* __restrict__ gz,
                                                     const bf16* __restrict__ a_save, float* __restrict__ wpart) {
    extern __shared__ __align__(16) unsigned char bw_smem[];
    bf16* const Gb = reinterpret_cast<bf16*>(bw_smem);
    bf16* const Ab = Gb + 2 * BW_NODES * LDG;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    float acc[16][4];
#pragma unroll
    for (int nt = 0; nt < 16; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    const long long ntiles = (G.U + BW_NODES - 1) / BW_NODES;
    // gz (64 x 64) and [h | m] (64 x 128) of a tile; rows past U are zero
    auto stage = [&](long long tile, int b) {
        const long long base = tile * BW_NODES;
        const unsigned gs = smem_u32(Gb + b * BW_NODES * LDG), as = smem_u32(Ab + b * BW_NODES * LDA);
        for (int k = threadIdx.x; k < BW_NODES * (H / 8); k += 128) {
            const int t = k / (H / 8), c = (k % (H / 8)) * 8;
            const bool live = base + t < G.U;
            copy16_async(gs + (t * LDG + c) * 2, gz + (live ? base + t : 0) * H + c, live);
        }
        for (int k = threadIdx.x; k < BW_NODES * (KIN / 8); k += 128) {
            const int t = k / (KIN / 8), c = (k % (KIN / 8)) * 8;
            const bool live = base + t < G.U;
            copy16_async(as + (t * LDA + c) * 2, a_save + (live ? base + t : 0) * KIN + c, live);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int b = 0;
    if (blockIdx.x < ntiles) stage(blockIdx.x, 0);
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, b ^= 1) {
        if (tile + gridDim.x < ntiles) {
            stage(tile + gridDim.x, b ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const bf16* Gs = Gb + b * BW_NODES * LDG;
        const bf16* As = Ab + b * BW_NODES * LDA;
#pragma unroll
        for (int ks = 0; ks < BW_NODES / 16; ++ks) {
            // A (m = out, k = node) = gz^T: matrices (out 0-7 | 8-15) x (node 0-7 | 8-15) from Gs[node][out]
            unsigned a0, a1, a2, a3;
            {
                const int mat = lane >> 3, r = lane & 7;
                const int node = ks * 16 + r + ((mat >> 1) << 3), out = warp * 16 + ((mat & 1) << 3);
                ldsm_x4_t(smem_u32(Gs + node * LDG + out), a0, a1, a2, a3);
            }
#pragma unroll
            for (int nt = 0; nt < 16; ++nt) {
                unsigned b0, b1;
                // B (k = node, n = in) from As[node][in]: transposed ldmatrix
                ldsm_x2_t(smem_u32(As + (ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LDA + nt * 8), b0, b1);
                mma16816(acc[nt], a0, a1, a2, a3, b0, b1);
            }
        }
        __syncthreads();  // the next stage overwrites this buffer
    }
    float* out = wpart + (size_t)blockIdx.x * H * KIN;
#pragma unroll
    for (int nt = 0; nt < 16; ++nt) {
        const int c = nt * 8 + 2 * tq;
        const int r0 = warp * 16 + g;
        *reinterpret_cast<float2*>(out + r0 * KIN + c) = make_float2(acc[nt][0], acc[nt][1]);
        *reinterpret_cast<float2*>(out + (r0 + 8) * KIN + c) = make_float2(acc[nt][2], acc[nt][3]);
    }
}

// Encoder backward: gz0 = gh0 * (z0 > 0); block partials of dW_enc (64 x 4) and db_enc. One
// warp per node, two features per lane summed in registers over the warp's nodes (bound by its
// 528 bytes per node; shared-memory atomics per node and weight took 685 us at 119k nodes, now
// 32 us).
__global__ void __launch_bounds__(256) k_enc_bwd(GView G, const float* __restrict__ r, const float* __restrict__ gh0,
                                                 const float* __restrict__ z0, float* __restrict__ part) {
    __shared__ float sg[8][OFF_L0];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float gw[2][NF] = {}, gb[2] = {0.f, 0.f};
    const long long nw = gridDim.x * 8LL;
#pragma unroll 4
    for (long long i = blockIdx.x * 8LL + warp; i < G.U; i += nw) {
        float x[NF];
        features(G, r, i, x);
        const float2 gh = *reinterpret_cast<const float2*>(gh0 + i * H + 2 * lane);
        const float2 z = *reinterpret_cast<const float2*>(z0 + i * H + 2 * lane);
        const float g0 = z.x > 0.f ? gh.x : 0.f, g1 = z.y > 0.f ? gh.y : 0.f;
        gb[0] += g0;
        gb[1] += g1;
#pragma unroll
        for (int f = 0; f < NF; ++f) {  // (a masked gradient takes nothing from a non-finite feature)
            if (g0 != 0.f) gw[0][f] += g0 * x[f];
            if (g1 != 0.f) gw[1][f] += g1 * x[f];
        }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        sg[warp][OFF_BE + 2 * lane + q] = gb[q];
#pragma unroll
        for (int f = 0; f < NF; ++f) sg[warp][OFF_WE + (2 * lane + q) * NF + f] = gw[q][f];
    }
    add_warps<OFF_L0>(sg, (int)OFF_L0, part + (size_t)blockIdx.x * OFF_L0);
}

// out[k] (+)= sum over nblk rows of part[b * stride + k], fixed order: 32 columns per block, eight
// warps over the rows (one thread per column took 14.7 us for 296 rows, now 4.9 us)
__global__ void __launch_bounds__(256) k_reduce_part(const float* __restrict__ part, int nblk, int stride, int count,
                                                     float* __restrict__ out, int accumulate) {
    __shared__ float sw[8][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (k < count) {
#pragma unroll 8
        for (int b = warp; b < nblk; b += 8) s += part[(size_t)b * stride + k];
    }
    sw[warp][lane] = s;
    __syncthreads();
    if (warp || k >= count) return;
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += sw[w][lane];
    out[k] = accumulate ? out[k] + t : t;
}

// Adam with decoupled weight decay on the FP32 master weights; refreshes the bf16 copies
// of the layer matrices.
__global__ void k_adam(int n, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, float lr, float wd, float b1, float b2, float c1, float c2,
                       float inv_batch, bf16* __restrict__ wbf) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float gk = g[k] * inv_batch;
    m[k] = b1 * m[k] + (1.f - b1) * gk;
    v[k] = b2 * v[k] + (1.f - b2) * gk * gk;
    const float mh = m[k] / c1, vh = v[k] / c2;
    w[k] -= lr * (mh / (sqrtf(vh) + 1e-8f) + wd * w[k]);
    const long long off = (long long)k - (long long)OFF_L0;
    if (off >= 0 && off < (long long)(NL * LSTRIDE)) {
        const int l = (int)(off / LSTRIDE), q = (int)(off % LSTRIDE);
        if (q < H * KIN) wbf[l * H * KIN + q] = __float2bfloat16(w[k]);
    }
}

__global__ void k_w_to_bf16(const float* __restrict__ w, bf16* __restrict__ wbf) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= NL * H * KIN) return;
    const int l = k / (H * KIN), q = k % (H * KIN);
    wbf[k] = __float2bfloat16(w[OFF_L0 + l * LSTRIDE + q]);
}

// |b|^2 (partials as k_loss)
__global__ void __launch_bounds__(256) k_norm2_d(long long U, const double* __restrict__ b, double* part) {
    double acc = 0;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < U; i += gridDim.x * 256LL) acc += b[i] * b[i];
    square_sum_partial(acc, part);
}

// sample input b / |b| and target D x / |b| (float), |b|^2 in *nb2
__global__ void k_make_sample(long long U, const double* __restrict__ b, const double* __restrict__ x,
                              const double* __restrict__ dinv, const double* nb2, float* __restrict__ r,
                              float* __restrict__ t) {
    const double inv = *nb2 > 0 ? 1.0 / sqrt(*nb2) : 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < U; i += (long long)gridDim.x * blockDim.x) {
        r[i] = (float)(b[i] * inv);
        t[i] = (float)(x[i] / dinv[i] * inv);
    }
}

__global__ void k_d2f(long long n, const double* __restrict__ a, const int* __restrict__ map, float* __restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[map ? map[i] : i] = (float)a[i];
}

__global__ void k_f2d_ref(long long n, const float* __restrict__ a, const int* __restrict__ u_of_ref, double* __restrict__ out) {
    for (long long rr = blockIdx.x * (long long)blockDim.x + threadIdx.x; rr < n; rr += (long long)gridDim.x * blockDim.x)
        out[rr] = (double)a[u_of_ref[rr]];
}

// ---- manufactured fields ----
__global__ void k_manufacture(long long U, const int* __restrict__ sorted_of_u, const double* __restrict__ sx,
                              const double* __restrict__ sy, const double* __restrict__ sz, const double* __restrict__ prm,
                              int nmodes, double* __restrict__ xe) {
    for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < U; u += (long long)gridDim.x * blockDim.x) {
        const int k = sorted_of_u[u];
        const double x = sx[k], y = sy[k], z = sz[k];
        double p = prm[0] + prm[1] * z;
        for (int m = 0; m < nmodes; ++m) {
            const double* q = prm + 2 + 5 * m;
            p += q[0] * sin(q[1] * x + q[2] * y + q[3] * z + q[4]);
        }
        xe[u] = p;
    }
}

__global__ void k_rhs(long long U, const int* __restrict__ row, const int* __restrict__ col,
                      const double* __restrict__ val, const double* __restrict__ xe, double* __restrict__ b) {
    long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (u >= U) return;
    double s = 0;
    for (int e = row[u]; e < row[u + 1]; ++e) s += val[e] * xe[col[e]];
    b[u] = s;
}

}  // namespace

// =========================================================================================
// host side
// =========================================================================================
static MpnnState& state(lsmps_ctx* ctx) {
    LSMPS_REQUIRE(ctx->mpnn != nullptr, LSMPS_ERR_STATE, "message-passing network not initialised");
    return *ctx->mpnn;
}

bool mpnn_ready(lsmps_ctx* ctx) { return ctx->mpnn != nullptr; }

void mpnn_destroy(lsmps_ctx* ctx) {
    delete ctx->mpnn;
    ctx->mpnn = nullptr;
}

static void upload_weights(lsmps_ctx* ctx, MpnnState& S) {
    float* dw = S.dw.ensure<float>(NPARAM);
    LSMPS_CUDA(cudaMemcpyAsync(dw, S.w.data(), NPARAM * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
    bf16* wbf = S.wbf.ensure<bf16>(NL * H * KIN);
    k_w_to_bf16<<<blocks_for(NL * H * KIN, 256), 256, 0, ctx->stream>>>(dw, wbf);
    LSMPS_CHECK_LAUNCH();
}

void mpnn_init(lsmps_ctx* ctx, uint32_t seed) {
    if (!ctx->mpnn) ctx->mpnn = new MpnnState();
    MpnnState& S = *ctx->mpnn;
    S.w.assign(NPARAM, 0.f);
    std::mt19937 rng(seed);
    std::normal_distribution<float> nd(0.f, 1.f);
    for (int c = 0; c < H * NF; ++c) S.w[OFF_WE + c] = nd(rng) * std::sqrt(2.f / NF);
    for (int l = 0; l < NL; ++l)
        for (int c = 0; c < H * KIN; ++c) S.w[OFF_L0 + l * LSTRIDE + c] = 0.5f * nd(rng) * std::sqrt(2.f / KIN);
    for (int c = 0; c < H; ++c) S.w[OFF_WD + c] = nd(rng) * std::sqrt(1.f / H);
    S.adam_t = 0;
    S.am.ensure<float>(NPARAM);
    S.av.ensure<float>(NPARAM);
    LSMPS_CUDA(cudaMemsetAsync(S.am.get<float>(), 0, NPARAM * sizeof(float), ctx->stream));
    LSMPS_CUDA(cudaMemsetAsync(S.av.get<float>(), 0, NPARAM * sizeof(float), ctx->stream));
    upload_weights(ctx, S);
    LSMPS_CUDA(cudaStreamSynchronize(ctx->stream));
}

void mpnn_get_weights(lsmps_ctx* ctx, float* w, size_t n) {
    MpnnState& S = state(ctx);
    LSMPS_REQUIRE(n == NPARAM, LSMPS_ERR_ARG, "weight buffer size differs from lsmps_mpnn_param_count()");
    LSMPS_CUDA(cudaMemcpyAsync(S.w.data(), S.dw.get<float>(), NPARAM * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    LSMPS_CUDA(cudaStreamSynchronize(ctx->stream));
    std::memcpy(w, S.w.data(), NPARAM * sizeof(float));
}

void mpnn_set_weights(lsmps_ctx* ctx, const float* w, size_t n) {
    if (!ctx->mpnn) mpnn_init(ctx, 0);
    MpnnState& S = *ctx->mpnn;
    LSMPS_REQUIRE(n == NPARAM, LSMPS_ERR_ARG, "weight buffer size differs from lsmps_mpnn_param_count()");
    S.w.assign(w, w + NPARAM);
    upload_weights(ctx, S);
    LSMPS_CUDA(cudaStreamSynchronize(ctx->stream));
}

// Edge weights and node features of the current assembled system into g.
static void build_graph(lsmps_ctx* ctx, MpnnGraph& g, bool copy_structure) {
    cudaStream_t s = ctx->stream;
    const long long U = ctx->U, nnz = ctx->nnz;
    g.U = U;
    g.nnz = nnz;
    if (copy_structure) {
        int* row = g.row.ensure<int>(U + 1);
        int* col = g.col.ensure<int>(nnz + 1);
        LSMPS_CUDA(cudaMemcpyAsync(row, ctx->A_row.get<int>(), (U + 1) * sizeof(int), cudaMemcpyDeviceToDevice, s));
        LSMPS_CUDA(cudaMemcpyAsync(col, ctx->A_col.get<int>(), nnz * sizeof(int), cudaMemcpyDeviceToDevice, s));
        g.prow = row;
        g.pcol = col;
    } else {
        g.prow = ctx->A_row.get<int>();
        g.pcol = ctx->A_col.get<int>();
    }
    float* ew = g.ew.ensure<float>(nnz + 1);
    float* feat = g.feat.ensure<float>(3 * U + 3);
    float* dg = g.dg.ensure<float>(U + 1);
    double* mean = ctx->scratch.get<double>() + 24;
    double* part = ctx->scratch.get<double>() + 1024;  // MEAN_BLOCKS doubles of the 2048-double scratch
    if (U) {
        k_graph_ew<<<148 * 8, 256, 0, s>>>(U, ctx->A_row.get<int>(), ctx->A_val.get<double>(),
                                          ctx->A_dinv.get<double>(), ew);
        k_diag_partials<<<MEAN_BLOCKS, 256, 0, s>>>(U, ctx->A_dinv.get<double>(), part);
        k_mean_finish<<<1, 256, 0, s>>>(U, part, MEAN_BLOCKS, mean);
        note_launches(2);
        k_graph_feat<<<blocks_for(U, 256), 256, 0, s>>>(U, ctx->A_row.get<int>(), ctx->A_dinv.get<double>(),
                                                       ctx->cls.get<uint8_t>(), ctx->sorted_of_u.get<int>(), mean, feat,
                                                       dg);
        LSMPS_CHECK_LAUNCH();
    }
}

static GView view(const MpnnGraph& g) {
    return GView{g.U,           g.prow,         g.pcol, g.ew.get<float>(), g.feat.get<float>(), g.dg.get<float>(),
                 (float)std::sqrt((double)std::max(1LL, g.U))};
}

static void ensure_workspace(MpnnState& S, long long U, bool training) {
    if (U <= S.cap && (!training || S.z[0].bytes >= (size_t)U * H * sizeof(float))) return;
    const long long cap = std::max(U, S.cap);
    for (int l = 0; l <= NL; ++l) S.h[l].ensure<bf16>(cap * H + 8);
    S.y.ensure<float>(cap + 8);
    if (training) {
        for (int l = 0; l < NL; ++l) S.a[l].ensure<bf16>(cap * KIN + 8);
        for (int l = 0; l <= NL; ++l) S.z[l].ensure<float>(cap * H + 8);
        S.gh[0].ensure<float>(cap * H + 8);
        S.gh[1].ensure<float>(cap * H + 8);
        S.gam.ensure<float>(cap * H + 8);
        S.gz.ensure<bf16>(cap * H + 8);
    }
    S.cap = cap;
}

// Launch shapes of the message-passing layer (k_layer_fwd): gathers in flight (4 NB rows per
// warp), warps per block, node order, blocks per SM.
struct LayerShape {
    int nb, warps;
    bool local;
    int bps;
};
constexpr LayerShape LAYER_SHAPES[] = {{4, 4, false, 4},  {8, 4, false, 4},  {4, 4, false, 6},  {8, 4, false, 6},
                                       {4, 8, true, 3},   {8, 8, true, 3},   {4, 12, true, 2},  {8, 12, true, 2},
                                       {4, 24, true, 1},  {8, 24, true, 1}};

template <int NB, int WARPS, bool LOCAL>
static void launch_layer_kernel(unsigned grid, cudaStream_t s, const GView& G, const bf16* hin, bf16* hout,
                                const bf16* W, const float* b, bf16* as, float* zs) {
    const size_t smem = (size_t)(H * LDA + WARPS * 16 * LDA) * sizeof(bf16) + H * sizeof(float);
    auto k = k_layer_fwd<NB, WARPS, LOCAL>;
    LSMPS_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k<<<grid, WARPS * 32, smem, s>>>(G, hin, hout, W, b, as, zs);
}

static void launch_layer(lsmps_ctx* ctx, MpnnState& S, const GView& G, bool training, int c, int l) {
    const LayerShape& sh = LAYER_SHAPES[c];
    const long long span = 16LL * sh.warps;  // nodes per block and round
    const unsigned lgrid =
        (unsigned)std::max<long long>(1, std::min<long long>((G.U + span - 1) / span, 148LL * sh.bps));
    const float* w = S.dw.get<float>();
    const bf16* wbf = S.wbf.get<bf16>();
    const bf16* hin = S.h[l].get<bf16>();
    bf16* hout = S.h[l + 1].get<bf16>();
    const bf16* W = wbf + l * H * KIN;
    const float* b = w + OFF_L0 + l * LSTRIDE + H * KIN;
    bf16* as = training ? S.a[l].get<bf16>() : nullptr;
    float* zs = training ? S.z[l + 1].get<float>() : nullptr;
    cudaStream_t s = ctx->stream;
#define LSMPS_LAYER_CASE(NB_, W_, L_)                                                     \
    if (sh.nb == NB_ && sh.warps == W_ && sh.local == L_) {                               \
        launch_layer_kernel<NB_, W_, L_>(lgrid, s, G, hin, hout, W, b, as, zs);           \
        LSMPS_CHECK_LAUNCH();                                                             \
        return;                                                                           \
    }
    LSMPS_LAYER_CASE(4, 4, false)
    LSMPS_LAYER_CASE(8, 4, false)
    LSMPS_LAYER_CASE(4, 8, true)
    LSMPS_LAYER_CASE(8, 8, true)
    LSMPS_LAYER_CASE(4, 12, true)
    LSMPS_LAYER_CASE(8, 12, true)
    LSMPS_LAYER_CASE(4, 24, true)
    LSMPS_LAYER_CASE(8, 24, true)
#undef LSMPS_LAYER_CASE
    LSMPS_REQUIRE(false, LSMPS_ERR_STATE, "unknown network layer launch shape");
}

// The autotuned launch shape of the layer for this graph size (layer 0 is the timed launch:
// it reads h[0] and writes h[1], so repeating it is harmless).
static int layer_shape(lsmps_ctx* ctx, MpnnState& S, const GView& G, bool training) {
    static const std::vector<std::string> names = [] {
        std::vector<std::string> v;
        for (const LayerShape& sh : LAYER_SHAPES)
            v.push_back("gathers" + std::to_string(4 * sh.nb) + "/warps" + std::to_string(sh.warps) +
                        (sh.local ? "-local" : "") + "/blocks" + std::to_string(sh.bps) + "xSM");
        return v;
    }();
    return autotune(ctx, "mpnn_layer_fwd", G.U, names, 2, [&](int c) { launch_layer(ctx, S, G, training, c, 0); });
}

// Forward pass over graph g for input r (float, unit norm); y in S.y.
static void forward(lsmps_ctx* ctx, MpnnState& S, const GView& G, const float* r, bool training) {
    cudaStream_t s = ctx->stream;
    ensure_workspace(S, G.U, training);
    if (!G.U) return;
    const float* w = S.dw.get<float>();
    const unsigned grid = std::min<unsigned>(blocks_for(G.U, 256), 148 * 8);
    k_enc<<<grid, 256, 0, s>>>(G, r, w, S.h[0].get<bf16>(), training ? S.z[0].get<float>() : nullptr);
    LSMPS_CHECK_LAUNCH();
    const int c = layer_shape(ctx, S, G, training);
    for (int l = 0; l < NL; ++l) launch_layer(ctx, S, G, training, c, l);
    k_dec<<<grid, 256, 0, s>>>(G, S.h[NL].get<bf16>(), w, S.y.get<float>());
    LSMPS_CHECK_LAUNCH();
}

// |y - t|^2 (t null: |y|^2) into *out (device, in S.red).
static void square_sum(lsmps_ctx* ctx, MpnnState& S, long long U, const float* y, const float* t, double* out) {
    double* part = S.red.get<double>() + 8;
    k_loss<<<LOSS_BLOCKS, 256, 0, ctx->stream>>>(U, y, t, part);
    LSMPS_CHECK_LAUNCH();
    k_sum_partials<<<1, 32, 0, ctx->stream>>>(part, LOSS_BLOCKS, out);
    LSMPS_CHECK_LAUNCH();
}

// Loss of (g, r, t) and, when grad != nullptr, its gradient accumulated into grad (device).
static double loss_and_grad(lsmps_ctx* ctx, MpnnState& S, const GView& G, const float* r, const float* t, double tnorm2,
                            float* grad, bool accumulate) {
    cudaStream_t s = ctx->stream;
    forward(ctx, S, G, r, grad != nullptr);
    double* lsum = S.red.ensure<double>(8 + LOSS_BLOCKS);
    const int kind = S.loss_kind;
    float* ay = S.ay.ensure<float>(S.cap + 8);
    if (kind != 1) {
        square_sum(ctx, S, G.U, S.y.get<float>(), t, lsum);
    }
    if (kind != 0) {
        k_apply_scaled<<<blocks_for(8 * G.U, 256), 256, 0, s>>>(G, S.y.get<float>(), ay);
        LSMPS_CHECK_LAUNCH();
        square_sum(ctx, S, G.U, ay, r, lsum + 1);  // |r - A D^-1 y|^2, |r| = 1
    }
    if (grad) {
        const float* w = S.dw.get<float>();
        const bf16* wbf = S.wbf.get<bf16>();
        const int nb = 148 * 2;
        LSMPS_CUDA(cudaFuncSetAttribute(k_layer_bwd_w, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BW_SMEM));
        float* part = S.gpart.ensure<float>((size_t)WG_BLOCKS * H * KIN + 16);
        float* gh_next = S.gh[0].get<float>();
        float* gh_cur = S.gh[1].get<float>();
        // dL/dy, then the decoder
        float* gy = S.gy.ensure<float>(S.cap + 8);
        float* q = S.q.ensure<float>(S.cap + 8);
        if (kind != 0) {
            LSMPS_CUDA(cudaMemsetAsync(q, 0, G.U * sizeof(float), s));
            k_scatter_res<<<blocks_for(8 * G.U, 256), 256, 0, s>>>(G, r, ay, q);
            LSMPS_CHECK_LAUNCH();
        }
        k_dldy<<<blocks_for(G.U, 256), 256, 0, s>>>(G.U, S.y.get<float>(), t, r, ay, q, G.dg,
                                                    (float)(2.0 / std::max(tnorm2, 1e-30)), kind, gy);
        k_dec_bwd<<<nb, 256, 0, s>>>(G, gy, S.h[NL].get<bf16>(), w, gh_next, part);
        LSMPS_CHECK_LAUNCH();
        k_reduce_part<<<blocks_for(H + 1, 32), 256, 0, s>>>(part, nb, H + 1, H + 1, grad + OFF_WD, accumulate ? 1 : 0);
        LSMPS_CHECK_LAUNCH();
        const unsigned lgrid = std::min<unsigned>((unsigned)((G.U + 63) / 64), 148 * 4);
        for (int l = NL - 1; l >= 0; --l) {
            float* bpart = part;  // [lgrid][64]
            k_layer_bwd_a<<<lgrid, 128, 0, s>>>(G, gh_next, S.z[l + 1].get<float>(), wbf + l * H * KIN,
                                                S.gz.get<bf16>(), gh_cur, S.gam.get<float>(), bpart);
            LSMPS_CHECK_LAUNCH();
            k_reduce_part<<<blocks_for(H, 32), 256, 0, s>>>(bpart, (int)lgrid, H, H, grad + OFF_L0 + l * LSTRIDE + H * KIN,
                                          accumulate ? 1 : 0);
            LSMPS_CHECK_LAUNCH();
            k_layer_bwd_agg<<<std::min<unsigned>(blocks_for(G.U * 32, 256), 148 * 16), 256, 0, s>>>(
                G, S.gam.get<float>(), gh_cur);
            LSMPS_CHECK_LAUNCH();
            k_layer_bwd_w<<<WG_BLOCKS, 128, BW_SMEM, s>>>(G, S.gz.get<bf16>(), S.a[l].get<bf16>(), part);
            LSMPS_CHECK_LAUNCH();
            k_reduce_part<<<blocks_for(H * KIN, 32), 256, 0, s>>>(part, WG_BLOCKS, H * KIN, H * KIN,
                                                                   grad + OFF_L0 + l * LSTRIDE, accumulate ? 1 : 0);
            LSMPS_CHECK_LAUNCH();
            std::swap(gh_next, gh_cur);
        }
        // encoder (gh_next holds dL/dh0)
        k_enc_bwd<<<nb, 256, 0, s>>>(G, r, gh_next, S.z[0].get<float>(), part);
        LSMPS_CHECK_LAUNCH();
        k_reduce_part<<<blocks_for(OFF_L0, 32), 256, 0, s>>>(part, nb, (int)OFF_L0, (int)OFF_L0, grad, accumulate ? 1 : 0);
        LSMPS_CHECK_LAUNCH();
    }
    double h[2] = {0, 0};
    LSMPS_CUDA(cudaMemcpyAsync(h, lsum, sizeof(h), cudaMemcpyDeviceToHost, s));
    LSMPS_CUDA(cudaStreamSynchronize(s));
    return (kind != 1 ? h[0] / std::max(tnorm2, 1e-30) : 0.0) + (kind != 0 ? h[1] : 0.0);
}

void mpnn_add_sample(lsmps_ctx* ctx) {
    MpnnState& S = state(ctx);
    LSMPS_REQUIRE(ctx->have_ppe && ctx->have_solution, LSMPS_ERR_STATE, "a training pair needs a solved system");
    cudaStream_t s = ctx->stream;
    const long long U = ctx->U;
    if (S.graph_gen != ctx->assembly_gen || S.graphs.empty()) {
        S.graphs.emplace_back(new MpnnGraph());
        build_graph(ctx, *S.graphs.back(), true);
        S.graph_gen = ctx->assembly_gen;
    }
    auto smp = std::make_unique<MpnnSample>();
    smp->graph = (int)S.graphs.size() - 1;
    float* r = smp->r.ensure<float>(U + 1);
    float* t = smp->t.ensure<float>(U + 1);
    double* nb2 = ctx->scratch.get<double>() + 28;
    double* red = S.red.ensure<double>(8 + LOSS_BLOCKS);
    k_norm2_d<<<LOSS_BLOCKS, 256, 0, s>>>(U, ctx->A_b.get<double>(), red + 8);
    k_sum_partials<<<1, 32, 0, s>>>(red + 8, LOSS_BLOCKS, nb2);
    note_launches(1);
    k_make_sample<<<1184, 256, 0, s>>>(U, ctx->A_b.get<double>(), ctx->vx.get<double>(), ctx->A_dinv.get<double>(),
                                        nb2, r, t);
    LSMPS_CHECK_LAUNCH();
    double* tn = red + 1;  // |t|^2, for the relative loss
    square_sum(ctx, S, U, t, nullptr, tn);
    LSMPS_CUDA(cudaMemcpyAsync(&smp->tnorm2, tn, sizeof(double), cudaMemcpyDeviceToHost, s));
    LSMPS_CUDA(cudaStreamSynchronize(s));
    S.samples.push_back(std::move(smp));
}

void mpnn_clear_samples(lsmps_ctx* ctx) {
    MpnnState& S = state(ctx);
    S.samples.clear();
    S.graphs.clear();
    S.graph_gen = -1;
}

int mpnn_sample_count(lsmps_ctx* ctx) { return ctx->mpnn ? (int)ctx->mpnn->samples.size() : 0; }

void mpnn_grad(lsmps_ctx* ctx, int index, float* grad_host, float* loss) {
    MpnnState& S = state(ctx);
    LSMPS_REQUIRE(index >= 0 && index < (int)S.samples.size(), LSMPS_ERR_ARG, "sample index out of range");
    const MpnnSample& smp = *S.samples[index];
    float* grad = S.grad.ensure<float>(NPARAM);
    const double L = loss_and_grad(ctx, S, view(*S.graphs[smp.graph]), smp.r.get<float>(), smp.t.get<float>(),
                                   smp.tnorm2, grad, false);
    if (loss) *loss = (float)L;
    if (grad_host) {
        LSMPS_CUDA(cudaMemcpyAsync(grad_host, grad, NPARAM * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
        LSMPS_CUDA(cudaStreamSynchronize(ctx->stream));
    }
}

void mpnn_train(lsmps_ctx* ctx, const lsmps_mpnn_train_opts* o, float* loss_out) {
    MpnnState& S = state(ctx);
    LSMPS_REQUIRE(!S.samples.empty(), LSMPS_ERR_STATE, "no training samples");
    LSMPS_REQUIRE(o->steps >= 0 && o->batch >= 1 && o->loss >= 0 && o->loss <= 2, LSMPS_ERR_ARG, "training options");
    S.loss_kind = o->loss;
    cudaStream_t s = ctx->stream;
    float* grad = S.grad.ensure<float>(NPARAM);
    std::mt19937 rng(o->seed);
    std::vector<int> order(S.samples.size());
    for (size_t k = 0; k < order.size(); ++k) order[k] = (int)k;
    size_t cursor = order.size();
    double last = 0;
    const float b1 = 0.9f, b2 = 0.999f;
    for (int step = 0; step < o->steps; ++step) {
        double sum = 0;
        for (int k = 0; k < o->batch; ++k) {
            if (cursor >= order.size()) {
                std::shuffle(order.begin(), order.end(), rng);
                cursor = 0;
            }
            const MpnnSample& smp = *S.samples[order[cursor++]];
            sum += loss_and_grad(ctx, S, view(*S.graphs[smp.graph]), smp.r.get<float>(), smp.t.get<float>(), smp.tnorm2,
                                 grad, k > 0);
        }
        ++S.adam_t;
        const float c1 = 1.f - std::pow(b1, (float)S.adam_t), c2 = 1.f - std::pow(b2, (float)S.adam_t);
        k_adam<<<blocks_for(NPARAM, 256), 256, 0, s>>>((int)NPARAM, S.dw.get<float>(), grad, S.am.get<float>(),
                                                       S.av.get<float>(), o->lr, o->weight_decay, b1, b2, c1, c2,
                                                       1.f / (float)o->batch, S.wbf.get<bf16>());
        LSMPS_CHECK_LAUNCH();
        last = sum / o->batch;
    }
    LSMPS_CUDA(cudaMemcpyAsync(S.w.data(), S.dw.get<float>(), NPARAM * sizeof(float), cudaMemcpyDeviceToHost, s));
    LSMPS_CUDA(cudaStreamSynchronize(s));
    if (loss_out) *loss_out = (float)last;
}

// Network guess for the current assembled system: y = net(rhs) (sorted numbering, float).
void mpnn_warm_start(lsmps_ctx* ctx, const float* rhs, float* y) {
    MpnnState& S = state(ctx);
    if (S.infer_gen != ctx->assembly_gen) {
        build_graph(ctx, S.infer, false);
        S.infer_gen = ctx->assembly_gen;
    }
    GView G = view(S.infer);
    forward(ctx, S, G, rhs, false);
    LSMPS_CUDA(cudaMemcpyAsync(y, S.y.get<float>(), G.U * sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
}

// One message-passing layer (layer 0, the tuned shape) on the current assembled system with
// the loaded weights; input features from the unit right-hand side b / |b|.
void mpnn_kernel_bench(lsmps_ctx* ctx, int reps, double* ms, double* bytes) {
    MpnnState& S = state(ctx);
    LSMPS_REQUIRE(ctx->have_ppe, LSMPS_ERR_STATE, "layer bench needs an assembled system");
    const long long U = ctx->U;
    if (U == 0) { *ms = 0; *bytes = 0; return; }
    float* rf = ctx->fph.ensure<float>(U + 1);
    float* yf = ctx->fx.ensure<float>(U + 1);
    std::vector<float> ones((size_t)U, (float)(1.0 / std::sqrt((double)U)));
    LSMPS_CUDA(cudaMemcpyAsync(rf, ones.data(), U * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
    mpnn_warm_start(ctx, rf, yf);  // graph, h[0], tuned shape
    GView G = view(S.infer);
    const int c = layer_shape(ctx, S, G, false);
    launch_layer(ctx, S, G, false, c, 0);
    ev_record(ctx, 14);
    for (int r = 0; r < reps; ++r) launch_layer(ctx, S, G, false, c, 0);
    ev_record(ctx, 15);
    *ms = ev_elapsed(ctx, 14, 15) / reps;
    *bytes = 256.0 * U + 8.0 * ctx->nnz;
}

void mpnn_infer(lsmps_ctx* ctx, const double* r_ref, double* y_ref) {
    state(ctx);
    LSMPS_REQUIRE(ctx->have_ppe, LSMPS_ERR_STATE, "inference needs an assembled system");
    cudaStream_t s = ctx->stream;
    const long long U = ctx->U;
    double* rd = ctx->vtmp.ensure<double>(2 * U + 2);
    float* rf = ctx->fph.ensure<float>(U + 1);
    float* yf = ctx->fx.ensure<float>(U + 1);
    LSMPS_CUDA(cudaMemcpyAsync(rd, r_ref, U * sizeof(double), cudaMemcpyHostToDevice, s));
    // reference numbering -> solver numbering: rf[u_of_ref[rr]] = r[rr]
    k_d2f<<<1184, 256, 0, s>>>(U, rd, ctx->u_of_ref.get<int>(), rf);
    LSMPS_CHECK_LAUNCH();
    mpnn_warm_start(ctx, rf, yf);
    k_f2d_ref<<<1184, 256, 0, s>>>(U, yf, ctx->u_of_ref.get<int>(), rd + U);
    LSMPS_CHECK_LAUNCH();
    LSMPS_CUDA(cudaMemcpyAsync(y_ref, rd + U, U * sizeof(double), cudaMemcpyDeviceToHost, s));
    LSMPS_CUDA(cudaStreamSynchronize(s));
}

void mpnn_save(lsmps_ctx* ctx, const char* path) {
    MpnnState& S = state(ctx);
    std::vector<float> w(NPARAM);
    mpnn_get_weights(ctx, w.data(), NPARAM);
    FILE* f = std::fopen(path, "wb");
    LSMPS_REQUIRE(f, LSMPS_ERR_IO, std::string("cannot write ") + path);
    const char magic[8] = {'L', 'S', 'M', 'P', 'N', 'N', '0', '1'};
    const uint64_t n = NPARAM;
    bool ok = std::fwrite(magic, 1, 8, f) == 8 && std::fwrite(&n, sizeof(n), 1, f) == 1 &&
              std::fwrite(w.data(), sizeof(float), NPARAM, f) == NPARAM;
    std::fclose(f);
    (void)S;
    LSMPS_REQUIRE(ok, LSMPS_ERR_IO, std::string("short write to ") + path);
}

void mpnn_load(lsmps_ctx* ctx, const char* path) {
    FILE* f = std::fopen(path, "rb");
    LSMPS_REQUIRE(f, LSMPS_ERR_IO, std::string("cannot read ") + path);
    char magic[8];
    uint64_t n = 0;
    std::vector<float> w(NPARAM);
    bool ok = std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, "LSMPNN01", 8) == 0 &&
              std::fread(&n, sizeof(n), 1, f) == 1 && n == NPARAM &&
              std::fread(w.data(), sizeof(float), NPARAM, f) == NPARAM;
    std::fclose(f);
    LSMPS_REQUIRE(ok, LSMPS_ERR_IO, std::string("not a network weights file: ") + path);
    mpnn_set_weights(ctx, w.data(), NPARAM);
}

size_t mpnn_param_count() { return NPARAM; }

void ppe_manufacture(lsmps_ctx* ctx, const double* params, int nmodes) {
    LSMPS_REQUIRE(ctx->have_ppe && !ctx->ppe_loaded, LSMPS_ERR_STATE,
                  "manufactured fields need an assembled particle system");
    LSMPS_REQUIRE(params && nmodes >= 0 && nmodes <= 64, LSMPS_ERR_ARG, "manufactured field parameters");
    cudaStream_t s = ctx->stream;
    const long long U = ctx->U;
    const int np = 2 + 5 * nmodes;
    double* prm = ctx->scratch.get<double>() + 64;  // 512-double scratch region
    LSMPS_CUDA(cudaMemcpyAsync(prm, params, np * sizeof(double), cudaMemcpyHostToDevice, s));
    if (U) {
        k_manufacture<<<1184, 256, 0, s>>>(U, ctx->sorted_of_u.get<int>(), ctx->sx.get<double>(), ctx->sy.get<double>(),
                                           ctx->sz.get<double>(), prm, nmodes, ctx->A_xexact.get<double>());
        k_rhs<<<blocks_for(U, 256), 256, 0, s>>>(U, ctx->A_row.get<int>(), ctx->A_col.get<int>(), ctx->A_val.get<double>(),
                                                 ctx->A_xexact.get<double>(), ctx->A_b.get<double>());
        LSMPS_CHECK_LAUNCH();
    }
    LSMPS_CUDA(cudaStreamSynchronize(s));
    ctx->have_solution = false;
}

}  // namespace lsmps_gpu
