// gnn.cu — the learned warm start's network (sps_gnn_* in include/sps_gnn.h):
// forward, hand-written backward, loss and Adam, all as CUDA kernels.
//
// Activations are kept per instance and node, row-major with the hidden width
// innermost ([instance][node][H], FP32), so every per-node kernel runs over the
// flattened node list of the whole batch and the weight gradients are sums
// over it.  With H = 64 the dense updates, forward and backward, run on the tensor
// cores (k_node64, k_back64: tcgen05, FP32 as three BF16 parts); on graphs with few
// rows the M products are made on the constraint side, whose own update is
// compensated FP32 (k_con_update).  H = 32 keeps register-tiled FP32 contractions and
// CSR SpMM aggregations.  Every reduction (weight gradients, losses, pooling) writes
// per-block partials that are summed in block order: training is bitwise
// reproducible.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/sps_gnn.h"
#include "gnn_internal.cuh"
#include "nvtx.cuh"

namespace {

constexpr int kT = 256;          // threads per block
constexpr int kTile = 32;        // nodes per tile in the dense kernels
constexpr int kMaxF = 8;         // input feature width limit

__device__ __forceinline__ float relu(float v) { return v > 0.f ? v : 0.f; }

// ---- input layer: h = relu(W f + b), W is H x F ------------------------------------
template <int H>
__global__ void __launch_bounds__(kT) k_input(const float* __restrict__ f, int64_t nodes, int F,
                                              const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias,
                                              float* __restrict__ h) {
    const int64_t total = nodes * H;
    for (int64_t t = blockIdx.x * (int64_t)kT + threadIdx.x; t < total; t += (int64_t)gridDim.x * kT) {
        const int64_t v = t / H;
        const int o = int(t % H);
        float acc = bias[o];
        for (int q = 0; q < F; ++q) acc += __bfloat162float(W[o * F + q]) * f[v * F + q];
        h[t] = relu(acc);
    }
}

// ---- aggregation: out[s, r] (+)= sum_k val[k] * in[s, idx[k]] ----------------------
// One warp per destination row of one instance; lane l owns features 2l, 2l+1
// (H = 64) or l (H = 32).
template <int H>
__global__ void __launch_bounds__(kT) k_agg(const int32_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                                            const float* __restrict__ val, const float* __restrict__ in,
                                            float* __restrict__ out, int n_dst, int n_src, int batch, int accumulate) {
    const int lane = threadIdx.x & 31;
    const int64_t rows = (int64_t)n_dst * batch;
    for (int64_t w = (blockIdx.x * (int64_t)kT + threadIdx.x) >> 5; w < rows; w += ((int64_t)gridDim.x * kT) >> 5) {
        const int64_t s = w / n_dst;
        const int r = int(w % n_dst);
        const float* src = in + s * (int64_t)n_src * H;
        const int b = ptr[r], e = ptr[r + 1];
        if (H == 64) {
            float2 acc = make_float2(0.f, 0.f);
            int k = b;
            for (; k + 4 <= e; k += 4) {
                float2 v[4];
                float a[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    a[u] = __ldg(val + k + u);
                    v[u] = __ldg(reinterpret_cast<const float2*>(src + (int64_t)__ldg(idx + k + u) * H) + lane);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) { acc.x += a[u] * v[u].x; acc.y += a[u] * v[u].y; }
            }
            for (; k < e; ++k) {
                const float a = __ldg(val + k);
                const float2 v = __ldg(reinterpret_cast<const float2*>(src + (int64_t)__ldg(idx + k) * H) + lane);
                acc.x += a * v.x;
                acc.y += a * v.y;
            }
            float2* o = reinterpret_cast<float2*>(out + w * H) + lane;
            if (accumulate) { const float2 p = *o; acc.x += p.x; acc.y += p.y; }
            *o = acc;
        } else {
            float acc = 0.f;
            for (int k = b; k < e; ++k) acc += __ldg(val + k) * __ldg(src + (int64_t)__ldg(idx + k) * H + lane);
            float* o = out + w * H + lane;
            if (accumulate) acc += *o;
            *o = acc;
        }
    }
}

// ---- dense node update, H = 32: out = relu(U h + M a + b) --------------------------
// A register-tiled FP32 contraction of the tile's [h | a] (kUpdNodes x 2H) with
// W^T = [U | M]^T (2H x H).  The block stages W^T (BF16 widened to FP32) once
// and, per tile, the nodes' h and a rows as they lie in memory (16-byte loads
// and stores).  Thread t owns nodes ng + 32 i (i < 4, ng = t / 8) and outputs
// 4 og + c (og = t % 8, c < 4): per four input features it reads four 16-byte node
// vectors and four 16-byte weight vectors from shared memory for 16 FMAs per
// feature.  Each output is bias + sum over k of W[o][k] x[k]
// in k order (h's features, then a's), one fmaf per k.
constexpr int kUpdNodes = 128;                 // nodes per tile
constexpr int kUpdStride = 2 * 32 + 4;         // padded tile row: 4 consecutive rows hit distinct banks

__global__ void __launch_bounds__(kT, 2) k_update(const float* __restrict__ h, const float* __restrict__ a,
                                                  const __nv_bfloat16* __restrict__ U,
                                                  const __nv_bfloat16* __restrict__ M,
                                                  const float* __restrict__ bias, float* __restrict__ out,
                                                  int64_t nodes) {
    static_assert(kT == 256, "thread layout: 8 output groups x 32 node groups");
    constexpr int H = 32, K2 = 2 * H, S = kUpdStride;
    extern __shared__ __align__(16) float sm[];
    float* Wt = sm;                           // [k][o], k < H from U, k >= H from M
    float* X = Wt + K2 * H;                   // [node][S]: h (k < H) then a
    for (int t = threadIdx.x; t < K2 * H; t += kT) {
        const int o = t / K2, k = t % K2;
        Wt[k * H + o] = __bfloat162float(k < H ? U[o * H + k] : M[o * H + (k - H)]);
    }
    const int og = threadIdx.x & 7, ng = threadIdx.x >> 3;
    const float* bp = bias + 4 * og;               // the parameter block's offsets need not be 16-byte aligned
    const float4 bo = make_float4(bp[0], bp[1], bp[2], bp[3]);
    const int64_t tiles = (nodes + kUpdNodes - 1) / kUpdNodes;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t base = tile * kUpdNodes;
        __syncthreads();
        for (int t = threadIdx.x; t < kUpdNodes * (K2 / 4); t += kT) {
            const int nd = t / (K2 / 4), q = t % (K2 / 4);
            const int64_t v = base + nd;
            float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
            if (v < nodes)
                val = q < H / 4 ? *reinterpret_cast<const float4*>(h + v * H + 4 * q)
                                : *reinterpret_cast<const float4*>(a + v * H + 4 * (q - H / 4));
            *reinterpret_cast<float4*>(X + nd * S + 4 * q) = val;
        }
        __syncthreads();
        float4 acc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = bo;
#pragma unroll 2
        for (int k = 0; k < K2; k += 4) {
            float4 xv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) xv[i] = *reinterpret_cast<const float4*>(X + (ng + 32 * i) * S + k);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const float4 w = *reinterpret_cast<const float4*>(Wt + (k + kk) * H + 4 * og);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float x = kk == 0 ? xv[i].x : kk == 1 ? xv[i].y : kk == 2 ? xv[i].z : xv[i].w;
                    acc[i].x = fmaf(w.x, x, acc[i].x);
                    acc[i].y = fmaf(w.y, x, acc[i].y);
                    acc[i].z = fmaf(w.z, x, acc[i].z);
                    acc[i].w = fmaf(w.w, x, acc[i].w);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t v = base + ng + 32 * i;
            if (v < nodes)
                *reinterpret_cast<float4*>(out + v * H + 4 * og) =
                    make_float4(relu(acc[i].x), relu(acc[i].y), relu(acc[i].z), relu(acc[i].w));
        }
    }
}

// ---- tensor-core helpers ---------------------------------------------------------------
namespace tc {
constexpr int kWaitPolls = 1 << 20;
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// K-major operand, 128-byte swizzle, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (int i = 0; i < kWaitPolls; ++i) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

// Of a kernel that gives up, for the MMAs in flight before it frees their memory: out of line,
// so that the loops keep their registers.
__device__ __noinline__ void last_wait(uint32_t bar, uint32_t parity) { mbar_wait(bar, parity); }

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
}  // namespace tc

// ---- the variable side's node update on the tensor cores (H = 64) --------------------
// relu(U h + M a + b) with a_j = sum_i a_ij hc_i is relu(U h + sum_i a_ij (M hc_i) + b):
// M is applied to the constraint nodes (a few thousand) instead of to every
// variable node's aggregate, so the aggregate is neither written nor read and
// the large contraction has K = 64 instead of 128 (graphs with few rows, forward64;
// on others Two adds the second product of the aggregate).  What is left is a stream: h
// in, out (512 bytes a node), the rows of M hc from L2.  On 1.28M nodes (16
// instances of the 200 x 400 family) a layer's aggregation and update took 180 +
// 300 us; now 229 us (0.66 GB, 96 us at the measured HBM rate: the chain staging ->
// MMA -> edges -> read-back of each tile, two blocks an SM, is what is left).
//
// FP32 activations as three BF16 parts (8 bits of mantissa each, all 24), the
// weights exact in BF16: three products per step, accumulated in FP32, agree
// with FP32 arithmetic.  A tile is 128 nodes: a part is 128 rows of 128 bytes
// (128-byte swizzle: 16-byte piece q of row r at piece q ^ (r & 7)), staged by all
// threads from registers that were loaded while the last tile was computed.
// Every wait is bounded; a block that gives up sets *err and stops.
namespace bf {
constexpr int kPart = 128 * 128;              // one BF16 part of a 128-node tile (16 KB)
constexpr int kW = 64 * 128;                  // a 64 x 64 weight matrix (8 KB)
// instruction descriptor: D F32, A and B BF16
__host__ __device__ constexpr uint32_t idesc(int M, int N, bool transA, bool transB) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((transA ? 1u : 0u) << 15) | ((transB ? 1u : 0u) << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
template <uint32_t Idesc>
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "n"(Idesc), "r"(accumulate) : "memory");
}
// four floats as three parts of four BF16 values, cut by truncation (masks and exact
// subtractions: the three parts of 8 bits add up to the float itself)
__device__ __forceinline__ uint32_t upper(float a, float b) {
    return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
__device__ __forceinline__ float cut(float v) { return __uint_as_float(__float_as_uint(v) & 0xffff0000u); }
template <bool Infinite>
__device__ __forceinline__ void split(const float4& x, uint2 (&p)[3]) {
    float4 r = x;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        p[q] = make_uint2(upper(r.x, r.y), upper(r.z, r.w));
        if (q < 2) r = make_float4(r.x - cut(r.x), r.y - cut(r.y), r.z - cut(r.z), r.w - cut(r.w));
        // Infinite: an infinity is its own first part.  inf - inf makes the sum of the parts NaN,
        // and a ReLU makes 0 of that (gradients pass through none: they stay NaN)
        if (Infinite && q == 0 && !(fabsf(x.x) + fabsf(x.y) + fabsf(x.z) + fabsf(x.w) < INFINITY))
            r = make_float4(isfinite(x.x) ? r.x : 0.f, isfinite(x.y) ? r.y : 0.f, isfinite(x.z) ? r.z : 0.f,
                            isfinite(x.w) ? r.w : 0.f);
    }
}
// piece f (four floats) of row r of a tile's parts
template <bool Infinite>
__device__ __forceinline__ void put(unsigned char* parts, int r, int f, const float4& x) {
    uint2 p[3];
    split<Infinite>(x, p);
    const int off = r * 128 + (((f >> 1) ^ (r & 7)) << 4) + ((f & 1) << 3);
#pragma unroll
    for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(parts + q * kPart + off) = p[q];
}
// W (64 x 64 BF16, row-major, any 2-byte alignment) as rows of 128 bytes; Trans: its transpose
template <bool Trans>
__device__ __forceinline__ void put_weights(unsigned char* dst, const __nv_bfloat16* __restrict__ W) {
    for (int t = threadIdx.x; t < 64 * 64; t += blockDim.x) {
        const int o = t >> 6, k = t & 63, r = Trans ? k : o, c = Trans ? o : k;
        *reinterpret_cast<__nv_bfloat16*>(dst + r * 128 + (((c >> 3) ^ (r & 7)) << 4) + ((c & 7) << 1)) = W[t];
    }
}
}  // namespace bf

// Input layer of a node with four features, outputs 4 f .. 4 f + 3 (as k_input).
struct InW {
    float4 w[4];
    float4 b;
    __device__ __forceinline__ void load(const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias, int f) {
        float wf[4][4], bf4[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            bf4[c] = bias[4 * f + c];
#pragma unroll
            for (int q = 0; q < 4; ++q) wf[c][q] = __bfloat162float(W[(4 * f + c) * 4 + q]);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) w[c] = make_float4(wf[c][0], wf[c][1], wf[c][2], wf[c][3]);
        b = make_float4(bf4[0], bf4[1], bf4[2], bf4[3]);
    }
    static __device__ __forceinline__ float one(const float4& w, float b, const float4& f) {
        return relu(fmaf(w.w, f.w, fmaf(w.z, f.z, fmaf(w.y, f.y, fmaf(w.x, f.x, b)))));
    }
    __device__ __forceinline__ float4 operator()(const float4& f) const {
        return make_float4(one(w[0], b.x, f), one(w[1], b.y, f), one(w[2], b.z, f), one(w[3], b.w, f));
    }
};

struct Node64 {
    const float* h;                           // nodes x 64, or with First the features (nodes x 4)
    const __nv_bfloat16* Win; const float* bin;   // First: the input layer
    const __nv_bfloat16* U;                   // 64 x 64
    const float* a; const __nv_bfloat16* M;   // Two: the second input (nodes x 64) and its weights
    const float* P;                           // rows added along the edges (null: none)
    const int32_t *ptr, *idx; const float* val;   // edges of a node; rows of instance s at P + s * rows * 64
    int n, rows;                              // nodes (at least 1: the kernel divides by it) and rows of an instance
    const float* bias;                        // null: neither bias nor ReLU
    float* out;                               // null: not stored
    int64_t nodes;
    const __nv_bfloat16* wx; const float* bx; float* x0;   // Heads: out . wx + bx
    float* pool;                              // Heads: column sums, [tile][instance of the tile][64]
    int32_t* err;
};

constexpr int node64_smem(bool two) { return (two ? 2 : 1) * bf::kW + 3 * bf::kPart + 1024; }   // + alignment
// 512 threads, two blocks an SM: 16 threads a row of 256 contiguous bytes, four
// rows a thread (64 registers: 160 bytes of spills with First, 32 without).  The node's edges are a chain of three dependent loads; with
// 256 threads (eight rows each, half the warps to overlap) a layer of 1.28M
// nodes took 230 us.
constexpr int kN64T = 512;

template <bool First, bool Heads, bool Two>
__global__ void __launch_bounds__(kN64T, 2) k_node64(const Node64 a) {
    extern __shared__ __align__(16) unsigned char n64_smem[];
    unsigned char* base = n64_smem + ((1024 - (tc::smem_u32(n64_smem) & 1023)) & 1023);
    unsigned char* Ws = base;
    unsigned char* As = base + (Two ? 2 : 1) * bf::kW;
    constexpr uint32_t kTmem = Two ? 128 : 64;                  // columns: an accumulator per input
    __shared__ uint64_t bar;
    __shared__ uint32_t tmem_slot;
    __shared__ float4 cs[2][kN64T / 32][16];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    bf::put_weights<false>(Ws, a.U);
    if (Two) bf::put_weights<false>(Ws + bf::kW, a.M);
    if (threadIdx.x == 0) {
        tc::mbar_init(tc::smem_u32(&bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(tc::smem_u32(&tmem_slot)), "r"(kTmem) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tmem_slot;
    const int col0 = 16 * (warp >> 2);                          // the warp's accumulator columns
    const uint32_t tq = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)col0;
    const int f = threadIdx.x & 15, r0 = threadIdx.x >> 4;      // the thread's piece of rows r0 + 32 i
    const int nodes = (int)a.nodes;
    InW in;
    if (First) in.load(a.Win, a.bin, f);
    const int tiles = (nodes + 127) / 128;
    uint32_t parity = 0u;
    bool ok = true;
    float4 x[4];
    int e[4], end[4];
    int next_inst = 0;                                          // first instance of the fetched tile
    auto fetch = [&](int tile) {
        const int s0 = next_inst = (int)((unsigned)tile * 128u / (unsigned)a.n);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int v = tile * 128 + r0 + 32 * i;
            const bool live = v < nodes;
            x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live)
                x[i] = First ? __ldg(reinterpret_cast<const float4*>(a.h) + v)
                             : __ldg(reinterpret_cast<const float4*>(a.h) + (int64_t)v * 16 + f);
            if (a.P) {
                int r = v - s0 * a.n;
                while (r >= a.n) r -= a.n;
                e[i] = live ? __ldg(a.ptr + r) : 0;
                end[i] = live ? __ldg(a.ptr + r + 1) : 0;
            }
        }
    };
    if (blockIdx.x < tiles) fetch(blockIdx.x);
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
#pragma unroll
        for (int i = 0; i < 4; ++i) bf::put<true>(As, r0 + 32 * i, f, First ? in(x[i]) : x[i]);
        bool second = true;                                    // Two: thread 0 issues the second product
        const auto multiply = [&](int half) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc::fence_before();
            __syncthreads();
            tc::fence_after();
            if (threadIdx.x == 0 && second) {
                const uint32_t as = tc::smem_u32(As), ws = tc::smem_u32(Ws) + half * bf::kW;
#pragma unroll
                for (int q = 2; q >= 0; --q)                   // the small parts first
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        bf::mma<bf::idesc(128, 64, false, false)>(tmem + 64 * half, tc::desc_sw128(as + q * bf::kPart + 32 * kk),
                                                                 tc::desc_sw128(ws + 32 * kk),
                                                                 (q == 2 && kk == 0) ? 0u : 1u);
                tc::mma_commit(tc::smem_u32(&bar));
            }
        };
        multiply(0);
        if constexpr (Two) {
            // the second input, into accumulators of its own: added to the first's, every one of its
            // products would be cut to the whole sum's last place (the tensor core does not round
            // to nearest: outputs were 1.1e-6 off FP64 over 45 random graphs, now 2.2e-7)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int v = tile * 128 + r0 + 32 * i;
                x[i] = v < nodes ? __ldg(reinterpret_cast<const float4*>(a.a) + (int64_t)v * 16 + f)
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            if (!tc::mbar_wait(tc::smem_u32(&bar), parity)) ok = false;   // the operands are read
            second = ok;
            parity ^= 1u;
#pragma unroll
            for (int i = 0; i < 4; ++i) bf::put<true>(As, r0 + 32 * i, f, x[i]);
            multiply(1);
        }
        // the edges' rows, while the MMAs run
        float4 y[4];
        const int v0 = tile * 128 + r0;
        const int s0 = next_inst;                                 // the tile's first instance
#pragma unroll
        for (int i = 0; i < 4; ++i) y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (a.P) {
            int most = 0;
            const float4* src[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                int at = s0 * a.rows;                             // the instance's first row
                for (int r = v0 + 32 * i - s0 * a.n; r >= a.n; r -= a.n) at += a.rows;
                most = max(most, end[i] - e[i]);
                src[i] = reinterpret_cast<const float4*>(a.P) + (int64_t)at * 16 + f;
            }
            for (int k = 0; k < most; ++k) {
                float w[4];
                float4 p[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const bool on = e[i] + k < end[i];
                    w[i] = on ? __ldg(a.val + e[i] + k) : 0.f;
                    p[i] = on ? __ldg(src[i] + (int64_t)__ldg(a.idx + e[i] + k) * 16) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    y[i].x = fmaf(w[i], p[i].x, y[i].x);
                    y[i].y = fmaf(w[i], p[i].y, y[i].y);
                    y[i].z = fmaf(w[i], p[i].z, y[i].z);
                    y[i].w = fmaf(w[i], p[i].w, y[i].w);
                }
            }
        }
        if (tile + (int)gridDim.x < tiles) fetch(tile + gridDim.x);
        if (!tc::mbar_wait(tc::smem_u32(&bar), parity)) ok = false;
        parity ^= 1u;
        tc::fence_after();
        {
            // the accumulators (a lane per node) through the operands' shared memory to
            // the staging layout: 16-byte piece c of row r at piece c ^ (r & 15)
            uint32_t d[16];
            tc::tmem_ld16(tq, d);
            if constexpr (Two) {
                uint32_t m[16];
                tc::tmem_ld16(tq + 64, m);
#pragma unroll
                for (int j = 0; j < 16; ++j) d[j] = __float_as_uint(__uint_as_float(d[j]) + __uint_as_float(m[j]));
            }
            const int row = 32 * (warp & 3) + lane;
            float4* D = reinterpret_cast<float4*>(As) + row * 16;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                D[(col0 / 4 + j) ^ (row & 15)] = make_float4(__uint_as_float(d[4 * j]), __uint_as_float(d[4 * j + 1]),
                                                             __uint_as_float(d[4 * j + 2]), __uint_as_float(d[4 * j + 3]));
        }
        __syncthreads();
        float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
        if (a.bias) bias = make_float4(a.bias[4 * f], a.bias[4 * f + 1], a.bias[4 * f + 2], a.bias[4 * f + 3]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = r0 + 32 * i;
            const float4 d = reinterpret_cast<const float4*>(As)[row * 16 + (f ^ (row & 15))];
            float4 t = make_float4(d.x + y[i].x + bias.x, d.y + y[i].y + bias.y, d.z + y[i].z + bias.z,
                                   d.w + y[i].w + bias.w);
            if (a.bias) t = make_float4(relu(t.x), relu(t.y), relu(t.z), relu(t.w));
            y[i] = t;
            if (a.out && v0 + 32 * i < nodes && ok) reinterpret_cast<float4*>(a.out)[(int64_t)(v0 + 32 * i) * 16 + f] = t;
        }
        if constexpr (Heads) {
            float wx[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) wx[c] = __bfloat162float(a.wx[4 * f + c]);
            const float bx = a.bx[0];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float t = y[i].x * wx[0] + y[i].y * wx[1] + y[i].z * wx[2] + y[i].w * wx[3];
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (f == 0 && v0 + 32 * i < nodes) a.x0[v0 + 32 * i] = t + bx;
            }
            // column sums of the tile's one or two instances (n >= 128): rows, then the warp's two row groups
            const int split = (s0 + 1) * a.n;
            const int sets = min(tile * 128 + 128, nodes) > split ? 2 : 1;
#pragma unroll
            for (int set = 0; set < 2; ++set) {
                float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int v = v0 + 32 * i;
                    if (v < nodes && (v >= split) == (set == 1)) {
                        t.x += y[i].x;
                        t.y += y[i].y;
                        t.z += y[i].z;
                        t.w += y[i].w;
                    }
                }
                t.x += __shfl_xor_sync(0xffffffffu, t.x, 16);
                t.y += __shfl_xor_sync(0xffffffffu, t.y, 16);
                t.z += __shfl_xor_sync(0xffffffffu, t.z, 16);
                t.w += __shfl_xor_sync(0xffffffffu, t.w, 16);
                if (lane < 16) cs[set][warp][f] = t;
            }
            __syncthreads();
            if (threadIdx.x < 128) {
                const int set = threadIdx.x >> 6, c = threadIdx.x & 63;
                if (set < sets) {
                    float t = 0.f;
#pragma unroll
                    for (int w = 0; w < kN64T / 32; ++w) t += reinterpret_cast<const float*>(&cs[set][w][0])[c];
                    a.pool[((int64_t)tile * 2 + set) * 64 + c] = t;
                }
            }
        }
        tc::fence_before();
        ok = __syncthreads_and(ok) != 0;                       // shared and tensor memory free for the next tile
        tc::fence_after();
        if (!ok) {
            if (threadIdx.x == 0) tc::last_wait(tc::smem_u32(&bar), second ? parity ^ 1u : parity);
            break;
        }
    }
    if (!ok && threadIdx.x == 0) atomicExch(a.err, 1);
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmem) : "memory");
}

// ---- backward of a 64 x 64 node map on the tensor cores -------------------------------
// z = dout where the map's output is positive; dh = z W, and this block's share of
// dW = sum_v z_v h_v^T and db = sum_v z_v.  dout is read, or formed from the heads'
// gradients; rows of the constraint side's gradient are added along the edges.
// (With M on the constraint side, da and the M gradient need only sum_j a_ij z_j:
// z is stored for that aggregation, half of what da and its scatter moved.)
// On CUDA cores, one shared-memory word per FMA, this took 1453 us for 640k nodes
// of K = 128; now 200-260 us (the stream, five arrays of 164 MB, takes 120 us at
// the measured HBM rate; each tile's chain of loads, MMAs and read-backs with two
// blocks an SM is what is left; 64 registers, 216-228 bytes of spills).
//
// FP32 as three BF16 parts.  Both products read the same shared-memory image of a
// 128-node tile, rows of 128 bytes with the 128-byte swizzle: as the K-major A of
// dh (M = nodes, K = 64 features, 16 per step), and as MN-major operands of dW
// (K = nodes, 16 per step): A = [z1; z2] (M = 128: two parts one above the other), B =
// [h1 | h2 | h3] (N = 192), then A = [z2; z3] with B = h1, h2 and h3 in one set of
// accumulators (only z3's rows are taken), which have dh's place once that is read:
// all nine products, so nothing of z h is left out.  The tensor core adds FP32
// accumulators without rounding to nearest, so dW is moved to registers and added
// there after every tile.
namespace bk {
constexpr int kThreads = 512;
constexpr int kSmem = bf::kW + 6 * bf::kPart + 1024;
constexpr uint32_t kTmem = 256;               // columns: dW parts 0..191, dh then z3 h 192..255
constexpr int kOut = 64 * 64 + 64;            // a block's partial: dW, db
constexpr int kHeadOut = 65;                  // dw, db of a head
// MN-major operand, 128-byte swizzle: 64-element blocks `block` bytes apart, 8-row groups 1024
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr, uint32_t block) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(block >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
}  // namespace bk

struct Back64 {
    const float* dout;                        // nodes x 64 (null: from the head)
    const float* dhead; const __nv_bfloat16* whead;       // head: dhead[v] whead + dlw[instance] wpool / n
    const float* dlw; const __nv_bfloat16* wpool;
    const float* Q; const int32_t *ptr, *idx; const float* val; int rows;   // rows added along the edges (null: none)
    const float* out;                         // the map's output (null: no mask)
    const float* h;                           // the map's input, or with First the features (nodes x 4)
    const __nv_bfloat16* Win; const float* bin;
    const __nv_bfloat16* W;                   // 64 x 64
    float* z;                                 // null: not stored
    float* dh; int accumulate;                // dh += instead of =
    float* part;                              // kOut per block
    float* hpart;                             // kHeadOut per block (head only)
    int n;                                    // nodes of an instance
    int64_t nodes;
    int32_t* err;
};

template <bool First>
__global__ void __launch_bounds__(bk::kThreads, 2) k_back64(const Back64 a) {
    extern __shared__ __align__(16) unsigned char bk_smem[];
    unsigned char* base = bk_smem + ((1024 - (tc::smem_u32(bk_smem) & 1023)) & 1023);
    unsigned char* Ws = base;
    unsigned char* Zs = base + bf::kW;
    unsigned char* Hs = Zs + 3 * bf::kPart;
    __shared__ uint64_t bars[3];
    __shared__ uint32_t tmem_slot;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    bf::put_weights<true>(Ws, a.W);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < 3; ++q) tc::mbar_init(tc::smem_u32(&bars[q]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(tc::smem_u32(&tmem_slot)), "r"(bk::kTmem) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tmem_slot;
    const int c0 = 16 * (warp >> 2);                            // the warp's columns of each 64
    const uint32_t tq = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c0;
    const int trow = 32 * (warp & 3) + lane;
    const int f = threadIdx.x & 15, r0 = threadIdx.x >> 4;
    const int nodes = (int)a.nodes, tiles = (nodes + 127) / 128;
    float acc[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[j] = 0.f;
    float4 zsum = make_float4(0.f, 0.f, 0.f, 0.f), hw = zsum;
    float hb = 0.f;
    uint32_t parity = 0u;
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int v0 = tile * 128 + r0;
        // z
        float4 z[4];
        if (a.dout) {           // plain loads: dh may take dout's place
#pragma unroll
            for (int i = 0; i < 4; ++i)
                z[i] = v0 + 32 * i < nodes ? reinterpret_cast<const float4*>(a.dout)[(int64_t)(v0 + 32 * i) * 16 + f]
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (a.Q || !a.dout) {
            const int s0 = (int)((unsigned)tile * 128u / (unsigned)a.n);
            if (a.Q) {
                int e[4], end[4], most = 0;
                const float4* src[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const bool live = v0 + 32 * i < nodes;
                    int at = s0 * a.rows, r = v0 + 32 * i - s0 * a.n;
                    while (r >= a.n) { r -= a.n; at += a.rows; }
                    e[i] = live ? __ldg(a.ptr + r) : 0;
                    end[i] = live ? __ldg(a.ptr + r + 1) : 0;
                    most = max(most, end[i] - e[i]);
                    src[i] = reinterpret_cast<const float4*>(a.Q) + (int64_t)at * 16 + f;
                }
                for (int k = 0; k < most; ++k) {
                    float w[4];
                    float4 p[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const bool on = e[i] + k < end[i];
                        w[i] = on ? __ldg(a.val + e[i] + k) : 0.f;
                        p[i] = on ? __ldg(src[i] + (int64_t)__ldg(a.idx + e[i] + k) * 16) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        z[i].x = fmaf(w[i], p[i].x, z[i].x);
                        z[i].y = fmaf(w[i], p[i].y, z[i].y);
                        z[i].z = fmaf(w[i], p[i].z, z[i].z);
                        z[i].w = fmaf(w[i], p[i].w, z[i].w);
                    }
                }
            } else {
                const float inv = 1.f / float(a.n);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const bool live = v0 + 32 * i < nodes;
                    int s = s0;
                    for (int r = v0 + 32 * i - s0 * a.n; r >= a.n; r -= a.n) ++s;
                    const float d = live ? __ldg(a.dhead + v0 + 32 * i) : 0.f, g = live ? __ldg(a.dlw + s) * inv : 0.f;
                    const __nv_bfloat16 *w = a.whead + 4 * f, *q = a.wpool + 4 * f;
                    z[i] = make_float4(fmaf(d, __bfloat162float(w[0]), g * __bfloat162float(q[0])),
                                       fmaf(d, __bfloat162float(w[1]), g * __bfloat162float(q[1])),
                                       fmaf(d, __bfloat162float(w[2]), g * __bfloat162float(q[2])),
                                       fmaf(d, __bfloat162float(w[3]), g * __bfloat162float(q[3])));
                }
            }
        }
        if (a.out) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int v = v0 + 32 * i;
                float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
                if (v < nodes) o = __ldg(reinterpret_cast<const float4*>(a.out) + (int64_t)v * 16 + f);
                if (a.hpart && v < nodes) {
                    const float d = __ldg(a.dhead + v);
                    hw.x = fmaf(d, o.x, hw.x);
                    hw.y = fmaf(d, o.y, hw.y);
                    hw.z = fmaf(d, o.z, hw.z);
                    hw.w = fmaf(d, o.w, hw.w);
                    hb += d;
                }
                z[i] = make_float4(o.x > 0.f ? z[i].x : 0.f, o.y > 0.f ? z[i].y : 0.f, o.z > 0.f ? z[i].z : 0.f,
                                   o.w > 0.f ? z[i].w : 0.f);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int v = v0 + 32 * i;
            if (a.z && v < nodes) reinterpret_cast<float4*>(a.z)[(int64_t)v * 16 + f] = z[i];
            zsum.x += z[i].x;
            zsum.y += z[i].y;
            zsum.z += z[i].z;
            zsum.w += z[i].w;
            bf::put<false>(Zs, r0 + 32 * i, f, z[i]);
        }
        // h
        if constexpr (First) {
            InW in;
            in.load(a.Win, a.bin, f);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int v = v0 + 32 * i;
                bf::put<false>(Hs, r0 + 32 * i, f, v < nodes ? in(__ldg(reinterpret_cast<const float4*>(a.h) + v))
                                                     : make_float4(0.f, 0.f, 0.f, 0.f));
            }
        } else {
            float4 x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                x[i] = v0 + 32 * i < nodes ? __ldg(reinterpret_cast<const float4*>(a.h) + (int64_t)(v0 + 32 * i) * 16 + f)
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 4; ++i) bf::put<false>(Hs, r0 + 32 * i, f, x[i]);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc::fence_before();
        __syncthreads();
        tc::fence_after();
        const uint32_t zs = tc::smem_u32(Zs), hs = tc::smem_u32(Hs), ws = tc::smem_u32(Ws);
        if (threadIdx.x == 0) {
#pragma unroll
            for (int q = 2; q >= 0; --q)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    bf::mma<bf::idesc(128, 64, false, false)>(tmem + 192, tc::desc_sw128(zs + q * bf::kPart + 32 * kk),
                                                             tc::desc_sw128(ws + 32 * kk), (q == 2 && kk == 0) ? 0u : 1u);
            tc::mma_commit(tc::smem_u32(&bars[0]));
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
                bf::mma<bf::idesc(128, 192, true, true)>(tmem, bk::desc_mn(zs + 2048 * kk, bf::kPart),
                                                        bk::desc_mn(hs + 2048 * kk, bf::kPart), kk ? 1u : 0u);
            tc::mma_commit(tc::smem_u32(&bars[1]));
        }
        if (!tc::mbar_wait(tc::smem_u32(&bars[0]), parity)) ok = false;
        tc::fence_after();
        uint32_t dh[16];
        tc::tmem_ld16(tq + 192, dh);
        tc::fence_before();
        ok = __syncthreads_and(ok) != 0;                        // dh read: its columns take z3 h
        tc::fence_after();
        if (threadIdx.x == 0 && ok) {
#pragma unroll
            for (int p = 2; p >= 0; --p)                       // the small parts first
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                    bf::mma<bf::idesc(128, 64, true, true)>(
                        tmem + 192, bk::desc_mn(zs + bf::kPart + 2048 * kk, bf::kPart),
                        bk::desc_mn(hs + p * bf::kPart + 2048 * kk, bf::kPart), (p == 2 && kk == 0) ? 0u : 1u);
            tc::mma_commit(tc::smem_u32(&bars[2]));
        }
        if (!ok) {
            if (threadIdx.x == 0)
                for (int q = 0; q < 2; ++q) tc::last_wait(tc::smem_u32(&bars[q]), parity);
            break;
        }
        if (!tc::mbar_wait(tc::smem_u32(&bars[1]), parity)) ok = false;
        tc::fence_after();
        uint32_t q[16];
#pragma unroll
        for (int p = 2; p >= 0; --p) {                          // z1 h3 + z2 h3 (rows apart), ... h2, ... h1
            tc::tmem_ld16(tq + 64 * p, q);
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[j] += __uint_as_float(q[j]);
        }
        if (!tc::mbar_wait(tc::smem_u32(&bars[2]), parity)) ok = false;
        parity ^= 1u;
        tc::fence_after();
        tc::tmem_ld16(tq + 192, q);
        if (trow >= 64)
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[j] += __uint_as_float(q[j]);
        // dh through shared memory to the staging layout (the operands are done with)
        float4* D = reinterpret_cast<float4*>(Zs) + trow * 16;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            D[(c0 / 4 + j) ^ (trow & 15)] = make_float4(__uint_as_float(dh[4 * j]), __uint_as_float(dh[4 * j + 1]),
                                                        __uint_as_float(dh[4 * j + 2]), __uint_as_float(dh[4 * j + 3]));
        tc::fence_before();
        ok = __syncthreads_and(ok) != 0;
        tc::fence_after();
        if (!ok && threadIdx.x == 0)
            for (int q = 1; q < 3; ++q) tc::last_wait(tc::smem_u32(&bars[q]), parity ^ 1u);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = r0 + 32 * i, v = v0 + 32 * i;
            float4 d = reinterpret_cast<const float4*>(Zs)[row * 16 + (f ^ (row & 15))];
            if (v >= nodes || !ok) continue;
            float4* o = reinterpret_cast<float4*>(a.dh) + (int64_t)v * 16 + f;
            if (a.accumulate) {
                const float4 p = *o;
                d = make_float4(d.x + p.x, d.y + p.y, d.z + p.z, d.w + p.w);
            }
            *o = d;
        }
        __syncthreads();                                        // Zs read before the next tile's staging
    }
    if (!ok && threadIdx.x == 0) atomicExch(a.err, 1);
    // the block's partials: rows r and r + 64 of dW, then the sums over the row groups, in order
    __syncthreads();
    float* S = reinterpret_cast<float*>(Zs);
    float* P = a.part + (int64_t)blockIdx.x * bk::kOut;
    if (trow >= 64)
#pragma unroll
        for (int j = 0; j < 16; ++j) S[(trow - 64) * 65 + c0 + j] = acc[j];
    __syncthreads();
    if (trow < 64)
#pragma unroll
        for (int j = 0; j < 16; ++j) P[trow * 64 + c0 + j] = acc[j] + S[trow * 65 + c0 + j];
    __syncthreads();
    float* R = S;                                               // [32 row groups][64]
    reinterpret_cast<float4*>(R)[r0 * 16 + f] = zsum;
    __syncthreads();
    if (threadIdx.x < 64) {
        float t = 0.f;
        for (int g = 0; g < 32; ++g) t += R[g * 64 + threadIdx.x];
        P[4096 + threadIdx.x] = t;
    }
    if (a.hpart) {
        __syncthreads();
        reinterpret_cast<float4*>(R)[r0 * 16 + f] = hw;
        if (f == 0) R[2048 + r0] = hb;
        __syncthreads();
        float* Hp = a.hpart + (int64_t)blockIdx.x * bk::kHeadOut;
        if (threadIdx.x < 64) {
            float t = 0.f;
            for (int g = 0; g < 32; ++g) t += R[g * 64 + threadIdx.x];
            Hp[threadIdx.x] = t;
        } else if (threadIdx.x == 64) {
            float t = 0.f;
            for (int g = 0; g < 32; ++g) t += R[2048 + g];
            Hp[64] = t;
        }
    }
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(bk::kTmem) : "memory");
}

// Input layer backward for four features (H = 64): z = (dout + rows along the edges)
// where the recomputed layer is positive; partials of dW (64 x 4) and db.
constexpr int kInOut = 64 * 4 + 64;
__global__ void __launch_bounds__(bk::kThreads, 2) k_in_back64(const Back64 a) {
    const int f = threadIdx.x & 15, r0 = threadIdx.x >> 4;
    const int nodes = (int)a.nodes;
    InW in;
    in.load(a.Win, a.bin, f);
    float g[4][4], gb[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        gb[c] = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) g[c][q] = 0.f;
    }
    for (int v = blockIdx.x * 32 + r0; v < nodes; v += gridDim.x * 32) {
        float4 z = __ldg(reinterpret_cast<const float4*>(a.dout) + (int64_t)v * 16 + f);
        const float4 x = __ldg(reinterpret_cast<const float4*>(a.h) + v);
        if (a.Q) {
            const int s = (int)((unsigned)v / (unsigned)a.n), r = v - s * a.n;
            const float4* src = reinterpret_cast<const float4*>(a.Q) + (int64_t)s * a.rows * 16 + f;
            for (int e = __ldg(a.ptr + r), end = __ldg(a.ptr + r + 1); e < end; ++e) {
                const float w = __ldg(a.val + e);
                const float4 p = __ldg(src + (int64_t)__ldg(a.idx + e) * 16);
                z = make_float4(fmaf(w, p.x, z.x), fmaf(w, p.y, z.y), fmaf(w, p.z, z.z), fmaf(w, p.w, z.w));
            }
        }
        const float4 o = in(x);
        const float zz[4] = {o.x > 0.f ? z.x : 0.f, o.y > 0.f ? z.y : 0.f, o.z > 0.f ? z.z : 0.f, o.w > 0.f ? z.w : 0.f};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            g[c][0] = fmaf(zz[c], x.x, g[c][0]);
            g[c][1] = fmaf(zz[c], x.y, g[c][1]);
            g[c][2] = fmaf(zz[c], x.z, g[c][2]);
            g[c][3] = fmaf(zz[c], x.w, g[c][3]);
            gb[c] += zz[c];
        }
    }
    // sums over the 32 row groups in order: [group][output][4 features, bias]
    __shared__ float R[32][64 * 5 / 2];                          // two halves of the outputs, one after the other
    float* P = a.part + (int64_t)blockIdx.x * kInOut;
    for (int half = 0; half < 2; ++half) {
        __syncthreads();
        if (f / 8 == half)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float* d = &R[r0][((f & 7) * 4 + c) * 5];
#pragma unroll
                for (int q = 0; q < 4; ++q) d[q] = g[c][q];
                d[4] = gb[c];
            }
        __syncthreads();
        for (int t = threadIdx.x; t < 160; t += bk::kThreads) {
            float sum = 0.f;
            for (int q = 0; q < 32; ++q) sum += R[q][t];
            const int o = 32 * half + t / 5, k = t % 5;
            if (k < 4) P[o * 4 + k] = sum;
            else P[256 + o] = sum;
        }
    }
}

// grad[p] += the sum over a job's blocks, in order, for every job (one launch for
// all weight gradients; eight loads in flight where one per block was 62 us each).
struct SumJob {
    const float* part;
    float* grad;
    int32_t blocks, stride, width;
};
constexpr int kMaxJobs = 80;                  // 8 layers x 7 + inputs and heads
struct SumJobs {
    SumJob job[kMaxJobs];
};
__global__ void __launch_bounds__(kT) k_sum_jobs(const __grid_constant__ SumJobs J) {
    const SumJob j = J.job[blockIdx.y];
    for (int p = blockIdx.x * kT + threadIdx.x; p < j.width; p += gridDim.x * kT) {
        float s = 0.f;
        for (int b = 0; b < j.blocks; b += 8) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = b + u < j.blocks ? __ldg(j.part + (int64_t)(b + u) * j.stride + p) : 0.f;
#pragma unroll
            for (int u = 0; u < 8; ++u) s += v[u];
        }
        j.grad[p] += s;
    }
}

// hi + lo += p with the sum's rounding kept in lo (Knuth's two-sum): long sums are
// made of short ones (eight products) added this way.
__device__ __forceinline__ void add2(float p, float& hi, float& lo) {
    const float t = __fadd_rn(hi, p), b = __fsub_rn(t, hi);
    lo += __fadd_rn(__fsub_rn(hi, __fsub_rn(t, b)), __fsub_rn(p, b));
    hi = t;
}
// the sum of the two: lo is NaN (inf - inf) once hi has left the finite numbers
__device__ __forceinline__ float sum2(float hi, float lo) { return isfinite(hi) ? hi + lo : hi; }

// Aggregation onto the constraints (H = 64): each row's edges in eight stretches (lane
// l: features 2 l, 2 l + 1; eight rows in flight), the stretches' sums added in order.
// Warps = 8: a block per row, a warp per stretch.  A warp per row left 4 800 warps with
// up to 400 dependent steps each on the constraint rows of the 200 x 400 family
// (62 us for 164 MB; now 46, compensated).  Warps = 1: a warp per row takes the stretches in turn,
// the same bits.  Sums of hundreds of terms, compensated.  First: the source is the
// input layer of the nodes' four features, recomputed per edge (16 bytes instead of
// 256).
template <bool First, int Warps>
__global__ void __launch_bounds__(kT) k_agg_rows(const int32_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                                                 const float* __restrict__ val, const float* __restrict__ in,
                                                 const __nv_bfloat16* __restrict__ Win, const float* __restrict__ bin,
                                                 float* __restrict__ out, int n_dst, int n_src, int rows,
                                                 int accumulate) {
    constexpr int kStretches = 8;
    static_assert(Warps == 1 || Warps == kStretches, "a warp per row or per stretch");
    __shared__ float2 part[Warps == 1 ? 1 : kStretches][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = Warps == 1 ? blockIdx.x * (kT / 32) + warp : (int)blockIdx.x;
    if (row >= rows) return;
    const int s = row / n_dst, r = row % n_dst;
    const int b = ptr[r], len = ptr[r + 1] - b;
    float4 w0, w1;
    float b0 = 0.f, b1 = 0.f;
    if (First) {
        const __nv_bfloat16* w = Win + 8 * lane;
        w0 = make_float4(__bfloat162float(w[0]), __bfloat162float(w[1]), __bfloat162float(w[2]), __bfloat162float(w[3]));
        w1 = make_float4(__bfloat162float(w[4]), __bfloat162float(w[5]), __bfloat162float(w[6]), __bfloat162float(w[7]));
        b0 = bin[2 * lane];
        b1 = bin[2 * lane + 1];
    }
    const float* src = in + (int64_t)s * n_src * (First ? 4 : 64);
    const auto stretch = [&](int q) {
        const int e0 = b + int((int64_t)len * q / kStretches), e1 = b + int((int64_t)len * (q + 1) / kStretches);
        float2 acc = make_float2(0.f, 0.f), low = acc;
        float an[8];                           // the next group's edges load with this group's rows
        int jn[8];
        auto edges = [&](int e) {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const bool ok = e + u < e1;
                an[u] = ok ? __ldg(val + e + u) : 0.f;
                jn[u] = ok ? __ldg(idx + e + u) : 0;
            }
        };
        edges(e0);
        for (int e = e0; e < e1; e += 8) {
            float a[8];
            float4 ff[8];
            float2 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                a[u] = an[u];
                if (First) ff[u] = __ldg(reinterpret_cast<const float4*>(src) + jn[u]);
                else v[u] = __ldg(reinterpret_cast<const float2*>(src + (int64_t)jn[u] * 64) + lane);
            }
            if (e + 8 < e1) edges(e + 8);
            float2 t = make_float2(0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (First) v[u] = make_float2(InW::one(w0, b0, ff[u]), InW::one(w1, b1, ff[u]));
                if (e + u >= e1) continue;         // no edge: node 0 may be infinite
                t.x = fmaf(a[u], v[u].x, t.x);
                t.y = fmaf(a[u], v[u].y, t.y);
            }
            add2(t.x, acc.x, low.x);
            add2(t.y, acc.y, low.y);
        }
        return make_float2(sum2(acc.x, low.x), sum2(acc.y, low.y));
    };
    float2 t;
    if constexpr (Warps == 1) {
        t = stretch(0);
#pragma unroll 1
        for (int q = 1; q < kStretches; ++q) {
            const float2 p = stretch(q);
            t.x += p.x;
            t.y += p.y;
        }
    } else {
        part[warp][lane] = stretch(warp);
        __syncthreads();
        if (warp) return;
        t = part[0][lane];
#pragma unroll
        for (int w = 1; w < kStretches; ++w) {
            t.x += part[w][lane].x;
            t.y += part[w][lane].y;
        }
    }
    float2* o = reinterpret_cast<float2*>(out + (int64_t)row * 64) + lane;
    if (accumulate) {
        const float2 p = *o;
        t.x += p.x;
        t.y += p.y;
    }
    *o = t;
}

// The constraint nodes' update (H = 64): relu(U h + M a + b) in compensated FP32, 16
// nodes a block, a thread one output of four.  There are few constraint nodes
// and each stands for hundreds of variables: a ReLU that takes the other side of
// zero than exact arithmetic changes the gradient by parts in 10^5, so this sum and
// the aggregation's are made more exactly than the tensor cores' FP32 sums (the
// gradient's error against FP64 on the 200 x 400 family: 2.4e-6 before).
constexpr int kConNodes = 16;
__global__ void __launch_bounds__(kT) k_con_update(const float* __restrict__ h, const float* __restrict__ a,
                                                   const __nv_bfloat16* __restrict__ U,
                                                   const __nv_bfloat16* __restrict__ M,
                                                   const float* __restrict__ bias, float* __restrict__ out,
                                                   int64_t nodes) {
    __shared__ float Wt[128 * 65];             // [k][o], rows of 65: a warp stages a row of U or M and reads along o
    __shared__ float4 X[kConNodes][32];
    for (int t = threadIdx.x; t < 64 * 64; t += kT) {
        const int o = t >> 6, k = t & 63;
        Wt[k * 65 + o] = __bfloat162float(U[t]);
        Wt[(k + 64) * 65 + o] = __bfloat162float(M[t]);
    }
    const int64_t v0 = (int64_t)blockIdx.x * kConNodes;
    for (int t = threadIdx.x; t < kConNodes * 32; t += kT) {
        const int nd = t >> 5, q = t & 31;
        const int64_t v = v0 + nd;
        X[nd][q] = v >= nodes ? make_float4(0.f, 0.f, 0.f, 0.f)
                   : q < 16 ? reinterpret_cast<const float4*>(h)[v * 16 + q] : reinterpret_cast<const float4*>(a)[v * 16 + q - 16];
    }
    __syncthreads();
    const int o = threadIdx.x & 63, g = threadIdx.x >> 6;
    float hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        hi[i] = bias[o];
        lo[i] = 0.f;
    }
    for (int q = 0; q < 32; q += 2) {
        float w[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) w[c] = Wt[(4 * q + c) * 65 + o];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 x = X[g + 4 * i][q], y = X[g + 4 * i][q + 1];
            const float t = fmaf(w[3], x.w, fmaf(w[2], x.z, fmaf(w[1], x.y, w[0] * x.x)));
            const float u = fmaf(w[7], y.w, fmaf(w[6], y.z, fmaf(w[5], y.y, w[4] * y.x)));
            add2(t + u, hi[i], lo[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (v0 + g + 4 * i < nodes) out[(v0 + g + 4 * i) * 64 + o] = relu(sum2(hi[i], lo[i]));
}

// The pooled head from k_node64's column sums of the variables (per tile, in order) and k_colsum_part's of the constraints.
__global__ void __launch_bounds__(1024) k_pool_finish64(const float* __restrict__ pc, int nbc,
                                                        const float* __restrict__ pv, int m, int n, int64_t nodes,
                                                        const __nv_bfloat16* __restrict__ wo,
                                                        const float* __restrict__ bo, float* __restrict__ pool,
                                                        float* __restrict__ lw) {
    __shared__ float sub[16][64];
    __shared__ float red[128];
    const int s = blockIdx.x, f = threadIdx.x & 63, g = threadIdx.x >> 6;
    const int64_t t0 = (int64_t)s * n / 128, t1 = ((int64_t)(s + 1) * n - 1) / 128;
    float acc = 0.f;
#pragma unroll 4
    for (int64_t t = t0 + g; t <= t1; t += 16)                    // a tile that starts in the instance before: its second set
        acc += pv[(t * 2 + (t * 128 < (int64_t)s * n ? 1 : 0)) * 64 + f];
    sub[g][f] = acc;
    __syncthreads();
    if (threadIdx.x < 128) {
        float t = 0.f;
        if (threadIdx.x < 64) {
            for (int b = 0; b < nbc; ++b) t += pc[((int64_t)s * nbc + b) * 64 + f];
            t /= float(m);
        } else {
            for (int q = 0; q < 16; ++q) t += sub[q][f];
            t /= float(n);
        }
        pool[s * 128 + threadIdx.x] = t;
        red[threadIdx.x] = t * __bfloat162float(wo[threadIdx.x]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int q = 0; q < 128; ++q) t += red[q];
        lw[s] = t + bo[0];
    }
}

// ---- heads: out[v] = w . h[v] + b (warp per node) ----------------------------------
template <int H>
__global__ void __launch_bounds__(kT) k_head(const float* __restrict__ h, const __nv_bfloat16* __restrict__ w,
                                             const float* __restrict__ b, float* __restrict__ out, int64_t nodes) {
    const int lane = threadIdx.x & 31;
    float w0 = __bfloat162float(w[lane]), w1 = H == 64 ? __bfloat162float(w[lane + 32]) : 0.f;
    for (int64_t v = (blockIdx.x * (int64_t)kT + threadIdx.x) >> 5; v < nodes; v += ((int64_t)gridDim.x * kT) >> 5) {
        float s = h[v * H + lane] * w0;
        if (H == 64) s += h[v * H + lane + 32] * w1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) out[v] = s + b[0];
    }
}

// ---- per-instance column sums of h over nodes (pooling), block partials ------------
// part[(s * nb + blk) * H + f] over node chunks of instance s (grid.y = instance).
template <int H>
__global__ void __launch_bounds__(kT) k_colsum_part(const float* __restrict__ h, int n, float* __restrict__ part) {
    const int s = blockIdx.y, f = threadIdx.x % H, lanes = kT / H, sub = threadIdx.x / H;
    __shared__ float red[kT];
    float acc = 0.f;
    for (int64_t v = blockIdx.x * (int64_t)lanes + sub; v < n; v += (int64_t)gridDim.x * lanes)
        acc += h[((int64_t)s * n + v) * H + f];
    red[threadIdx.x] = acc;
    __syncthreads();
    if (sub == 0) {
        for (int q = 1; q < lanes; ++q) acc += red[q * H + f];
        part[((int64_t)s * gridDim.x + blockIdx.x) * H + f] = acc;
    }
}

// pool[s][0:H] = mean over constraints, pool[s][H:2H] = mean over variables;
// log_omega[s] = wo . pool + bo
template <int H>
__global__ void k_pool_finish(const float* __restrict__ pc, int nbc, const float* __restrict__ pv, int nbv, int m,
                              int n, const __nv_bfloat16* __restrict__ wo, const float* __restrict__ bo,
                              float* __restrict__ pool, float* __restrict__ lw) {
    const int s = blockIdx.x, f = threadIdx.x;
    __shared__ float red[2 * H];
    if (f < 2 * H) {
        float acc = 0.f;
        if (f < H) { for (int b = 0; b < nbc; ++b) acc += pc[((int64_t)s * nbc + b) * H + f]; acc /= float(m); }
        else { for (int b = 0; b < nbv; ++b) acc += pv[((int64_t)s * nbv + b) * H + f - H]; acc /= float(n); }
        pool[s * 2 * H + f] = acc;
        red[f] = acc * __bfloat162float(wo[f]);
    }
    __syncthreads();
    if (f == 0) {
        float t = 0.f;
        for (int q = 0; q < 2 * H; ++q) t += red[q];
        lw[s] = t + bo[0];
    }
}

// ---- loss and output gradients --------------------------------------------------------
// d = out - target; dout = coef * d; block partial of sum d^2 (per block, in order)
__global__ void __launch_bounds__(kT) k_sq_loss(const float* __restrict__ out, const float* __restrict__ tgt,
                                                int64_t count, float coef, float* __restrict__ dout,
                                                double* __restrict__ part) {
    __shared__ double red[kT];
    double acc = 0.0;
    for (int64_t t = blockIdx.x * (int64_t)kT + threadIdx.x; t < count; t += (int64_t)gridDim.x * kT) {
        const float d = out[t] - tgt[t];
        dout[t] = coef * d;
        acc += double(d) * double(d);
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = kT / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// ---- head backward: dh[v] = dout[v] w + dlw[s] wo_part / N; partials of dw, db -------
// part[blk][0:H] = sum dout h, part[blk][H] = sum dout (H+1 per block)
template <int H>
__global__ void __launch_bounds__(kT) k_head_back(const float* __restrict__ h, const float* __restrict__ dout,
                                                  const __nv_bfloat16* __restrict__ w, const float* __restrict__ dlw,
                                                  const __nv_bfloat16* __restrict__ wo_part, int n, int batch,
                                                  float* __restrict__ dh, float* __restrict__ part) {
    const int f = threadIdx.x % H, lanes = kT / H, sub = threadIdx.x / H;
    const float wf = __bfloat162float(w[f]), wof = __bfloat162float(wo_part[f]) / float(n);
    const int64_t nodes = (int64_t)n * batch;
    float gw = 0.f, gb = 0.f;
    for (int64_t v = blockIdx.x * (int64_t)lanes + sub; v < nodes; v += (int64_t)gridDim.x * lanes) {
        const float d = dout[v];
        dh[v * H + f] = d * wf + dlw[v / n] * wof;
        gw += d * h[v * H + f];
        if (f == 0) gb += d;
    }
    __shared__ float red[kT];
    __shared__ float redb[kT / 32 + 1];
    red[threadIdx.x] = gw;
    if (f == 0) redb[sub] = gb;
    __syncthreads();
    if (sub == 0) {
        for (int q = 1; q < lanes; ++q) gw += red[q * H + f];
        part[(int64_t)blockIdx.x * (H + 1) + f] = gw;
        if (f == 0) {
            for (int q = 1; q < lanes; ++q) gb += redb[q];
            part[(int64_t)blockIdx.x * (H + 1) + H] = gb;
        }
    }
}

// ---- dense node update backward, H = 32 ----------------------------------------------
// z = U h + M a + b, out = relu(z), dz = dout * (out > 0):
//   dh (=/+=) U^T dz, da = M^T dz, partials of dU = sum dz h^T, dM = sum dz a^T, db = sum dz.
// Thread t: node t / 8 and input features (t % 8) + 8 i for dh / da; weight-gradient
// entries o = t / 4, k = (t % 4) + 4 i (8 of dU and 8 of dM in half of the threads).
__global__ void __launch_bounds__(kT) k_update_back(const float* __restrict__ dout, const float* __restrict__ out,
                                                    const float* __restrict__ h, const float* __restrict__ a,
                                                    const __nv_bfloat16* __restrict__ U,
                                                    const __nv_bfloat16* __restrict__ M, float* __restrict__ dh,
                                                    int dh_accumulate, float* __restrict__ da,
                                                    float* __restrict__ part, int64_t nodes) {
    constexpr int H = 32, OP = H / 8, ZS = H + 1;
    constexpr int WK = H / 4;                                  // weight columns per thread
    extern __shared__ __align__(16) float sm[];
    float* Us = sm;                 // [o][k]
    float* Ms = Us + H * H;
    float* Z = Ms + H * H;          // dz tile [kTile][ZS]
    float* Hs = Z + kTile * ZS;     // h tile
    float* As = Hs + kTile * ZS;    // a tile
    for (int t = threadIdx.x; t < H * H; t += kT) {
        Us[t] = __bfloat162float(U[t]);
        Ms[t] = __bfloat162float(M[t]);
    }
    const int node = threadIdx.x >> 3, g = threadIdx.x & 7;
    const int o0 = threadIdx.x >> 2, wk0 = threadIdx.x & 3;    // weight-gradient ownership
    float gU[WK], gM[WK], gb = 0.f;
#pragma unroll
    for (int i = 0; i < WK; ++i) gU[i] = gM[i] = 0.f;
    const int64_t tiles = (nodes + kTile - 1) / kTile;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t base = tile * kTile;
        __syncthreads();
        for (int t = threadIdx.x; t < kTile * H; t += kT) {
            const int nd = t / H, k = t % H;
            const int64_t v = base + nd;
            const bool ok = v < nodes;
            Z[nd * ZS + k] = ok && out[v * H + k] > 0.f ? dout[v * H + k] : 0.f;
            Hs[nd * ZS + k] = ok ? h[v * H + k] : 0.f;
            As[nd * ZS + k] = ok ? a[v * H + k] : 0.f;
        }
        __syncthreads();
        // input gradients of this thread's node
        float gh[OP], ga[OP];
#pragma unroll
        for (int i = 0; i < OP; ++i) { gh[i] = 0.f; ga[i] = 0.f; }
        const float* z = Z + node * ZS;
        for (int o = 0; o < H; ++o) {
            const float zo = z[o];
#pragma unroll
            for (int i = 0; i < OP; ++i) {
                gh[i] += Us[o * H + g + 8 * i] * zo;
                ga[i] += Ms[o * H + g + 8 * i] * zo;
            }
        }
        const int64_t v = base + node;
        if (v < nodes) {
#pragma unroll
            for (int i = 0; i < OP; ++i) {
                const int64_t q = v * H + g + 8 * i;
                dh[q] = dh_accumulate ? dh[q] + gh[i] : gh[i];
                da[q] = ga[i];
            }
        }
        // weight gradients over the tile
        for (int nd = 0; nd < kTile && o0 < H; ++nd) {
            const float zo = Z[nd * ZS + o0];
            if (wk0 == 0) gb += zo;
#pragma unroll
            for (int i = 0; i < WK; ++i) {
                const int k = wk0 + 4 * i;
                gU[i] += zo * Hs[nd * ZS + k];
                gM[i] += zo * As[nd * ZS + k];
            }
        }
    }
    // block partial: [dU (H*H) | dM (H*H) | db (H)]
    float* P = part + (int64_t)blockIdx.x * (2 * H * H + H);
    if (o0 >= H) return;
#pragma unroll
    for (int i = 0; i < WK; ++i) {
        const int k = wk0 + 4 * i;
        P[o0 * H + k] = gU[i];
        P[H * H + o0 * H + k] = gM[i];
    }
    if (wk0 == 0) P[2 * H * H + o0] = gb;
}

// input layer backward: dz = dout * (h > 0); partials of dW (H x F) and db (H)
template <int H>
__global__ void __launch_bounds__(kT) k_input_back(const float* __restrict__ dout, const float* __restrict__ h,
                                                   const float* __restrict__ f, int F, int64_t nodes,
                                                   float* __restrict__ part) {
    const int o = threadIdx.x % H, lanes = kT / H, sub = threadIdx.x / H;
    float gw[kMaxF], gb = 0.f;
    for (int q = 0; q < kMaxF; ++q) gw[q] = 0.f;
    for (int64_t v = blockIdx.x * (int64_t)lanes + sub; v < nodes; v += (int64_t)gridDim.x * lanes) {
        const float z = h[v * H + o] > 0.f ? dout[v * H + o] : 0.f;
        gb += z;
        for (int q = 0; q < F; ++q) gw[q] += z * f[v * F + q];
    }
    __shared__ float red[kT * (kMaxF + 1)];
    for (int q = 0; q < F; ++q) red[q * kT + threadIdx.x] = gw[q];
    red[kMaxF * kT + threadIdx.x] = gb;
    __syncthreads();
    if (sub == 0) {
        float* P = part + (int64_t)blockIdx.x * (H * F + H);
        for (int q = 0; q < F; ++q) {
            float s = 0.f;
            for (int l = 0; l < lanes; ++l) s += red[q * kT + l * H + o];
            P[o * F + q] = s;
        }
        float s = 0.f;
        for (int l = 0; l < lanes; ++l) s += red[kMaxF * kT + l * H + o];
        P[H * F + o] = s;
    }
}

// grad[p] += scale * sum_b part[b][p] (blocks in order)
__global__ void k_sum_parts(const float* __restrict__ part, int nb, int width, float scale, float* __restrict__ grad) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < width; p += gridDim.x * blockDim.x) {
        float s = 0.f;
        for (int b = 0; b < nb; ++b) s += part[(int64_t)b * width + p];
        grad[p] += scale * s;
    }
}

// log-omega head gradients: dwo += sum_s dlw[s] pool[s], dbo += sum_s dlw[s]
template <int H>
__global__ void k_omega_back(const float* __restrict__ dlw, const float* __restrict__ pool, int batch,
                             float* __restrict__ gwo, float* __restrict__ gbo) {
    const int f = threadIdx.x;
    if (f < 2 * H) {
        float s = 0.f;
        for (int b = 0; b < batch; ++b) s += dlw[b] * pool[b * 2 * H + f];
        gwo[f] += s;
    }
    if (f == 0) {
        float s = 0.f;
        for (int b = 0; b < batch; ++b) s += dlw[b];
        gbo[0] += s;
    }
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m1,
                       float* __restrict__ m2, __nv_bfloat16* __restrict__ pb, int64_t count, float lr, float b1,
                       float b2, float eps, float c1, float c2) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count; t += (int64_t)gridDim.x * blockDim.x) {
        const float gt = g[t];
        const float a = b1 * m1[t] + (1.f - b1) * gt;
        const float b = b2 * m2[t] + (1.f - b2) * gt * gt;
        m1[t] = a;
        m2[t] = b;
        const float v = p[t] - lr * (a / c1) / (sqrtf(b / c2) + eps);
        p[t] = v;
        pb[t] = __float2bfloat16_rn(v);
    }
}

__global__ void k_to_bf16(const float* __restrict__ p, __nv_bfloat16* __restrict__ pb, int64_t count) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count; t += (int64_t)gridDim.x * blockDim.x)
        pb[t] = __float2bfloat16_rn(p[t]);
}

// ---- LP features (lp_features): constraint side, one warp per (instance, row) --------
// cmin = min of c over the row's columns (0 for an empty row); fc = [b, kind, cmin, 1]
__global__ void __launch_bounds__(kT) k_lp_con_features(const int32_t* __restrict__ ptr,
                                                         const int32_t* __restrict__ idx,
                                                         const int8_t* __restrict__ kind,
                                                         const float* __restrict__ c, const float* __restrict__ b,
                                                         int n, int m, int batch, float* __restrict__ fc,
                                                         float* __restrict__ cmin) {
    const int lane = threadIdx.x & 31;
    const int64_t rows = (int64_t)m * batch;
    for (int64_t w = (blockIdx.x * (int64_t)kT + threadIdx.x) >> 5; w < rows; w += ((int64_t)gridDim.x * kT) >> 5) {
        const int64_t s = w / m;
        const int r = int(w % m);
        const float* cs = c + s * (int64_t)n;
        float v = INFINITY;
        for (int k = ptr[r] + lane; k < ptr[r + 1]; k += 32) v = fminf(v, cs[idx[k]]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) {
            const float cm = ptr[r + 1] > ptr[r] ? v : 0.f;
            cmin[w] = cm;
            fc[w * 4 + 0] = b[w];
            fc[w * 4 + 1] = float(kind[r]);
            fc[w * 4 + 2] = cm;
            fc[w * 4 + 3] = 1.f;
        }
    }
}

// variable side, one thread per (instance, column): fv = [c, mean gap over '<=' rows,
// mean gap over '=' rows, 1] with gap = c - cmin(row)
__global__ void __launch_bounds__(kT) k_lp_var_features(const int32_t* __restrict__ ptr,
                                                        const int32_t* __restrict__ idx,
                                                        const int8_t* __restrict__ kind,
                                                        const float* __restrict__ c, const float* __restrict__ cmin,
                                                        int n, int m, int batch, float* __restrict__ fv) {
    const int64_t total = (int64_t)n * batch;
    for (int64_t t = blockIdx.x * (int64_t)kT + threadIdx.x; t < total; t += (int64_t)gridDim.x * kT) {
        const int64_t s = t / n;
        const int j = int(t % n);
        const float cj = c[t];
        float sle = 0.f, seq = 0.f;
        int nle = 0, neq = 0;
        for (int k = ptr[j]; k < ptr[j + 1]; ++k) {
            const int r = idx[k];
            const float d = cj - cmin[s * m + r];
            if (kind[r]) { sle += d; ++nle; } else { seq += d; ++neq; }
        }
        fv[t * 4 + 0] = cj;
        fv[t * 4 + 1] = sle / float(nle > 0 ? nle : 1);
        fv[t * 4 + 2] = seq / float(neq > 0 ? neq : 1);
        fv[t * 4 + 3] = 1.f;
    }
}

}  // namespace

// ===========================================================================
// Host object
// ===========================================================================
struct sps_gnn {
    sps_gnn_graph g{};
    sps_gnn_options opt{};
    int H = 64, L = 3, Fv = 1, Fc = 1, n = 0, m = 0, B = 1;
    // H = 64: the route of forward64; the input layer of the variables' four features is
    // recomputed where it is read (16 bytes a node instead of 256)
    bool few_rows = false, in4 = false;
    int lpf = 0;                 // lp_features: inputs are scaled c and b, expanded on the device
    float *craw = nullptr, *braw = nullptr, *cmin = nullptr;
    int8_t* kind = nullptr;
    int64_t nnz = 0, np = 0;
    cudaStream_t st = nullptr;
    std::vector<void*> dev;
    std::string err;
    // graph: CSR by constraint (a_c and a_v values), CSR by variable (a_v and a_c values)
    int32_t *cptr, *cidx, *vptr, *vidx;
    float *ac_c, *av_c, *av_v, *ac_v;
    // parameters
    float *P, *G, *M1, *M2;
    __nv_bfloat16* PB;
    int64_t step = 0;
    // offsets into the parameter vector
    int64_t oWv, obv, oWc, obc, oL0, per_layer, oWx, obx, oWy, oby, oWo, obo;
    // activations (max batch)
    float *fv, *fc, *xt, *yt, *lt;
    std::vector<float*> HV, HC, AV, AC;
    float *dHV, *dHC, *dHV2, *dHC2, *dA;
    float *x0, *y0, *lw, *pool, *dx0, *dy0, *dlw;
    int32_t* d_err = nullptr;    // set by a tensor-core kernel that gave up waiting (internal error)
    float *part;              // weight-gradient block partials
    double* lpart;            // loss partials
    float *MH = nullptr, *AG = nullptr;   // H = 64: M hc of the layer being computed; sum_j a_ij z_j
    float *pcp, *pvp;         // pooling partials
    int nb_dense = 0, nb_pool_c = 0, nb_pool_v = 0, nb_loss = 0;
    int64_t part_floats = 0;

    ~sps_gnn() {
        for (void* p : dev) cudaFree(p);
        if (st) cudaStreamDestroy(st);
    }
    template <class T>
    cudaError_t alloc(T** p, size_t count) {
        void* q = nullptr;
        const cudaError_t e = cudaMalloc(&q, std::max<size_t>(count, 1) * sizeof(T));
        if (e == cudaSuccess) dev.push_back(q);
        *p = static_cast<T*>(q);
        return e;
    }
    int fail(int code, const std::string& msg) {
        err = msg;
        return code;
    }
    int64_t layer_off(int l) const { return oL0 + per_layer * l; }
};

namespace {

thread_local std::string g_gnn_create_error;

#define GNN_CK(call)                                                                         \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess)                                                               \
            return g->fail(e_ == cudaErrorMemoryAllocation ? -3 : -2,                        \
                           std::string(#call) + ": " + cudaGetErrorString(e_));              \
    } while (0)

constexpr int kUpdateSmem = sizeof(float) * (2 * 32 * 32 + kUpdNodes * kUpdStride);
constexpr int kUpdateBackSmem = sizeof(float) * (2 * 32 * 32 + 3 * kTile * (32 + 1));

// Dynamic shared memory of the width's kernels; false if the device refuses.
bool set_smem_attrs(int H) {
    const auto size = [](auto k, int bytes) {
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
    };
    if (H == 32) return size(k_update, kUpdateSmem) && size(k_update_back, kUpdateBackSmem);
    for (auto k : {k_node64<false, false, false>, k_node64<false, true, false>, k_node64<true, false, false>,
                   k_node64<true, true, false>})
        if (!size(k, node64_smem(false))) return false;
    for (auto k : {k_node64<false, false, true>, k_node64<false, true, true>})
        if (!size(k, node64_smem(true))) return false;
    return size(k_back64<false>, bk::kSmem) && size(k_back64<true>, bk::kSmem);
}

int grid_for(int64_t work, int per_block) {
    const int64_t b = (work + per_block - 1) / per_block;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, 152 * 8));
}

// After the stream is synchronised: a tensor-core update that gave up waiting
// for its MMAs left its flag (the outputs of that forward are not valid).
int device_error(sps_gnn* g) {
    int32_t e = 0;
    if (!g->d_err) return 0;
    if (cudaMemcpyAsync(&e, g->d_err, sizeof(e), cudaMemcpyDeviceToHost, g->st) != cudaSuccess ||
        cudaStreamSynchronize(g->st) != cudaSuccess)
        return g->fail(-2, "reading the network's error flag failed");
    return e ? g->fail(-2, "internal error: a tensor-core kernel stopped waiting for its MMAs") : 0;
}

// The aggregation onto the constraints (H = 64) of the variable nodes `in`, or of
// the input layer of their features (first).  A block per row where rows of at least
// 64 edges are too few to fill the GPU with a warp each: 500 rows of 240 edges, one
// instance, predict 0.283 ms against 0.340 with a warp per row; 16 000 rows of 100
// edges 0.795 against 0.755.
void agg_rows64(sps_gnn* g, const float* val, const float* in, bool first, float* out, int batch, int accumulate) {
    const __nv_bfloat16* W = g->PB + g->oWv;
    const float* b = g->P + g->obv;
    const int rows = g->m * batch;
    const bool long_rows = g->nnz >= 64 * (int64_t)g->m, block = long_rows && rows < 16384;
    // plain sums where rows are short, or so many beside the variables that one instance's
    // fill the GPU (20 000 x 20 000 of 100 edges a row, predict 1.41 ms compensated)
    if (!first && (!long_rows || (!g->few_rows && g->m >= 16 * 152))) {
        k_agg<64><<<grid_for((int64_t)rows * 32, kT), kT, 0, g->st>>>(g->cptr, g->cidx, val, in, out, g->m, g->n, batch,
                                                                     accumulate);
        return;
    }
    const auto k = first ? (block ? k_agg_rows<true, 8> : k_agg_rows<true, 1>)
                         : (block ? k_agg_rows<false, 8> : k_agg_rows<false, 1>);
    k<<<block ? rows : (rows + kT / 32 - 1) / (kT / 32), kT, 0, g->st>>>(g->cptr, g->cidx, val, in, W, b, out, g->m,
                                                                         g->n, rows, accumulate);
}

template <bool First, bool Heads, bool Two = false>
void node64(sps_gnn* g, const Node64& a) {
    const int64_t tiles = (a.nodes + 127) / 128;
    k_node64<First, Heads, Two><<<(int)std::min<int64_t>(tiles, 2 * 152), kN64T, node64_smem(Two), g->st>>>(a);
}

// The arguments that every launch of k_node64 has: nodes of an instance, of the batch.
Node64 node_args(const sps_gnn* g, int n, int64_t nodes) {
    Node64 a{};
    a.n = n;
    a.nodes = nodes;
    a.err = g->d_err;
    return a;
}

// Forward pass, H = 64.  keep: the variables' last activations are stored too (the
// backward pass reads them).
// M is applied on the constraint side (k_node64 with edges), and the constraints'
// sums are compensated (k_con_update), where there are few rows for the variables and
// their columns are short: edges per variable at most a quarter of the variables per
// row (sps_gnn::few_rows).  Elsewhere both sides add up their neighbours first and
// apply U and M in one pass (k_node64 with two inputs).  predict, ms, few rows' form
// against the other: 500 x 60 000 of 2 edges a column, 16 instances 1.25 / 1.63; 400 x
// 40 000 of 4 0.48 / 0.50, of 16 0.74 / 0.69; 8000 x 128 000 of 4 0.77 / 0.65 (its
// gradient 1.62 / 1.79); 8000 x 40 000 of 13 0.64 / 0.44; 200 000 x 200 000 of 5 3.07 /
// 0.93; 40 000 x 500 of 1570 4.4 / 0.90.
int forward64(sps_gnn* g, int batch, bool keep) {
    const int n = g->n, m = g->m, L = g->L;
    const int64_t NV = (int64_t)n * batch, NC = (int64_t)m * batch;
    const __nv_bfloat16* W = g->PB;
    const float* P = g->P;
    cudaStream_t st = g->st;
    const bool few = g->few_rows;
    if (!g->in4) k_input<64><<<grid_for(NV * 64, kT), kT, 0, st>>>(g->fv, NV, g->Fv, W + g->oWv, P + g->obv, g->HV[0]);
    k_input<64><<<grid_for(NC * 64, kT), kT, 0, st>>>(g->fc, NC, g->Fc, W + g->oWc, P + g->obc, g->HC[0]);
    const bool heads = n >= 128;                  // a tile of 128 nodes then has at most two instances
    for (int l = 0; l < L; ++l) {
        const int64_t o = g->layer_off(l);
        const int64_t oUc = o, oMc = o + 4096, obc = o + 8192;
        const int64_t oUv = obc + 64, oMv = oUv + 4096, obv = oMv + 4096;
        const bool first = l == 0 && g->in4, last = l == L - 1;
        agg_rows64(g, g->ac_c, first ? g->fv : g->HV[l], first, g->AC[l], batch, 0);
        Node64 p = node_args(g, m, NC);
        if (few) {
            k_con_update<<<(int)((NC + kConNodes - 1) / kConNodes), kT, 0, st>>>(g->HC[l], g->AC[l], W + oUc, W + oMc,
                                                                                P + obc, g->HC[l + 1], NC);
            p.h = g->HC[l + 1];
            p.U = W + oMv;
            p.out = g->MH;
            node64<false, false>(g, p);
        } else {
            p.h = g->HC[l];
            p.U = W + oUc;
            p.a = g->AC[l];
            p.M = W + oMc;
            p.bias = P + obc;
            p.out = g->HC[l + 1];
            node64<false, false, true>(g, p);
            // the aggregate passes through the backward pass's buffer
            k_agg<64><<<grid_for(NV * 32, kT), kT, 0, st>>>(g->vptr, g->vidx, g->av_v, g->HC[l + 1], g->dHV2, n, m, batch, 0);
        }
        Node64 a = node_args(g, n, NV);
        a.h = first ? g->fv : g->HV[l];
        a.Win = W + g->oWv;
        a.bin = P + g->obv;
        a.U = W + oUv;
        if (few) {
            a.P = g->MH;
            a.ptr = g->vptr;
            a.idx = g->vidx;
            a.val = g->av_v;
        } else {
            a.a = g->dHV2;
            a.M = W + oMv;
        }
        a.rows = m;
        a.bias = P + obv;
        a.out = last && heads && !keep ? nullptr : g->HV[l + 1];
        a.wx = W + g->oWx;
        a.bx = P + g->obx;
        a.x0 = g->x0;
        a.pool = g->pvp;
        if (!few) { if (last && heads) node64<false, true, true>(g, a); else node64<false, false, true>(g, a); }
        else if (last && heads) { if (first) node64<true, true>(g, a); else node64<false, true>(g, a); }
        else { if (first) node64<true, false>(g, a); else node64<false, false>(g, a); }
    }
    k_head<64><<<grid_for(NC * 32, kT), kT, 0, st>>>(g->HC[L], W + g->oWy, P + g->oby, g->y0, NC);
    k_colsum_part<64><<<dim3(g->nb_pool_c, batch), kT, 0, st>>>(g->HC[L], m, g->pcp);
    if (heads) {
        k_pool_finish64<<<batch, 1024, 0, st>>>(g->pcp, g->nb_pool_c, g->pvp, m, n, NV, W + g->oWo, P + g->obo, g->pool,
                                               g->lw);
    } else {
        k_head<64><<<grid_for(NV * 32, kT), kT, 0, st>>>(g->HV[L], W + g->oWx, P + g->obx, g->x0, NV);
        k_colsum_part<64><<<dim3(g->nb_pool_v, batch), kT, 0, st>>>(g->HV[L], n, g->pvp);
        k_pool_finish<64><<<batch, 128, 0, st>>>(g->pcp, g->nb_pool_c, g->pvp, g->nb_pool_v, m, n, W + g->oWo,
                                                 P + g->obo, g->pool, g->lw);
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : g->fail(-2, std::string("forward: ") + cudaGetErrorString(e));
}

// Forward pass over `batch` instances whose features are already on the device.
// (keep: as forward64)
template <int H>
int forward(sps_gnn* g, int batch, bool keep);
template <>
int forward<64>(sps_gnn* g, int batch, bool keep) { return forward64(g, batch, keep); }
template <>
int forward<32>(sps_gnn* g, int batch, bool) {
    constexpr int H = 32;
    const int n = g->n, m = g->m, L = g->L;
    const int64_t NV = (int64_t)n * batch, NC = (int64_t)m * batch;
    const __nv_bfloat16* W = g->PB;
    const float* P = g->P;
    cudaStream_t st = g->st;
    k_input<H><<<grid_for(NV * H, kT), kT, 0, st>>>(g->fv, NV, g->Fv, W + g->oWv, P + g->obv, g->HV[0]);
    k_input<H><<<grid_for(NC * H, kT), kT, 0, st>>>(g->fc, NC, g->Fc, W + g->oWc, P + g->obc, g->HC[0]);
    for (int l = 0; l < L; ++l) {
        const int64_t o = g->layer_off(l);
        const int64_t oUc = o, oMc = o + H * H, obc = o + 2 * H * H;
        const int64_t oUv = obc + H, oMv = oUv + H * H, obv = oMv + H * H;
        k_agg<H><<<grid_for(NC * 32, kT), kT, 0, st>>>(g->cptr, g->cidx, g->ac_c, g->HV[l], g->AC[l], m, n, batch, 0);
        k_update<<<g->nb_dense, kT, kUpdateSmem, st>>>(g->HC[l], g->AC[l], W + oUc, W + oMc, P + obc, g->HC[l + 1], NC);
        k_agg<H><<<grid_for(NV * 32, kT), kT, 0, st>>>(g->vptr, g->vidx, g->av_v, g->HC[l + 1], g->AV[l], n, m, batch,
                                                       0);
        k_update<<<g->nb_dense, kT, kUpdateSmem, st>>>(g->HV[l], g->AV[l], W + oUv, W + oMv, P + obv, g->HV[l + 1], NV);
    }
    k_head<H><<<grid_for(NV * 32, kT), kT, 0, st>>>(g->HV[L], W + g->oWx, P + g->obx, g->x0, NV);
    k_head<H><<<grid_for(NC * 32, kT), kT, 0, st>>>(g->HC[L], W + g->oWy, P + g->oby, g->y0, NC);
    k_colsum_part<H><<<dim3(g->nb_pool_c, batch), kT, 0, st>>>(g->HC[L], m, g->pcp);
    k_colsum_part<H><<<dim3(g->nb_pool_v, batch), kT, 0, st>>>(g->HV[L], n, g->pvp);
    k_pool_finish<H><<<batch, 2 * H, 0, st>>>(g->pcp, g->nb_pool_c, g->pvp, g->nb_pool_v, m, n, W + g->oWo,
                                              P + g->obo, g->pool, g->lw);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : g->fail(-2, std::string("forward: ") + cudaGetErrorString(e));
}

// Blocks of a tensor-core node kernel over `nodes` nodes.
int node_blocks(int64_t nodes) { return (int)std::min<int64_t>((nodes + 127) / 128, 2 * 152); }

// The weight gradients of all layers (H = 64) into g->G, given the losses' output
// gradients dx0, dy0, dlw: see k_back64 for what each side keeps.
int backward64(sps_gnn* g, int batch) {
    const int n = g->n, m = g->m, L = g->L;
    const int64_t NV = (int64_t)n * batch, NC = (int64_t)m * batch;
    const __nv_bfloat16* W = g->PB;
    const float* P = g->P;
    cudaStream_t st = g->st;
    const int bv = node_blocks(NV), bc = node_blocks(NC);
    SumJobs jobs;
    int nj = 0;
    float* part = g->part;                                      // handed out piece by piece
    auto take = [&](int blocks, int stride) {
        float* p = part;
        part += (int64_t)blocks * stride;
        return p;
    };
    auto sum = [&](const float* p, int blocks, int stride, int width, int64_t off) {
        jobs.job[nj++] = SumJob{p, g->G + off, blocks, stride, width};
    };
    Back64 var{};                                               // what the variable side's passes share
    var.ptr = g->vptr;
    var.idx = g->vidx;
    var.val = g->ac_v;
    var.rows = m;
    var.Win = W + g->oWv;
    var.bin = P + g->obv;
    var.n = n;
    var.nodes = NV;
    var.err = g->d_err;
    Back64 con{};
    con.Win = W + g->oWc;
    con.bin = P + g->obc;
    con.n = m;
    con.nodes = NC;
    con.err = g->d_err;
    const bool in4 = g->in4;
    // rows of the constraint side's gradient are added along a variable's edges where it is
    // read, or first: a tile's chain of edges outlasts the stream it saves from about eight
    // edges a column on (gradient, along the edges / first: 200 000 x 200 000 of 5 2.92 /
    // 2.83 ms, 500 x 60 000 of 2 4.60 / 4.79, 8000 x 40 000 of 13 1.15 / 1.08, 500 x 8000 of 31
    // 0.58 / 0.52, 40 000 x 500 of 1570 4.3 / 1.9)
    const bool edges = g->nnz < 8 * (int64_t)n;
    float *dhv = g->dHV, *dhc = g->dHC, *dhc_next = g->dHC2;
    for (int l = L - 1; l >= 0; --l) {
        const int64_t o = g->layer_off(l);
        const int64_t oUc = o, oMc = o + 4096, obc = o + 8192;
        const int64_t oUv = obc + 64, oMv = oUv + 4096, obv = oMv + 4096;
        const bool first = l == 0 && in4, last = l == L - 1;
        if (!last && !edges)
            k_agg<64><<<grid_for(NV * 32, kT), kT, 0, st>>>(g->vptr, g->vidx, g->ac_v, g->dA, dhv, n, m, batch, 1);
        // variable update: z, dh (in place of dout) and the gradients of Uv, bv (and of the x head)
        Back64 a = var;
        a.dout = last ? nullptr : dhv;
        a.Q = last || !edges ? nullptr : g->dA;
        a.dhead = g->dx0;
        a.whead = W + g->oWx;
        a.dlw = g->dlw;
        a.wpool = W + g->oWo + 64;
        a.out = g->HV[l + 1];
        a.h = first ? g->fv : g->HV[l];
        a.W = W + oUv;
        a.z = g->dHV2;
        a.dh = dhv;
        a.part = take(bv, bk::kOut);
        a.hpart = last ? take(bv, bk::kHeadOut) : nullptr;
        if (first) k_back64<true><<<bv, bk::kThreads, bk::kSmem, st>>>(a);
        else k_back64<false><<<bv, bk::kThreads, bk::kSmem, st>>>(a);
        sum(a.part, bv, bk::kOut, 4096, oUv);
        sum(a.part + 4096, bv, bk::kOut, 64, obv);
        if (last) sum(a.hpart, bv, bk::kHeadOut, 65, g->oWx);
        // sum_j a_ij z_j: the gradients of Mv and, added to the y head's or the next layer's, of HC[l + 1]
        agg_rows64(g, g->av_c, g->dHV2, false, g->AG, batch, 0);
        Back64 b = con;
        b.dout = g->AG;
        b.h = g->HC[l + 1];
        b.W = W + oMv;
        b.dh = dhc;
        b.accumulate = 1;
        b.part = take(bc, bk::kOut);
        if (last) {     // the y head: dHC = dy0 wy + dlw wo / m
            k_head_back<64><<<g->nb_dense, kT, 0, st>>>(g->HC[L], g->dy0, W + g->oWy, g->dlw, W + g->oWo, m, batch, dhc,
                                                        take(g->nb_dense, 65));
            sum(part - (int64_t)g->nb_dense * 65, g->nb_dense, 65, 65, g->oWy);
        }
        k_back64<false><<<bc, bk::kThreads, bk::kSmem, st>>>(b);
        sum(b.part, bc, bk::kOut, 4096, oMv);
        // constraint update: dHC[l], and dA of the aggregation for the variables
        Back64 c = con;
        c.dout = dhc;
        c.out = g->HC[l + 1];
        c.h = g->HC[l];
        c.W = W + oUc;
        c.dh = dhc_next;
        c.part = take(bc, bk::kOut);
        k_back64<false><<<bc, bk::kThreads, bk::kSmem, st>>>(c);
        sum(c.part, bc, bk::kOut, 4096, oUc);
        sum(c.part + 4096, bc, bk::kOut, 64, obc);
        c.h = g->AC[l];
        c.W = W + oMc;
        c.dh = g->dA;
        c.part = take(bc, bk::kOut);
        k_back64<false><<<bc, bk::kThreads, bk::kSmem, st>>>(c);
        sum(c.part, bc, bk::kOut, 4096, oMc);
        std::swap(dhc, dhc_next);
    }
    // input layers
    if (in4) {
        Back64 a = var;
        a.dout = dhv;
        a.Q = g->dA;                // (in4: short columns)
        a.h = g->fv;
        a.part = take(2 * 152, kInOut);
        k_in_back64<<<2 * 152, bk::kThreads, 0, st>>>(a);
        sum(a.part, 2 * 152, kInOut, 320, g->oWv);
    } else {
        k_agg<64><<<grid_for(NV * 32, kT), kT, 0, st>>>(g->vptr, g->vidx, g->ac_v, g->dA, dhv, n, m, batch, 1);
        const int w = 64 * g->Fv + 64;
        float* p = take(g->nb_dense, w);
        k_input_back<64><<<g->nb_dense, kT, 0, st>>>(dhv, g->HV[0], g->fv, g->Fv, NV, p);
        sum(p, g->nb_dense, w, w, g->oWv);
    }
    {
        const int w = 64 * g->Fc + 64;
        float* p = take(g->nb_dense, w);
        k_input_back<64><<<g->nb_dense, kT, 0, st>>>(dhc, g->HC[0], g->fc, g->Fc, NC, p);
        sum(p, g->nb_dense, w, w, g->oWc);
    }
    k_sum_jobs<<<dim3(16, nj), kT, 0, st>>>(jobs);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : g->fail(-2, std::string("backward: ") + cudaGetErrorString(e));
}

// The loss from its partials (waits for the stream).
int read_loss(sps_gnn* g, int batch, double* loss) {
    if (!loss) return 0;
    const int nbl = g->nb_loss;
    std::vector<double> lp(2 * nbl + 1);
    GNN_CK(cudaMemcpyAsync(lp.data(), g->lpart, sizeof(double) * lp.size(), cudaMemcpyDeviceToHost, g->st));
    GNN_CK(cudaStreamSynchronize(g->st));
    double sx = 0, sy = 0;
    for (int b = 0; b < nbl; ++b) { sx += lp[b]; sy += lp[nbl + b]; }
    const float ax = g->opt.loss_x, ay = g->opt.loss_y, ao = g->opt.loss_omega;
    *loss = (ax * sx / g->n + ay * sy / g->m + ao * lp[2 * nbl]) / batch;
    return 0;
}

// Loss (host value) and gradient into g->G (zeroed here) for `batch` instances
// whose features and targets are on the device.
template <int H>
int backward(sps_gnn* g, int batch, double* loss) {
    const int n = g->n, m = g->m, L = g->L;
    const int64_t NV = (int64_t)n * batch, NC = (int64_t)m * batch;
    const __nv_bfloat16* W = g->PB;
    cudaStream_t st = g->st;
    const float ax = g->opt.loss_x, ay = g->opt.loss_y, ao = g->opt.loss_omega;
    GNN_CK(cudaMemsetAsync(g->G, 0, sizeof(float) * g->np, st));
    // output gradients: loss = (1/B) sum_s [ax/n |x0-xt|^2 + ay/m |y0-yt|^2 + ao (lw-lt)^2]
    const int nbl = g->nb_loss;
    k_sq_loss<<<nbl, kT, 0, st>>>(g->x0, g->xt, NV, 2.f * ax / (float(n) * batch), g->dx0, g->lpart);
    k_sq_loss<<<nbl, kT, 0, st>>>(g->y0, g->yt, NC, 2.f * ay / (float(m) * batch), g->dy0, g->lpart + nbl);
    k_sq_loss<<<1, kT, 0, st>>>(g->lw, g->lt, batch, 2.f * ao / float(batch), g->dlw, g->lpart + 2 * nbl);
    if constexpr (H == 64) {
        k_omega_back<H><<<1, 2 * H, 0, st>>>(g->dlw, g->pool, batch, g->G + g->oWo, g->G + g->obo);
        if (int rc = backward64(g, batch)) return rc;
    } else {
        // heads
        const int nbh = g->nb_dense;
        k_head_back<H><<<nbh, kT, 0, st>>>(g->HV[L], g->dx0, W + g->oWx, g->dlw, W + g->oWo + H, n, batch, g->dHV,
                                           g->part);
        k_sum_parts<<<4, 256, 0, st>>>(g->part, nbh, H + 1, 1.f, g->G + g->oWx);
        k_head_back<H><<<nbh, kT, 0, st>>>(g->HC[L], g->dy0, W + g->oWy, g->dlw, W + g->oWo, m, batch, g->dHC, g->part);
        k_sum_parts<<<4, 256, 0, st>>>(g->part, nbh, H + 1, 1.f, g->G + g->oWy);
        k_omega_back<H><<<1, 2 * H, 0, st>>>(g->dlw, g->pool, batch, g->G + g->oWo, g->G + g->obo);
        // layers, last to first.  dHV / dHC hold the gradient of HV[l+1] / HC[l+1].
        float *dhv = g->dHV, *dhc = g->dHC, *dhv_next = g->dHV2, *dhc_next = g->dHC2;
        const int width = 2 * H * H + H;
        for (int l = L - 1; l >= 0; --l) {
            const int64_t o = g->layer_off(l);
            const int64_t oUc = o, oMc = o + H * H;
            const int64_t oUv = oMc + H * H + H, oMv = oUv + H * H;
            // variable update: HV[l+1] = relu(Uv HV[l] + Mv AV[l] + bv)
            k_update_back<<<nbh, kT, kUpdateBackSmem, st>>>(dhv, g->HV[l + 1], g->HV[l], g->AV[l], W + oUv,
                                                                     W + oMv, dhv_next, 0, g->dA, g->part, NV);
            k_sum_parts<<<32, 256, 0, st>>>(g->part, nbh, width, 1.f, g->G + oUv);
            // AV[l] = agg_v(HC[l+1]): dHC[l+1] += agg over constraints with a_v values
            k_agg<H><<<grid_for(NC * 32, kT), kT, 0, st>>>(g->cptr, g->cidx, g->av_c, g->dA, dhc, m, n, batch, 1);
            // constraint update: HC[l+1] = relu(Uc HC[l] + Mc AC[l] + bc)
            k_update_back<<<nbh, kT, kUpdateBackSmem, st>>>(dhc, g->HC[l + 1], g->HC[l], g->AC[l], W + oUc,
                                                                     W + oMc, dhc_next, 0, g->dA, g->part, NC);
            k_sum_parts<<<32, 256, 0, st>>>(g->part, nbh, width, 1.f, g->G + oUc);
            // AC[l] = agg_c(HV[l]): dHV[l] += agg over variables with a_c values
            k_agg<H><<<grid_for(NV * 32, kT), kT, 0, st>>>(g->vptr, g->vidx, g->ac_v, g->dA, dhv_next, n, m, batch, 1);
            std::swap(dhv, dhv_next);
            std::swap(dhc, dhc_next);
        }
        // input layers
        k_input_back<H><<<nbh, kT, 0, st>>>(dhv, g->HV[0], g->fv, g->Fv, NV, g->part);
        k_sum_parts<<<4, 256, 0, st>>>(g->part, nbh, H * g->Fv + H, 1.f, g->G + g->oWv);
        k_input_back<H><<<nbh, kT, 0, st>>>(dhc, g->HC[0], g->fc, g->Fc, NC, g->part);
        k_sum_parts<<<4, 256, 0, st>>>(g->part, nbh, H * g->Fc + H, 1.f, g->G + g->oWc);
    }
    GNN_CK(cudaGetLastError());
    return read_loss(g, batch, loss);
}

int upload_inputs(sps_gnn* g, int batch, const float* vf, const float* cf, const float* xt, const float* yt,
                  const float* lt) {
    cudaStream_t st = g->st;
    const size_t nv = (size_t)g->n * batch, nc = (size_t)g->m * batch;
    if (g->lpf) {
        GNN_CK(cudaMemcpyAsync(g->craw, vf, sizeof(float) * nv, cudaMemcpyHostToDevice, st));
        GNN_CK(cudaMemcpyAsync(g->braw, cf, sizeof(float) * nc, cudaMemcpyHostToDevice, st));
        k_lp_con_features<<<grid_for((int64_t)nc * 32, kT), kT, 0, st>>>(g->cptr, g->cidx, g->kind, g->craw, g->braw,
                                                                       g->n, g->m, batch, g->fc, g->cmin);
        k_lp_var_features<<<grid_for((int64_t)nv, kT), kT, 0, st>>>(g->vptr, g->vidx, g->kind, g->craw, g->cmin,
                                                                  g->n, g->m, batch, g->fv);
        GNN_CK(cudaGetLastError());
    } else {
        GNN_CK(cudaMemcpyAsync(g->fv, vf, sizeof(float) * nv * g->Fv, cudaMemcpyHostToDevice, st));
        GNN_CK(cudaMemcpyAsync(g->fc, cf, sizeof(float) * nc * g->Fc, cudaMemcpyHostToDevice, st));
    }
    if (xt) GNN_CK(cudaMemcpyAsync(g->xt, xt, sizeof(float) * nv, cudaMemcpyHostToDevice, st));
    if (yt) GNN_CK(cudaMemcpyAsync(g->yt, yt, sizeof(float) * nc, cudaMemcpyHostToDevice, st));
    if (lt) GNN_CK(cudaMemcpyAsync(g->lt, lt, sizeof(float) * batch, cudaMemcpyHostToDevice, st));
    return 0;
}

int check_batch(sps_gnn* g, int32_t batch, const float* vf, const float* cf) {
    if (batch < 1 || batch > g->B) return g->fail(-1, "batch must be in [1, max_batch]");
    if (!vf || !cf) return g->fail(-1, "null features");
    return 0;
}

// Scaled-uniform initialisation (fan-in), deterministic in the seed.
void init_params(std::vector<float>& p, const sps_gnn* g) {
    uint64_t s = g->opt.seed * 6364136223846793005ULL + 1442695040888963407ULL;
    auto uni = [&]() {
        s ^= s >> 12; s ^= s << 25; s ^= s >> 27;
        return double((s * 2685821657736338717ULL) >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
    };
    const int H = g->H;
    auto fill = [&](int64_t off, int64_t count, double fan_in) {
        const double a = std::sqrt(3.0 / std::max(1.0, fan_in));
        for (int64_t t = 0; t < count; ++t) p[off + t] = float(a * uni());
    };
    std::fill(p.begin(), p.end(), 0.f);
    fill(g->oWv, (int64_t)H * g->Fv, g->Fv);
    fill(g->oWc, (int64_t)H * g->Fc, g->Fc);
    for (int l = 0; l < g->L; ++l) {
        const int64_t o = g->layer_off(l);
        fill(o, 2LL * H * H, 2.0 * H);                       // Uc, Mc
        fill(o + 2LL * H * H + H, 2LL * H * H, 2.0 * H);     // Uv, Mv
    }
    fill(g->oWx, H, H);
    fill(g->oWy, H, H);
    fill(g->oWo, 2 * H, 2.0 * H);
}

template <int H>
int run_loss_grad(sps_gnn* g, int batch, double* loss) {
    if (int rc = forward<H>(g, batch, true)) return rc;
    return backward<H>(g, batch, loss);
}

}  // namespace

namespace sps {
namespace gnn {

int device_io(sps_gnn* g, DeviceIO* io) {
    if (!g || !io) return -1;
    io->n = g->n;
    io->m = g->m;
    io->max_batch = g->B;
    io->lp_features = g->lpf;
    io->device = g->opt.device;
    io->stream = g->st;
    io->c_in = g->craw;
    io->b_in = g->braw;
    io->x0 = g->x0;
    io->y0 = g->y0;
    io->log_omega = g->lw;
    return 0;
}

int check_device_error(sps_gnn* g) { return g ? device_error(g) : -1; }

int forward_in_place(sps_gnn* g, int batch) {
    if (!g || !g->lpf || batch < 1 || batch > g->B) return g ? g->fail(-1, "forward_in_place needs lp_features") : -1;
    k_lp_con_features<<<grid_for((int64_t)g->m * batch * 32, kT), kT, 0, g->st>>>(
        g->cptr, g->cidx, g->kind, g->craw, g->braw, g->n, g->m, batch, g->fc, g->cmin);
    k_lp_var_features<<<grid_for((int64_t)g->n * batch, kT), kT, 0, g->st>>>(g->vptr, g->vidx, g->kind, g->craw,
                                                                          g->cmin, g->n, g->m, batch, g->fv);
    if (cudaGetLastError() != cudaSuccess) return g->fail(-2, "feature kernels failed to launch");
    return g->H == 64 ? forward<64>(g, batch, false) : forward<32>(g, batch, false);
}

}  // namespace gnn
}  // namespace sps

extern "C" {

int sps_gnn_options_init(sps_gnn_options* o) {
    if (!o) return -1;
    std::memset(o, 0, sizeof(*o));
    o->hidden = 64;
    o->layers = 3;
    o->seed = 0;
    o->lr = 1e-3f;
    o->beta1 = 0.9f;
    o->beta2 = 0.999f;
    o->eps = 1e-8f;
    o->loss_x = 1.f;
    o->loss_y = 1.f;
    o->loss_omega = 0.1f;
    o->max_batch = 8;
    o->device = 0;
    return 0;
}

int sps_gnn_create(const sps_gnn_graph* gr, const sps_gnn_options* opt_in, sps_gnn** out) {
    g_gnn_create_error.clear();
    if (!gr || !out) { g_gnn_create_error = "null graph or output"; return -1; }
    *out = nullptr;
    sps_gnn_options opt;
    if (opt_in) opt = *opt_in; else sps_gnn_options_init(&opt);
    if (opt.hidden != 32 && opt.hidden != 64) { g_gnn_create_error = "hidden must be 32 or 64"; return -1; }
    if (opt.layers < 1 || opt.layers > 8 || opt.max_batch < 1) { g_gnn_create_error = "layers in 1..8, max_batch >= 1"; return -1; }
    if (gr->n_var < 1 || gr->n_con < 1 || gr->f_var < 1 || gr->f_var > kMaxF || gr->f_con < 1 || gr->f_con > kMaxF ||
        !gr->con_ptr) {
        g_gnn_create_error = "graph needs n_var, n_con >= 1, feature widths in 1..8 and con_ptr";
        return -1;
    }
    const int m = gr->n_con, n = gr->n_var;
    if (gr->con_ptr[0] != 0) { g_gnn_create_error = "con_ptr[0] != 0"; return -1; }
    for (int i = 0; i < m; ++i)
        if (gr->con_ptr[i + 1] < gr->con_ptr[i]) { g_gnn_create_error = "con_ptr not monotone"; return -1; }
    const int64_t nnz = gr->con_ptr[m];
    if (nnz > 0 && (!gr->con_idx || !gr->con_val)) { g_gnn_create_error = "null con_idx / con_val"; return -1; }
    for (int64_t k = 0; k < nnz; ++k)
        if (gr->con_idx[k] < 0 || gr->con_idx[k] >= n || !std::isfinite(gr->con_val[k])) {
            g_gnn_create_error = "edge " + std::to_string(k) + ": variable out of range or non-finite value";
            return -1;
        }
    if (opt.lp_features && (gr->f_var != 1 || gr->f_con != 1)) {
        g_gnn_create_error = "lp_features takes one input per variable (c) and per row (b): f_var = f_con = 1";
        return -1;
    }
    auto g = new sps_gnn();
    g->g = *gr;
    g->opt = opt;
    g->lpf = opt.lp_features ? 1 : 0;
    g->H = opt.hidden; g->L = opt.layers;
    g->Fv = g->lpf ? 4 : gr->f_var;
    g->Fc = g->lpf ? 4 : gr->f_con;
    g->n = n; g->m = m; g->B = opt.max_batch; g->nnz = nnz;
    const int H = g->H;
    g->few_rows = 4.0 * double(m) * double(nnz) <= double(n) * double(n);
    g->in4 = H == 64 && g->Fv == 4 && g->few_rows;
    // parameter offsets
    int64_t o = 0;
    g->oWv = o; o += (int64_t)H * g->Fv; g->obv = o; o += H;
    g->oWc = o; o += (int64_t)H * g->Fc; g->obc = o; o += H;
    g->oL0 = o; g->per_layer = 4LL * H * H + 2 * H; o += g->per_layer * g->L;
    g->oWx = o; o += H; g->obx = o; o += 1;
    g->oWy = o; o += H; g->oby = o; o += 1;
    g->oWo = o; o += 2 * H; g->obo = o; o += 1;
    g->np = o;
    // host graph: degrees, normalised values, CSR by variable
    std::vector<int32_t> degc(m), degv(n, 0), vptr(n + 1, 0), vidx(nnz);
    std::vector<float> ac_c(nnz), av_c(nnz), av_v(nnz), ac_v(nnz);
    std::vector<int8_t> kd(m, 0);
    for (int i = 0; i < m; ++i) degc[i] = gr->con_ptr[i + 1] - gr->con_ptr[i];
    for (int64_t k = 0; k < nnz; ++k) degv[gr->con_idx[k]]++;
    for (int j = 0; j < n; ++j) vptr[j + 1] = vptr[j] + degv[j];
    std::vector<int32_t> fill(vptr.begin(), vptr.end() - 1);
    for (int i = 0; i < m; ++i)
        for (int32_t k = gr->con_ptr[i]; k < gr->con_ptr[i + 1]; ++k) {
            const int j = gr->con_idx[k];
            const float a = gr->con_val[k];
            ac_c[k] = a / float(degc[i]);
            av_c[k] = a / float(degv[j]);
            const int32_t q = fill[j]++;
            vidx[q] = i;
            av_v[q] = av_c[k];
            ac_v[q] = ac_c[k];
        }
    int rc = 0;
    {
        sps_gnn* gg = g;
        auto setup = [&]() -> int {
            sps_gnn* g = gg;
            GNN_CK(cudaSetDevice(opt.device));
            GNN_CK(cudaStreamCreateWithFlags(&g->st, cudaStreamNonBlocking));
            if (!set_smem_attrs(H)) return g->fail(-2, "shared-memory attribute");
            GNN_CK(g->alloc(&g->cptr, m + 1)); GNN_CK(g->alloc(&g->cidx, nnz));
            GNN_CK(g->alloc(&g->vptr, n + 1)); GNN_CK(g->alloc(&g->vidx, nnz));
            GNN_CK(g->alloc(&g->ac_c, nnz)); GNN_CK(g->alloc(&g->av_c, nnz));
            GNN_CK(g->alloc(&g->av_v, nnz)); GNN_CK(g->alloc(&g->ac_v, nnz));
            auto up = [&](void* d, const void* s, size_t b) {
                return b ? cudaMemcpyAsync(d, s, b, cudaMemcpyHostToDevice, g->st) : cudaSuccess;
            };
            GNN_CK(up(g->cptr, gr->con_ptr, 4 * (size_t)(m + 1))); GNN_CK(up(g->cidx, gr->con_idx, 4 * (size_t)nnz));
            GNN_CK(up(g->vptr, vptr.data(), 4 * (size_t)(n + 1))); GNN_CK(up(g->vidx, vidx.data(), 4 * (size_t)nnz));
            GNN_CK(up(g->ac_c, ac_c.data(), 4 * (size_t)nnz)); GNN_CK(up(g->av_c, av_c.data(), 4 * (size_t)nnz));
            GNN_CK(up(g->av_v, av_v.data(), 4 * (size_t)nnz)); GNN_CK(up(g->ac_v, ac_v.data(), 4 * (size_t)nnz));
            GNN_CK(g->alloc(&g->P, g->np)); GNN_CK(g->alloc(&g->G, g->np));
            GNN_CK(g->alloc(&g->M1, g->np)); GNN_CK(g->alloc(&g->M2, g->np));
            GNN_CK(g->alloc(&g->PB, g->np));
            const int64_t B = g->B, NV = (int64_t)n * B, NC = (int64_t)m * B;
            GNN_CK(g->alloc(&g->fv, NV * g->Fv)); GNN_CK(g->alloc(&g->fc, NC * g->Fc));
            if (g->lpf) {
                GNN_CK(g->alloc(&g->craw, NV)); GNN_CK(g->alloc(&g->braw, NC)); GNN_CK(g->alloc(&g->cmin, NC));
                GNN_CK(g->alloc(&g->kind, m));
                if (gr->con_kind)
                    for (int i = 0; i < m; ++i) kd[i] = gr->con_kind[i] ? 1 : 0;
                GNN_CK(up(g->kind, kd.data(), (size_t)m));
            }
            GNN_CK(g->alloc(&g->xt, NV)); GNN_CK(g->alloc(&g->yt, NC)); GNN_CK(g->alloc(&g->lt, B));
            g->HV.resize(g->L + 1); g->HC.resize(g->L + 1); g->AV.resize(g->L); g->AC.resize(g->L);
            // (H = 64: the variables' aggregates are not stored, nor an input layer that is recomputed)
            for (int l = 0; l <= g->L; ++l) {
                if (l > 0 || !g->in4) GNN_CK(g->alloc(&g->HV[l], NV * H));
                GNN_CK(g->alloc(&g->HC[l], NC * H));
            }
            for (int l = 0; l < g->L; ++l) {
                if (H == 32) GNN_CK(g->alloc(&g->AV[l], NV * H));
                GNN_CK(g->alloc(&g->AC[l], NC * H));
            }
            GNN_CK(g->alloc(&g->dHV, NV * H)); GNN_CK(g->alloc(&g->dHV2, NV * H));
            GNN_CK(g->alloc(&g->dHC, NC * H)); GNN_CK(g->alloc(&g->dHC2, NC * H));
            GNN_CK(g->alloc(&g->dA, (H == 64 ? NC : std::max(NV, NC)) * H));
            GNN_CK(g->alloc(&g->x0, NV)); GNN_CK(g->alloc(&g->y0, NC)); GNN_CK(g->alloc(&g->lw, B));
            GNN_CK(g->alloc(&g->dx0, NV)); GNN_CK(g->alloc(&g->dy0, NC)); GNN_CK(g->alloc(&g->dlw, B));
            GNN_CK(g->alloc(&g->pool, 2 * H * B));
            GNN_CK(g->alloc(&g->d_err, 1));
            GNN_CK(cudaMemsetAsync(g->d_err, 0, sizeof(int32_t), g->st));
            g->nb_dense = 152 * 2;
            g->nb_loss = 152 * 2;
            g->nb_pool_c = std::max(1, std::min(64, (m + 31) / 32));
            g->nb_pool_v = std::max(1, std::min(152, (n + 31) / 32));
            g->part_floats = (int64_t)g->nb_dense * (2 * H * H + H);
            if (H == 64) {      // backward64's partials, all layers
                const int64_t bv = node_blocks(NV), bc = node_blocks(NC);
                g->part_floats = g->L * (bv + 3 * bc) * bk::kOut + bv * bk::kHeadOut +
                                 (int64_t)g->nb_dense * (65 + kInOut + 2 * (64 * kMaxF + 64));
            }
            GNN_CK(g->alloc(&g->part, g->part_floats));
            GNN_CK(g->alloc(&g->lpart, 2 * g->nb_loss + 1));
            GNN_CK(g->alloc(&g->pcp, (int64_t)g->nb_pool_c * H * B));
            GNN_CK(g->alloc(&g->pvp, std::max<int64_t>((int64_t)g->nb_pool_v * H * B, (NV + 127) / 128 * 128)));
            if (H == 64) { GNN_CK(g->alloc(&g->MH, NC * H)); GNN_CK(g->alloc(&g->AG, NC * H)); }
            std::vector<float> p(g->np);
            init_params(p, g);
            GNN_CK(up(g->P, p.data(), sizeof(float) * g->np));
            GNN_CK(cudaMemsetAsync(g->M1, 0, sizeof(float) * g->np, g->st));
            GNN_CK(cudaMemsetAsync(g->M2, 0, sizeof(float) * g->np, g->st));
            k_to_bf16<<<grid_for(g->np, 256), 256, 0, g->st>>>(g->P, g->PB, g->np);
            GNN_CK(cudaGetLastError());
            GNN_CK(cudaStreamSynchronize(g->st));
            return 0;
        };
        rc = setup();
    }
    if (rc) {
        g_gnn_create_error = g->err;
        delete g;
        return rc;
    }
    *out = g;
    return 0;
}

int sps_gnn_predict(sps_gnn* g, int32_t batch, const float* vf, const float* cf, float* x0, float* y0, float* lw) {
    sps::NvtxRange nvtx_range("sps_gnn_predict");
    if (!g) return -1;
    if (int rc = check_batch(g, batch, vf, cf)) return rc;
    GNN_CK(cudaSetDevice(g->opt.device));
    if (int rc = upload_inputs(g, batch, vf, cf, nullptr, nullptr, nullptr)) return rc;
    const int rc = g->H == 64 ? forward<64>(g, batch, false) : forward<32>(g, batch, false);
    if (rc) return rc;
    const size_t nv = (size_t)g->n * batch, nc = (size_t)g->m * batch;
    if (x0) GNN_CK(cudaMemcpyAsync(x0, g->x0, sizeof(float) * nv, cudaMemcpyDeviceToHost, g->st));
    if (y0) GNN_CK(cudaMemcpyAsync(y0, g->y0, sizeof(float) * nc, cudaMemcpyDeviceToHost, g->st));
    if (lw) GNN_CK(cudaMemcpyAsync(lw, g->lw, sizeof(float) * batch, cudaMemcpyDeviceToHost, g->st));
    GNN_CK(cudaStreamSynchronize(g->st));
    return device_error(g);
}

int sps_gnn_loss_grad(sps_gnn* g, int32_t batch, const float* vf, const float* cf, const float* xt, const float* yt,
                      const float* lt, double* loss, float* grad) {
    if (!g) return -1;
    if (int rc = check_batch(g, batch, vf, cf)) return rc;
    if (!xt || !yt || !lt) return g->fail(-1, "null targets");
    GNN_CK(cudaSetDevice(g->opt.device));
    if (int rc = upload_inputs(g, batch, vf, cf, xt, yt, lt)) return rc;
    const int rc = g->H == 64 ? run_loss_grad<64>(g, batch, loss) : run_loss_grad<32>(g, batch, loss);
    if (rc) return rc;
    if (grad) {
        GNN_CK(cudaMemcpyAsync(grad, g->G, sizeof(float) * g->np, cudaMemcpyDeviceToHost, g->st));
        GNN_CK(cudaStreamSynchronize(g->st));
    }
    return device_error(g);
}

int sps_gnn_train_step(sps_gnn* g, int32_t batch, const float* vf, const float* cf, const float* xt, const float* yt,
                       const float* lt, double* loss) {
    sps::NvtxRange nvtx_range("sps_gnn_train_step");
    if (!g) return -1;
    if (int rc = check_batch(g, batch, vf, cf)) return rc;
    if (!xt || !yt || !lt) return g->fail(-1, "null targets");
    GNN_CK(cudaSetDevice(g->opt.device));
    if (int rc = upload_inputs(g, batch, vf, cf, xt, yt, lt)) return rc;
    const int rc = g->H == 64 ? run_loss_grad<64>(g, batch, loss) : run_loss_grad<32>(g, batch, loss);
    if (rc) return rc;
    g->step += 1;
    const float c1 = 1.f - std::pow(g->opt.beta1, float(g->step)), c2 = 1.f - std::pow(g->opt.beta2, float(g->step));
    k_adam<<<grid_for(g->np, 256), 256, 0, g->st>>>(g->P, g->G, g->M1, g->M2, g->PB, g->np, g->opt.lr,
                                                    g->opt.beta1, g->opt.beta2, g->opt.eps, c1, c2);
    GNN_CK(cudaGetLastError());
    return device_error(g);     // (synchronises the stream)
}

int64_t sps_gnn_num_params(const sps_gnn* g) { return g ? g->np : -1; }

int sps_gnn_get_params(sps_gnn* g, float* out) {
    if (!g || !out) return -1;
    GNN_CK(cudaSetDevice(g->opt.device));
    GNN_CK(cudaMemcpyAsync(out, g->P, sizeof(float) * g->np, cudaMemcpyDeviceToHost, g->st));
    GNN_CK(cudaStreamSynchronize(g->st));
    return 0;
}

int sps_gnn_set_params(sps_gnn* g, const float* in) {
    if (!g || !in) return -1;
    for (int64_t t = 0; t < g->np; ++t)
        if (!std::isfinite(in[t])) return g->fail(-1, "non-finite parameter");
    GNN_CK(cudaSetDevice(g->opt.device));
    GNN_CK(cudaMemcpyAsync(g->P, in, sizeof(float) * g->np, cudaMemcpyHostToDevice, g->st));
    GNN_CK(cudaMemsetAsync(g->M1, 0, sizeof(float) * g->np, g->st));
    GNN_CK(cudaMemsetAsync(g->M2, 0, sizeof(float) * g->np, g->st));
    k_to_bf16<<<grid_for(g->np, 256), 256, 0, g->st>>>(g->P, g->PB, g->np);
    GNN_CK(cudaGetLastError());
    GNN_CK(cudaStreamSynchronize(g->st));
    g->step = 0;
    return 0;
}

const char* sps_gnn_last_error(const sps_gnn* g) { return g ? g->err.c_str() : g_gnn_create_error.c_str(); }

void sps_gnn_destroy(sps_gnn* g) { delete g; }

}  // extern "C"
