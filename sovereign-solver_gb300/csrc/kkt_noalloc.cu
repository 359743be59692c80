// kkt_noalloc.cu — relative KKT error of a given point, computed without
// allocating any device memory (sps_kkt_noalloc in include/sps_pdhg.h).
//
// Who needs it: callers that hold the LP and the point in device memory they
// own and cannot call cudaMalloc at that moment — code running inside another
// framework's memory pool or a fixed device-memory budget, and latency-critical
// loops where a cudaMalloc/cudaFree would synchronise the device.  It is the
// same FP64 check that sps_solve runs on its own (allocated) workspace, as a
// variant whose scratch is a file-scope device array.
//
// Order-independent K^T y.  The caller gives K in CSR only, so K^T y is a
// scatter of the products a_ij * y_i into the columns.  Floating-point atomic
// adds would make the sum depend on the order the hardware runs them in.
// Instead every product is cut into three integer digits on grids fixed for
// the whole call (units U, U 2^-b, U 2^-2b, U a power of two above the largest
// |a_ij y_i|, b chosen so that no column sum of one digit can exceed 2^51), and
// the digits are added with 64-bit integer atomics.  Integer sums do not depend
// on order, so the result is bitwise reproducible; it carries about 3b bits
// below the largest product (b = 51 - ceil(log2(nnz + 1)), e.g. 117 bits for
// 1e4 nonzeros, 60 bits for 2^31), as good as or better than an FP64 sum.
//
// Scratch: g_noalloc_scratch, kScratchWords 8-byte words (about 6.3 MB), held
// by every GPU that loads the library until the process exits:
//   [0, 3 kMaxCols)                        three digit accumulators per column
//   [kPartBase, + 2 kMaxBlocks kParts)     per-block partial sums of the two passes
//   [kMaxBase, + kMaxBlocks)               per-block largest |a_ij y_i| (bits)
//   kTicketSlot                            ticket of the column pass
// (all written by the call's first pass before they are read: no clearing launches)
// Limits: n <= kMaxCols (262144) columns; any number of rows.
// Every call shares the array: two calls that overlap on the GPU (different
// streams, or different host threads without ordering) race and return
// garbage; order them on one stream.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <string>

#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/sps_pdhg.h"

namespace sps {
void set_create_error(const std::string& msg);   // defined in api.cu (message for sps_last_error(NULL))
}

namespace {

constexpr int kThreads = 256;
constexpr int kMaxBlocks = 1024;
constexpr int kParts = 4;
constexpr int kMaxCols = 1 << 18;
constexpr int kDigits = 3;
constexpr int kPartBase = kDigits * kMaxCols;
constexpr int kMaxBase = kPartBase + 2 * kMaxBlocks * kParts;
constexpr int kTicketSlot = kMaxBase + kMaxBlocks;
constexpr int kScratchWords = kTicketSlot + 31;

static __device__ __align__(256) double g_noalloc_scratch[kScratchWords];

// ---- device address of g_noalloc_scratch, looked up once per CUDA context.
// The key is the context's unique id (cuCtxGetId), so a context created after
// cudaDeviceReset, or a caller's own non-primary context, gets its own lookup
// instead of a stale address.  The driver functions come through the runtime's
// entry-point query, so the library needs no link against libcuda.
using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

std::mutex g_mu;
constexpr int kCacheSlots = 64;
unsigned long long g_ctx_id[kCacheSlots] = {};
double* g_addr[kCacheSlots] = {};
int g_used = 0;
CtxGetCurrentFn g_get_current = nullptr;
CtxGetIdFn g_get_id = nullptr;
bool g_fns_tried = false;

// Id of the calling thread's current context; false when none is current or the
// driver query is unavailable.
bool current_ctx_id(unsigned long long* id) {
    if (!g_fns_tried) {
        g_fns_tried = true;
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_get_current = reinterpret_cast<CtxGetCurrentFn>(f);
        f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_get_id = reinterpret_cast<CtxGetIdFn>(f);
        cudaGetLastError();
    }
    if (!g_get_current || !g_get_id) return false;
    CUcontext ctx = nullptr;
    if (g_get_current(&ctx) != CUDA_SUCCESS || !ctx) return false;
    return g_get_id(ctx, id) == CUDA_SUCCESS;
}

int scratch_address(double** out) {
    std::lock_guard<std::mutex> lk(g_mu);
    unsigned long long id = 0;
    bool have_id = current_ctx_id(&id);
    if (have_id)
        for (int i = 0; i < g_used; ++i)
            if (g_ctx_id[i] == id) {
                *out = g_addr[i];
                return SPS_OK;
            }
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
        cudaGetLastError();
        sps::set_create_error(std::string("cudaGetSymbolAddress(g_noalloc_scratch): ") + cudaGetErrorString(e));
        return SPS_ERR_CUDA;
    }
    if (!have_id) have_id = current_ctx_id(&id);   // the lookup above made the primary context current
    if (have_id && g_used < kCacheSlots) {
        g_ctx_id[g_used] = id;
        g_addr[g_used] = static_cast<double*>(p);
        ++g_used;
    }
    *out = static_cast<double*>(p);
    return SPS_OK;
}

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums of N values over the block in a fixed order, into out[0, N) (a thread per
// value adds the warps; FP64 additions are 62 cycles each on this GPU).  Ends
// with a barrier.
template <int N>
__device__ __forceinline__ void block_total(double (&v)[N], double* out) {
    __shared__ double sm[kThreads / 32][N];
    long long any = 0;             // a warp without values writes its zeros at once
#pragma unroll
    for (int q = 0; q < N; ++q) any |= __double_as_longlong(v[q]);
    if (__any_sync(0xffffffffu, any != 0))
#pragma unroll
        for (int q = 0; q < N; ++q) v[q] = warp_sum(v[q]);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int q = 0; q < N; ++q) sm[threadIdx.x >> 5][q] = v[q];
    __syncthreads();
    if (threadIdx.x < N) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w) s += sm[w][threadIdx.x];
        out[threadIdx.x] = s;
    }
    __syncthreads();
}

__device__ __forceinline__ unsigned long long block_max(unsigned long long v) {
    __shared__ unsigned long long sm[kThreads / 32];
    for (int o = 16; o > 0; o >>= 1) v = max(v, (unsigned long long)__shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
    __syncthreads();
    v = sm[0];
#pragma unroll
    for (int w = 1; w < kThreads / 32; ++w) v = max(v, sm[w]);
    return v;
}

// Grid of the digits: e0 = exponent with max|a_ij y_i| < 2^e0, b bits per digit.
struct Grid {
    int e0, b;
    bool finite;
};

// All threads of the block; max_blocks: the blocks of the first pass.
__device__ __forceinline__ Grid grid_of(const sps_device_lp& lp, const double* s, int max_blocks) {
    const int m = lp.m_ub + lp.m_eq;
    const long long nnz = m > 0 ? (long long)max(lp.indptr[m], 0) : 0ll;
    unsigned long long bits = 0ull;
    for (int b = threadIdx.x; b < max_blocks; b += kThreads)
        bits = max(bits, __ldcg(reinterpret_cast<const unsigned long long*>(s + kMaxBase) + b));
    bits = block_max(bits);
    Grid g;
    g.finite = bits < 0x7FF0000000000000ull;
    const int ex = (int)(bits >> 52);                 // biased exponent of the largest |product|
    g.e0 = (ex == 0 ? -1022 : ex - 1022);             // 2^(e0-1) <= max < 2^e0 (subnormals: 2^-1022)
    int lg = 0;
    while ((1ll << lg) <= nnz && lg < 62) ++lg;       // ceil(log2(nnz + 1))
    g.b = max(8, 51 - lg);
    return g;
}

// Rows of a warp: 32 / Lanes at a time (8, 16 or 32 lanes each: see row_lanes; most
// rows hold a few dozen nonzeros: a warp per row left its lanes idle and its next row's
// offsets one round trip away), rows of over kLongRow nonzeros by the whole warp after
// them.  visit(i, k, end, lanes) runs the lane's share of row i: nonzeros k, k + lanes,
// ...; done(i, row, lanes) ends it, in all of the row's lanes.
constexpr int kRowLanes = 8;
constexpr int kLongRow = 256;
template <int Lanes, class Visit, class Done>
__device__ __forceinline__ void rows_of_warp(const int32_t* __restrict__ ptr, int m, const Visit& visit, const Done& done) {
    constexpr int per = 32 / Lanes;
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * kThreads) >> 5;
    for (int i0 = ((blockIdx.x * kThreads + threadIdx.x) >> 5) * per; i0 < m; i0 += warps * per) {
        const int i = i0 + lane / Lanes;
        const int b = i < m ? ptr[i] : 0, e = i < m ? ptr[i + 1] : 0;
        const bool lng = Lanes < 32 && e - b > kLongRow;
        if (!lng) visit(i, b + (lane & (Lanes - 1)), e, Lanes);
        unsigned todo = __ballot_sync(0xffffffffu, lng && (lane & (Lanes - 1)) == 0);
        done(i, i < m && !lng, Lanes);
        while (todo) {                              // warp-uniform
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const int il = __shfl_sync(0xffffffffu, i, src);
            const int bl = __shfl_sync(0xffffffffu, b, src), el = __shfl_sync(0xffffffffu, e, src);
            visit(il, bl + lane, el, 32);
            done(il, true, 32);
        }
    }
}

// Pass 1: largest |a_ij y_i| (as bits: non-negative doubles order like their bit
// patterns, so an integer max is order-independent), one per block; clears the
// columns' accumulators for pass 2 and the ticket of pass 3.
template <int Lanes>
__global__ void __launch_bounds__(kThreads) na_max(sps_device_lp lp, const double* __restrict__ y,
                                                     double* __restrict__ s) {
    const int m = lp.m_ub + lp.m_eq;
    for (int j = blockIdx.x * kThreads + threadIdx.x; j < lp.n; j += gridDim.x * kThreads)
#pragma unroll
        for (int d = 0; d < kDigits; ++d) s[(size_t)d * kMaxCols + j] = 0.0;
    unsigned long long mx = 0ull;
    const double* __restrict__ val = lp.values;
    rows_of_warp<Lanes>(lp.indptr, m,
        [&](int i, int k, int e, int lanes) {
            if (k >= e) return;
            const double yi = y[i];
#pragma unroll 4
            for (; k < e; k += lanes) {
                const double p = fabs(val[k] * yi);
                const unsigned long long pb = isnan(p) ? 0x7FF8000000000000ull : __double_as_longlong(p);
                mx = max(mx, pb);
            }
        },
        [](int, bool, int) {});
    mx = block_max(mx);
    if (threadIdx.x != 0) return;
    reinterpret_cast<unsigned long long*>(s + kMaxBase)[blockIdx.x] = mx;
    if (blockIdx.x == 0) *reinterpret_cast<unsigned int*>(s + kTicketSlot) = 0u;
}

// Pass 2: residual of K x against the rhs (<= rows count only violations),
// rhs^T y, ||rhs||^2, sign violations of y on <= rows, and the digits of every
// product a_ij y_i added into column j's accumulators.  The digits are cut from
// the product's mantissa with integer shifts (as magnitudes, with the
// product's sign): cut with FP64 scalings and conversions, about twenty
// operations of the FP64 pipe per nonzero, this pass took 217 us on 1.5M
// nonzeros; with two left, 49 us (the 64-bit atomics, up to three per nonzero,
// are what is left).  The whole call: 60k x 150k, 1.5M nonzeros 578 -> 105 us,
// 5k x 12k 183 -> 35 us, 300 x 700 48 -> 31 us.
template <int Lanes>
__global__ void __launch_bounds__(kThreads) na_rows(sps_device_lp lp, const double* __restrict__ x,
                                                     const double* __restrict__ y, double* __restrict__ s, int max_blocks) {
    double v[kParts] = {0.0, 0.0, 0.0, 0.0};
    const int m = lp.m_ub + lp.m_eq;
    const int lane = threadIdx.x & 31;
    const Grid g = grid_of(lp, s, max_blocks);
    unsigned long long* acc = reinterpret_cast<unsigned long long*>(s);
    const int unit = g.e0 - kDigits * g.b;                 // the finest grid's exponent
    const unsigned long long mask = (1ull << g.b) - 1ull;
    const double* __restrict__ val = lp.values;
    const int32_t* __restrict__ idx = lp.indices;
    double sum = 0.0;
    rows_of_warp<Lanes>(lp.indptr, m,
        [&](int i, int k, int e, int lanes) {
            if (k >= e) return;
            const double yi = y[i];
#pragma unroll 2
            for (; k < e; k += lanes) {
                const double a = val[k];
                const int j = idx[k];
                sum += a * x[j];
                if (!g.finite) continue;
                const unsigned long long bits = __double_as_longlong(a * yi);
                const int ex = (int)(bits >> 52) & 0x7ff;
                unsigned long long mant = bits & 0xfffffffffffffull;
                if (ex) mant |= 1ull << 52;
                int sh = (ex ? ex - 1075 : -1074) - unit;  // the product is mant 2^sh finest units
                if (sh < 0) {                              // only the last digit rounds (to nearest)
                    mant = sh < -53 ? 0ull : ((mant >> (-sh - 1)) + 1ull) >> 1;
                    sh = 0;
                }
                const bool neg = (long long)bits < 0;
#pragma unroll
                for (int d = 0; d < kDigits; ++d) {
                    const int r = (kDigits - 1 - d) * g.b - sh;   // the digit's place in mant
                    const unsigned long long q = (r > 63 ? 0ull : r >= 0 ? mant >> r : -r > 63 ? 0ull : mant << -r) &
                                                 (d == 0 ? ~0ull : mask);
                    if (q) atomicAdd(acc + (size_t)d * kMaxCols + j, neg ? 0ull - q : q);
                }
            }
        },
        [&](int i, bool row, int lanes) {
            double t = sum;
            sum = 0.0;
            for (int o = lanes / 2; o >= kRowLanes; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
#pragma unroll
            for (int o = kRowLanes / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (!row || (lane & (lanes - 1)) != 0) return;
            const double b = lp.rhs[i], yi = y[i];
            double res = t - b;
            double sign = 0.0;
            if (i < lp.m_ub) {
                res = fmax(res, 0.0);
                sign = fmax(yi, 0.0);
            }
            v[0] += res * res;
            v[1] += b * yi;
            v[2] += b * b;
            v[3] += sign * sign;
        });
    block_total(v, s + kPartBase + blockIdx.x * kParts);
}

// 2^e as a factor; scalbn where that is no normal number.
__device__ __forceinline__ double scaled(double v, int e) {
    return e >= -1022 && e <= 1023 ? v * __hiloint2double((e + 1023) << 20, 0) : scalbn(v, e);
}

// Pass 3, one thread per column, and the final reduction in the last block.
// out: rel_kkt, rel_primal, rel_dual, rel_gap, primal objective, dual objective.
__global__ void __launch_bounds__(kThreads) na_cols(sps_device_lp lp, const double* __restrict__ x,
                                                     double* __restrict__ s, int row_blocks, int max_blocks,
                                                     double* __restrict__ out) {
    double v[kParts] = {0.0, 0.0, 0.0, 0.0};
    const Grid g = grid_of(lp, s, max_blocks);
    const long long* acc = reinterpret_cast<const long long*>(s);
    for (int j = blockIdx.x * kThreads + threadIdx.x; j < lp.n; j += gridDim.x * kThreads) {
        const double cj = lp.c[j], lo = lp.lb[j], hi = lp.ub[j];
        const bool hl = isfinite(lo), hh = isfinite(hi);
        double aty = 0.0;      // coarse digit first: two roundings in a fixed order
        for (int d = 0; d < kDigits; ++d) aty += scaled((double)acc[(size_t)d * kMaxCols + j], g.e0 - (d + 1) * g.b);
        if (!g.finite) aty = NAN;
        const double r = cj - aty;
        const double lam = (hl && hh) ? r : hl ? fmax(r, 0.0) : hh ? fmin(r, 0.0) : 0.0;
        const double d = r - lam;
        v[0] += d * d;
        v[1] += cj * x[j];
        v[2] += (hl ? lo * fmax(lam, 0.0) : 0.0) + (hh ? hi * fmin(lam, 0.0) : 0.0);
        v[3] += cj * cj;
    }
    block_total(v, s + kPartBase + (kMaxBlocks + blockIdx.x) * kParts);
    __shared__ bool last;
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned int* ticket = reinterpret_cast<unsigned int*>(s + kTicketSlot);
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    // both passes' block partials: thread t adds blocks t, t + 256, ... of each, then the
    // block's fixed tree (one thread took them one by one, an L2 round trip each:
    // 0.4 of the 0.58 ms of a call on 1.5M nonzeros)
    double w[2 * kParts] = {};
    for (int b = threadIdx.x; b < row_blocks; b += kThreads)
        for (int q = 0; q < kParts; ++q) w[q] += __ldcg(s + kPartBase + b * kParts + q);
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kThreads)
        for (int q = 0; q < kParts; ++q) w[kParts + q] += __ldcg(s + kPartBase + kMaxBlocks * kParts + b * kParts + q);
    __shared__ double fin[2 * kParts];
    block_total(w, fin);
    if (threadIdx.x != 0) return;
    const double *R = fin, *Cc = fin + kParts;
    const double rp = sqrt(R[0]) / (1.0 + sqrt(R[2]));
    const double rd = sqrt(Cc[0] + R[3]) / (1.0 + sqrt(Cc[3]));
    const double po = Cc[1], dob = R[1] + Cc[2];
    const double gap = fabs(po - dob) / (1.0 + fabs(po) + fabs(dob));
    out[0] = fmax(rp, fmax(rd, gap));
    out[1] = rp;
    out[2] = rd;
    out[3] = gap;
    out[4] = po;
    out[5] = dob;
}

int blocks_for(int64_t threads) {
    return (int)std::min<int64_t>(kMaxBlocks, std::max<int64_t>(1, (threads + kThreads - 1) / kThreads));
}

// Lanes of a row: 32 while the rows then fill one block per SM, down to 8 (the rows'
// lengths are not known here).  Ten rows of 20 000 nonzeros took 2.00 ms with 8 lanes, four
// rows to a warp, 0.59 with 32; 5000 rows of 20 take 36 us with 8 and 45 with 32.
int row_lanes(int64_t m) {
    int lanes = 32;
    while (lanes > kRowLanes && m * lanes > 152 * kThreads) lanes /= 2;
    return lanes;
}

}  // namespace

extern "C" int sps_kkt_noalloc(const sps_device_lp* lp, const double* x, const double* y, double* out,
                               void* stream) {
    if (!lp || !x || !y || !out) {
        sps::set_create_error("sps_kkt_noalloc: null argument");
        return SPS_ERR_INVALID;
    }
    const int m = lp->m_ub + lp->m_eq;
    if (lp->n < 0 || lp->m_ub < 0 || lp->m_eq < 0) {
        sps::set_create_error("sps_kkt_noalloc: negative dimension");
        return SPS_ERR_INVALID;
    }
    if (lp->n > kMaxCols) {
        sps::set_create_error("sps_kkt_noalloc: n = " + std::to_string(lp->n) +
                              " exceeds the no-allocation limit of 262144 columns");
        return SPS_ERR_INVALID;
    }
    // rows need all four matrix/rhs arrays, even when they hold no nonzeros
    if ((m > 0 && (!lp->indptr || !lp->indices || !lp->values || !lp->rhs)) ||
        (lp->n > 0 && (!lp->c || !lp->lb || !lp->ub))) {
        sps::set_create_error("sps_kkt_noalloc: null device array");
        return SPS_ERR_INVALID;
    }
    double* s = nullptr;
    if (int rc = scratch_address(&s)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int lanes = row_lanes(m);
    const int row_blocks = blocks_for((int64_t)m * lanes), col_blocks = blocks_for(lp->n);
    const int max_blocks = std::max(row_blocks, col_blocks);      // the first pass clears 3 n accumulators too
    const auto largest = lanes == 32 ? na_max<32> : lanes == 16 ? na_max<16> : na_max<8>;
    const auto rows = lanes == 32 ? na_rows<32> : lanes == 16 ? na_rows<16> : na_rows<8>;
    largest<<<max_blocks, kThreads, 0, st>>>(*lp, y, s);
    rows<<<row_blocks, kThreads, 0, st>>>(*lp, x, y, s, max_blocks);
    na_cols<<<col_blocks, kThreads, 0, st>>>(*lp, x, s, row_blocks, max_blocks, out);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        sps::set_create_error(std::string("sps_kkt_noalloc: ") + cudaGetErrorString(e));
        return SPS_ERR_CUDA;
    }
    return SPS_OK;
}
