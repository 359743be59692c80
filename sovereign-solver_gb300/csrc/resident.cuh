// resident.cuh — a whole window of PDHG attempts in one launch, for LPs whose
// matrix fits the shared memory of one thread-block cluster.
//
// What bounds them: nothing moves that HBM or L2 would notice (a 200 x 500 LP
// is 80 KB).  As two launches an attempt took 15-24 us whatever the size:
// launch gaps, the control block's and the gathers' round trips to L2, the last
// block's ticket, and several hundred instructions per thread of schedule
// dispatch around a handful of products.  Here one block, or one cluster of
// blocks, runs every attempt of a window:
//   * the matrix entries a warp needs lie in its block's shared memory, packed
//     in the order it reads them; the vectors the passes gather from (x', y')
//     lie in every block's shared memory;
//   * each lane keeps the state of the rows and columns it owns (at most two of
//     each) in registers for the whole window;
//   * the passes are separated by a block or cluster barrier; new entries and
//     partial sums go to every block through distributed shared memory, and
//     every block adds all partials and takes the step decision itself
//     (decide.cuh), so no decision is broadcast;
//   * one warp of each block owns no rows: it adds the partials and takes the
//     decision (a chain of FP64 divisions, over a thousand cycles at this GPU's
//     FP64 rate) while the others already form K^T y'.
//
// Same numbers as the launched passes, bit for bit: a task is what one warp of
// a launched pass does (Bin, visit_bins: at most two units when every bin has
// the blocks it needs), in that warp's order, and the partial sums are added in
// the launched pass's tree.
#pragma once

#include "kernels.cuh"

namespace sps {

constexpr int kResMaxCluster = 16;
// Threads of a resident block: 512 (128 registers each), or in FP32 1024 where an LP needs them.
constexpr int kResThreads = 512;
template <class V>
constexpr int res_max_threads() { return sizeof(V) == 4 ? 1024 : kResThreads; }

// One warp's share of a pass.  SLICED and SLAB units: lane t owns row r0 + t
// and its entries lie 32 apart; WARP units: one row, its entries dealt to the
// lanes in turn, lane 0 owns the row.
struct ResTask {
    int32_t mode;             // BinMode, -1 = none
    int32_t kind, rend;       // row kind; end of the bin's rows
    int32_t part;             // which partial sum the task's epilogues add up to
    int32_t ent;              // first entry in the block's shared entries (unit 1's follow unit 0's)
    int32_t slab, slab_c, slab_n;   // SLAB: the unit's row of lane partials, its place among the slice's units
    struct Unit {
        int32_t r0, steps;    // first row; entries per lane (-1: no unit)
        int32_t src, cnt;     // entries in the layout: src .. src + cnt (zeros up to 32 * steps)
    } u[2];
};

// The block's shared memory: its entries, y' and the lane partials of SLAB units, and in
// adaptive mode x, the candidate and all partial sums, in reference mode x'.
template <class V>
__host__ __device__ constexpr size_t res_smem_bytes(const ResShape& s, int64_t n, int64_t m, bool adaptive) {
    return (sizeof(V) + 4) * (size_t)s.entries + sizeof(V) * ((size_t)n + m + 32 * (size_t)s.slab_rows) +
           (adaptive ? sizeof(V) * ((size_t)n + 2 * (size_t)s.row_parts + 2 * (size_t)s.col_parts) : 0);
}

__device__ __forceinline__ uint32_t res_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t res_map(uint32_t a, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void res_store(uint32_t a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void res_store(uint32_t a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
// *p = v in the shared memory of every block of the cluster
template <bool Multi, class V>
__device__ __forceinline__ void res_share(V* p, V v, int blocks) {
    if constexpr (!Multi) {
        *p = v;
    } else {
        const uint32_t a = res_addr(p);
        for (int q = 0; q < blocks; ++q) res_store(res_map(a, q), v);
    }
}

// All threads of all blocks: what any of them wrote before it is visible after it.
template <bool Multi>
__device__ __forceinline__ void res_barrier() {
    if constexpr (Multi)
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    else
        __syncthreads();
}

// The block's matrix entries: (index, value) pairs in FP32, two arrays in FP64.
template <class V>
struct ResEntries;
template <>
struct ResEntries<float> {
    int2* e;
    __device__ ResEntries(void* p, int) : e(static_cast<int2*>(p)) {}
    __device__ __forceinline__ void put(int i, int j, float v) { e[i] = make_int2(j, __float_as_int(v)); }
    __device__ __forceinline__ void get(int i, int& j, float& v) const {
        const int2 q = e[i];
        j = q.x;
        v = __int_as_float(q.y);
    }
};
template <>
struct ResEntries<double> {
    double* v_;
    int* j_;
    __device__ ResEntries(void* p, int count) : v_(static_cast<double*>(p)), j_(reinterpret_cast<int*>(v_ + count)) {}
    __device__ __forceinline__ void put(int i, int j, double v) { j_[i] = j; v_[i] = v; }
    __device__ __forceinline__ void get(int i, int& j, double& v) const { j = j_[i]; v = v_[i]; }
};

// What a lane keeps of its warp's task over the window.
struct ResLane {
    int ent = 0, s0 = -1, s1 = -1, part = 0;
    int r[2] = {-1, -1};      // the rows the lane owns (-1: none)
    bool strided = false, kind = false, sums = false;   // WARP units; '<=' rows; the task has epilogues
    __device__ __forceinline__ bool any() const { return s0 >= 0; }
    template <class V>
    __device__ __forceinline__ void load(const ResTask& t, const Layout<V>& L, ResEntries<V>& E) {
        if (t.mode < 0) return;
        const int lane = threadIdx.x & 31;
        ent = t.ent;
        s0 = t.u[0].steps;
        s1 = t.u[1].steps;
        part = t.part;
        strided = t.mode == BM_WARP;
        kind = t.kind != 0;
        sums = t.slab_c == 0;
        int at = t.ent + lane;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (t.u[h].steps < 0) continue;
            const int row = t.u[h].r0 + (strided ? 0 : lane);
            if (sums && (strided ? lane == 0 : row < t.rend)) r[h] = row;
            for (int k = 0; k < t.u[h].steps; ++k, at += 32) {
                const int q = 32 * k + lane;
                const bool ok = q < t.u[h].cnt;
                E.put(at, ok ? __ldg(L.idx + t.u[h].src + q) : 0, ok ? __ldg(L.val + t.u[h].src + q) : V(0));
            }
        }
    }
};

// The lane's dot products of the task's two units with the vector g, four steps
// of each at a time (steps are padded to that unless both units have fewer; the
// padding adds zeros).
template <class V>
__device__ __forceinline__ void res_dots(const ResEntries<V>& E, const ResLane& t, const V* g, V (&acc)[2]) {
    V a0 = V(0), a1 = V(0);
    const int s0 = t.s0, s1 = t.s1;
    int p = t.ent + (threadIdx.x & 31), q = p + 32 * s0;
    int k = 0;
    if (max(s0, s1) < 4) {     // the columns of assignment and transportation LPs
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            int j;
            V v;
            if (u < s0) {
                E.get(p + 32 * u, j, v);
                a0 = mad(v, g[j], a0);
            }
            if (u < s1) {
                E.get(q + 32 * u, j, v);
                a1 = mad(v, g[j], a1);
            }
        }
        k = 4;
    }
    for (; k < min(s0, s1); k += 4, p += 128, q += 128) {
        int j[8];
        V v[8];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            E.get(p + 32 * u, j[u], v[u]);
            E.get(q + 32 * u, j[4 + u], v[4 + u]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            a0 = mad(v[u], g[j[u]], a0);
            a1 = mad(v[4 + u], g[j[4 + u]], a1);
        }
    }
    V rest = s0 > s1 ? a0 : a1;
    int r = s0 > s1 ? p : q;
    for (const int s = max(s0, s1); k < s; k += 4, r += 128) {
        int j[4];
        V v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) E.get(r + 32 * u, j[u], v[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) rest = mad(v[u], g[j[u]], rest);
    }
    if (s0 > s1) a0 = rest;
    else a1 = rest;
    if (t.strided) {
        a0 = group_sum<32>(a0);
        a1 = group_sum<32>(a1);
    }
    acc[0] = a0;
    acc[1] = a1;
}

// SLAB slices of several units: the units' lane partials, added in unit order
// by the slice's first unit (all units of a slice are tasks of one block).
struct ResSlab { int row = 0, n = 0; };        // the unit's row of lane partials; units of its slice (0: no SLAB unit)
template <class V>
__device__ __forceinline__ void res_slab(const ResSlab& t, bool first, V* slab, V& acc) {
    const int lane = threadIdx.x & 31;
    if (t.n > 1) slab[32 * t.row + lane] = acc;
    __syncthreads();
    if (t.n > 1 && first) {
        V s = V(0);
#pragma unroll 4
        for (int w = 0; w < t.n; ++w) s += slab[32 * (t.row + w) + lane];
        acc = s;
    }
}

// One warp: sum over 256 threads, thread t holding the sum of src[t], src[t +
// 256], ... of `count` values: block_sum's tree (a butterfly per warp, then the
// warps in order).  get(i) is value i.
template <int NP, class V, class Get>
__device__ __forceinline__ void res_tree(V (&tot)[NP], int count, const Get& get) {
    const int lane = threadIdx.x & 31;
    if (count <= 32) {         // the other warps add zeros, and lanes past the values too: those steps are left out
#pragma unroll
        for (int p = 0; p < NP; ++p) tot[p] = V(0);
        if (lane < count) get(lane, tot);
        int o = 16;
        while (o >= count) o >>= 1;
        for (; o > 0; o >>= 1)
#pragma unroll
            for (int p = 0; p < NP; ++p) tot[p] += __shfl_xor_sync(0xffffffffu, tot[p], o);
        return;                // lane 0 holds the sum
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) tot[p] = V(0);
    for (int g = 0; g * 32 < count && g < kWarps; ++g) {
        V v[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) v[p] = V(0);
        for (int b = g * 32 + lane; b < count; b += kBlock) get(b, v);
#pragma unroll
        for (int p = 0; p < NP; ++p) tot[p] += group_sum<32>(v[p]);
    }
}

// One warp: a pass's total from the partial sums of its warps (NP each) and its
// SLAB slots, in the order of publish_partials and gather_all_partials.
template <int NP, class V>
__device__ __forceinline__ void res_total(V (&tot)[NP], const V* wp, int warps, int slots) {
    res_tree<NP>(tot, warps / kWarps, [&](int b, V (&v)[NP]) {
        constexpr int N = kWarps * NP, per = 16 / sizeof(V);      // 16-byte reads
        V a[N];
        const int4* src = reinterpret_cast<const int4*>(wp + b * N);
#pragma unroll
        for (int i = 0; i < N / per; ++i) reinterpret_cast<int4*>(a)[i] = src[i];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            V s = V(0);
#pragma unroll
            for (int q = 0; q < kWarps; ++q) s += a[q * NP + p];
            v[p] += s;
        }
    });
    if (slots == 0) return;
    V st[NP];
    res_tree<NP>(st, slots, [&](int b, V (&v)[NP]) {
#pragma unroll
        for (int p = 0; p < NP; ++p) v[p] += wp[(warps + b) * NP + p];
    });
#pragma unroll
    for (int p = 0; p < NP; ++p) tot[p] += st[p];
}

// ---- the step decision ------------------------------------------------------
// decide_step divides three times in a row and compares in FP64: about 3 800
// cycles of one thread (every dependent FP64 operation is 62 cycles on this GPU),
// while every warp waits.  Here it is a chain of ten such operations with the
// same values: what depends on the attempt number alone is formed during the
// row pass, a quotient is a product with a reciprocal corrected once by its
// remainder (Markstein's correction), and whether it is the rounded quotient is checked
// off the chain, by the exact remainder; positive values are compared as integers.  Operands
// outside the ranges this needs, and the quotients the check leaves open, take
// decide_step itself.
__device__ __forceinline__ int64_t res_bits(double v) { return __double_as_longlong(v); }
__device__ __forceinline__ bool res_mid(double v) {       // 2^-300 <= |v| < 2^300
    return ((unsigned)(__double2hiint(v) >> 20) & 0x7ffu) - 723u < 600u;
}
// q is a / b rounded to nearest (q > 0 near it, r = a - q b exactly): the remainder is below half
// a unit in the last place of q times b.  A power of two has a finer grid below it: left open.
__device__ __forceinline__ bool res_rounded(double q, double r, double b) {
    const int h = __double2hiint(q);
    const double half = __hiloint2double(((h >> 20) - 53) << 20, 0);
    return res_mid(q) && ((h & 0xfffff) | __double2loint(q)) != 0 && res_bits(fabs(r)) < res_bits(half * b);
}
// V(a / b) from y = 1 / b rounded to nearest.  In FP32: a y is within two units in the last place
// (of FP64) of the quotient, so it rounds as the quotient does unless it lies that
// near to the middle between two floats.  ok: the value is certain.
__device__ __forceinline__ void res_quot(double a, double, double y, float* out, bool* ok) {
    const double q = a * y;
    const unsigned low = (unsigned)__double2loint(q) & 0x1fffffffu;
    *ok = ((unsigned)(__double2hiint(q) >> 20) & 0x7ffu) - 903u < 240u && low - 0x0ffffffcu > 8u;   // a normal float
    *out = float(q);
}
__device__ __forceinline__ void res_quot(double a, double b, double y, double* out, bool* ok) {
    double q = a * y;
    q = __fma_rn(__fma_rn(-q, b, a), y, q);
    *ok = res_rounded(q, __fma_rn(-q, b, a), b);
    *out = q;
}
__device__ __forceinline__ void res_twice(float v, double* b, float* bf) { *bf = 2.f * fabsf(v); *b = double(*bf); }
__device__ __forceinline__ void res_twice(double v, double* b, float* bf) { *b = 2.0 * fabs(v); *bf = float(*b); }

template <class V>
struct ResDecide {
    double omega_inv, shrink, grow;                // 1 / omega; 1 - (k+1)^-0.3; (1 + (k+1)^-0.6) eta
    double next;
    int acc, usual;
    __device__ __forceinline__ void window(const Ctl& c) { omega_inv = 1.0 / c.omega; }
    __device__ __forceinline__ void ready(const Ctl& c) {
        const float kk = float(c.iters + 2);
        shrink = 1.0 - double(powf(kk, -0.3f));
        grow = (1.0 + double(powf(kk, -0.6f))) * c.eta;
        usual = res_mid(c.omega) && res_mid(c.eta) && res_mid(c.dx2) && res_mid(grow);
    }
    __device__ __forceinline__ void operator()(Ctl& c, V dy2v, V interv, V* tau, V* wgt) {
        const double w = c.omega, eta = c.eta, wi = omega_inv;
        const double dy2 = double(dy2v);
        double b;
        float bf;
        res_twice(interv, &b, &bf);
        if (usual && res_mid(dy2) && (__float_as_uint(bf) >> 23) - 27u < 200u) {      // 2^-100 <= bf < 2^100
            const double y0 = double(__frcp_rn(bf));
            const double y = __fma_rn(y0, __fma_rn(-b, y0, 1.0), y0);         // 1 / b to about 2^-46
            double d = dy2 * wi;
            d = __fma_rn(__fma_rn(-d, w, dy2), wi, d);
            const double move = __fma_rn(w, c.dx2, d);
            double q = move * y;
            q = __fma_rn(__fma_rn(-q, b, move), y, q);
            const double a0 = shrink * q;
            const double nx = res_bits(a0) < res_bits(grow) ? a0 : grow;
            bool sure;
            res_quot(nx, w, wi, tau, &sure);
            if (sure && res_mid(nx) && res_rounded(d, __fma_rn(-d, w, dy2), w) &&
                res_rounded(q, __fma_rn(-q, b, move), b)) {
                next = nx;
                acc = res_bits(eta) <= res_bits(q);
                *wgt = V(acc ? eta : c.eta_used);
                return;
            }
        }
        usual = 0;
        decide_step(c, dy2, double(interv));
        next = c.eta;
        acc = c.accepted;
        *tau = V(c.eta / w);
        *wgt = V(c.eta_used);
    }
    // the rest of decide_step, after the other warps have their step sizes
    __device__ __forceinline__ void record(Ctl& c) const {
        if (usual) {
            c.iters += 1;
            c.window += 1;
            c.accepted = acc;
            if (acc) {
                c.cur = 1 - c.cur;
                c.eta_used = c.eta;
                c.w_sum += c.eta;
                c.accepted_total += 1;
            }
            c.eta = next;
        }
        c.apply = 0;
    }
};

// The attempts of one window (check_interval of them, fewer when the solve ends).
// 200 x 500 on one block: 195 us for 64 attempts, 7.2 cycles per issued instruction at
// barriers, 2.7 on shared memory.  The 1024-thread form has 64 registers and spills
// 104-112 bytes.
template <class V, bool Multi, int Threads>
__global__ void __launch_bounds__(Threads, 1) ad_resident(const __grid_constant__ Args<V> a) {
    extern __shared__ __align__(16) unsigned char res_buf[];
    __shared__ Ctl c;
    __shared__ V s_sigma, s_tau, s_wgt;
    __shared__ int s_acc, s_done;
    __shared__ ResDecide<V> decide;                // the deciding thread's
    const ResShape& S = a.res;
    const int blocks = Multi ? S.blocks : 1, rank = Multi ? (int)blockIdx.x : 0;
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool control = wid == S.warps;
    ResEntries<V> E(res_buf, S.entries);
    V* wr = reinterpret_cast<V*>(res_buf + (sizeof(V) + 4) * (size_t)S.entries);   // row pass: dy2, inter per warp, then per SLAB slice
    V* wc = wr + 2 * S.row_parts;                  // column pass: dx2 per warp
    V* wj = wc + S.col_parts;                      // rejected attempt: dx2 per warp
    V* xb = wj + S.col_parts;                      // x and the candidate
    V* sy = xb + 2 * (size_t)a.n;
    V* slab = sy + a.m;
    const int row_slots = a.csr.nsegrows;
    if (threadIdx.x == 0) {
        c = *a.ctl;
        s_sigma = V(c.eta * c.omega);
        s_done = c.done || c.iters >= c.max_iters;
    }
    __syncthreads();
    if (s_done) return;                            // every block reads the same
    int cur = c.cur;
    const int64_t left = c.max_iters - c.iters;
    const int W = (int)(left < a.check_interval ? left : a.check_interval);
    for (int j = threadIdx.x; j < a.n; j += blockDim.x) {
        xb[j] = a.X[0][j];
        xb[a.n + j] = a.X[1][j];
    }
    for (int i = threadIdx.x; i < 2 * S.row_parts + 2 * S.col_parts; i += blockDim.x) wr[i] = V(0);
    ResLane rt, ct;
    ResSlab rs;
    if (!control) {
        const ResTask& t = a.res_rows[rank * S.warps + wid];
        rt.load(t, a.csr, E);
        if (t.mode == BM_SLAB) rs = ResSlab{t.slab, t.slab_n};
        ct.load(a.res_cols[rank * S.warps + wid], a.csc, E);
    }
    V ax[2], y[2], b[2], ys[2], yl[2], x[2], cand[2], cc[2], lo[2], hi[2], xs[2], xl[2], aty[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (rt.r[h] >= 0) {
            const int r = rt.r[h];
            ax[h] = a.AX[cur][r];
            y[h] = a.Y[cur][r];
            b[h] = a.b[r];
            ys[h] = a.ys[r];
            yl[h] = a.yl[r];
        }
        if (ct.r[h] >= 0) {
            const int j = ct.r[h];
            x[h] = a.X[cur][j];
            cand[h] = a.X[1 - cur][j];
            cc[h] = a.c[j];
            lo[h] = lo_at(a, j);
            hi[h] = hi_at(a, j);
            xs[h] = a.xs[j];
            xl[h] = a.xl[j];
            aty[h] = a.ATY[cur][j];
        }
    }
    if (control && lane == 0) decide.window(c);
    res_barrier<Multi>();
    bool rejected = false;                         // the last column pass took the rejected branch
    int w = 0;
    for (; w < W; ++w) {
        // row pass: K x', y' = proj(y + sigma (b - (2 K x' - K x))), as AdRowStepEpi
        V axn[2], yn[2];
        if (control) {
            if (w > 0) {                           // the candidate's movement, from the last column pass
                V d[1];
                res_total<1>(d, rejected ? wj : wc, S.col_parts, 0);
                if (lane == 0) c.dx2 = double(d[0]);
            }
            if (lane == 0) decide.ready(c);
            if (S.slab_rows) __syncthreads();
        } else {
            if (rt.any()) res_dots(E, rt, xb + (size_t)(1 - cur) * a.n, axn);
            if (S.slab_rows) res_slab(rs, rt.sums, slab, axn[0]);
            if (rt.sums) {
                const V sigma = s_sigma;
                V dy2 = V(0), inter = V(0);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (rt.r[h] >= 0) {
                        V y2 = mad(sigma, b[h] - (axn[h] + axn[h] - ax[h]), y[h]);
                        if (rt.kind) y2 = fmin(y2, V(0));
                        yn[h] = y2;
                        res_share<Multi>(sy + rt.r[h], y2, blocks);
                        const V dy = y2 - y[h];
                        dy2 = mad(dy, dy, dy2);
                        inter = mad(dy, axn[h] - ax[h], inter);
                    }
                dy2 = group_sum<32>(dy2);
                inter = group_sum<32>(inter);
                if (lane == 0) {
                    res_share<Multi>(wr + 2 * rt.part, dy2, blocks);
                    res_share<Multi>(wr + 2 * rt.part + 1, inter, blocks);
                }
            }
        }
        res_barrier<Multi>();
        V g[2];
        if (control) {
            V t[2];
            res_total<2>(t, wr, S.row_warps, row_slots);
            if (lane == 0) {
                V tau, wgt;
                decide(c, t[0], t[1], &tau, &wgt);
                s_acc = decide.acc;
                s_done = c.done;
                s_tau = tau;
                s_wgt = wgt;
            }
        } else if (ct.any()) {
            res_dots(E, ct, sy, g);
        }
        __syncthreads();
        if (s_done) break;
        const V tau = s_tau, wgt = s_wgt;
        rejected = !s_acc;
        if (control && lane == 0) {
            decide.record(c);
            s_sigma = V(c.eta * c.omega);
        }
        if (s_acc) {
            cur ^= 1;
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (rt.r[h] >= 0) {
                    ax[h] = axn[h];
                    y[h] = yn[h];
                    ys[h] = mad(wgt, yn[h] - yl[h], ys[h]);
                }
            if (ct.any()) {
                V dx2 = V(0);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (ct.r[h] >= 0) {
                        aty[h] = g[h];
                        x[h] = cand[h];
                        xs[h] = mad(wgt, x[h] - xl[h], xs[h]);
                        cand[h] = clampv(mad(-tau, cc[h] - g[h], x[h]), lo[h], hi[h]);
                        res_share<Multi>(xb + (size_t)(1 - cur) * a.n + ct.r[h], cand[h], blocks);
                        const V d = cand[h] - x[h];
                        dx2 = mad(d, d, dx2);
                    }
                dx2 = group_sum<32>(dx2);
                if (lane == 0) res_share<Multi>(wc + ct.part, dx2, blocks);
            }
        } else {
            // the candidate again with the smaller step; its movement is summed in the
            // launched pass's order for this case (columns dealt to the pass's threads)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (ct.r[h] >= 0) {
                    cand[h] = clampv(mad(-tau, cc[h] - aty[h], x[h]), lo[h], hi[h]);
                    res_share<Multi>(xb + (size_t)(1 - cur) * a.n + ct.r[h], cand[h], blocks);
                }
            res_barrier<Multi>();
            const V *xc = xb + (size_t)cur * a.n, *xn = xb + (size_t)(1 - cur) * a.n;
            for (int p = rank + blocks * wid; p < S.col_parts; p += blocks * (S.warps + 1)) {
                V dx2 = V(0);
                for (int j = 32 * p + lane; j < a.n; j += 32 * S.col_parts) {
                    const V d = xn[j] - xc[j];
                    dx2 = mad(d, d, dx2);
                }
                dx2 = group_sum<32>(dx2);
                if (lane == 0) res_share<Multi>(wj + p, dx2, blocks);
            }
        }
        res_barrier<Multi>();
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (rt.r[h] >= 0) {
            const int r = rt.r[h];
            a.AX[cur][r] = ax[h];
            a.Y[cur][r] = y[h];
            a.ys[r] = ys[h];
        }
        if (ct.r[h] >= 0) {
            const int j = ct.r[h];
            a.X[cur][j] = x[h];
            a.X[1 - cur][j] = cand[h];
            a.ATY[cur][j] = aty[h];
            a.xs[j] = xs[h];
        }
    }
    if (rank == 0 && control) {
        if (w > 0 && !s_done) {
            V d[1];
            res_total<1>(d, rejected ? wj : wc, S.col_parts, 0);
            if (lane == 0) c.dx2 = double(d[0]);
        }
        if (lane == 0) *a.ctl = c;
    }
}

// Reference mode: the iterations of one window (RfColStepEpi, RfRowStepEpi; no
// sums, so every warp works).
template <class V, bool Multi, int Threads>
__global__ void __launch_bounds__(Threads, 1) rf_resident(const __grid_constant__ Args<V> a) {
    extern __shared__ __align__(16) unsigned char res_buf[];
    const ResShape& S = a.res;
    const int blocks = Multi ? S.blocks : 1, rank = Multi ? (int)blockIdx.x : 0;
    const int wid = threadIdx.x >> 5;
    ResEntries<V> E(res_buf, S.entries);
    V* sx = reinterpret_cast<V*>(res_buf + (sizeof(V) + 4) * (size_t)S.entries);
    V* sy = sx + a.n;
    V* slab = sy + a.m;
    Ctl* ctl = a.ctl;
    const int64_t iters = ctl->iters, left = ctl->max_iters - iters;
    if (ctl->done || left <= 0) return;                    // every block reads the same
    const int W = (int)(left < a.check_interval ? left : a.check_interval);
    ResLane rt, ct;
    ResSlab rs;
    {
        const ResTask& t = a.res_rows[rank * S.warps + wid];
        rt.load(t, a.csr, E);
        if (t.mode == BM_SLAB) rs = ResSlab{t.slab, t.slab_n};
        ct.load(a.res_cols[rank * S.warps + wid], a.csc, E);
    }
    for (int i = threadIdx.x; i < a.m; i += blockDim.x) sy[i] = a.Y[0][i];
    V x[2], xs[2], xbar[2], tau[2], cc[2], y[2], ys[2], sg[2], b[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (rt.r[h] >= 0) {
            const int r = rt.r[h];
            y[h] = a.Y[0][r];
            ys[h] = a.ys[r];
            sg[h] = a.sigma[r];
            b[h] = a.b[r];
        }
        if (ct.r[h] >= 0) {
            const int j = ct.r[h];
            x[h] = a.X[0][j];
            xs[h] = a.xs[j];
            tau[h] = a.tau[j];
            cc[h] = a.c[j];
        }
    }
    res_barrier<Multi>();
    for (int w = 0; w < W; ++w) {
        V g[2];
        if (ct.any()) {
            res_dots(E, ct, sy, g);
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (ct.r[h] >= 0) {
                    V x2 = rn_sub(x[h], rn_mul(tau[h], rn_sub(cc[h], g[h])));
                    x2 = fmax(x2, V(0));
                    xbar[h] = rn_sub(rn_mul(V(2), x2), x[h]);
                    res_share<Multi>(sx + ct.r[h], xbar[h], blocks);
                    x[h] = x2;
                    xs[h] = rn_add(xs[h], x2);
                }
        }
        res_barrier<Multi>();
        if (rt.any()) res_dots(E, rt, sx, g);
        if (S.slab_rows) res_slab(rs, rt.sums, slab, g[0]);
        if (rt.sums) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (rt.r[h] >= 0) {
                    y[h] = rn_add(y[h], rn_mul(sg[h], rn_sub(b[h], g[h])));
                    res_share<Multi>(sy + rt.r[h], y[h], blocks);
                    ys[h] = rn_add(ys[h], y[h]);
                }
        }
        res_barrier<Multi>();
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (rt.r[h] >= 0) {
            const int r = rt.r[h];
            a.Y[0][r] = y[h];
            a.ys[r] = ys[h];
        }
        if (ct.r[h] >= 0) {
            const int j = ct.r[h];
            a.X[0][j] = x[h];
            a.xs[j] = xs[h];
            a.xbar[j] = xbar[h];
        }
    }
    if (rank == 0 && threadIdx.x == 0) {
        ctl->iters = iters + W;
        ctl->window += W;
    }
}

}  // namespace sps
