// Test helper (host code only, no GPU needed): the batch's device memory
// (sovereign-solver_gb300/csrc/batch.cu) on a device of a given size, for
// tests/test_batch_memory.py.  The runtime calls of the host code are replaced by
// stand-ins over host memory.  It runs on the CPU alone: no device may be visible, so that
// the launches among the host code do nothing (it ends at once where one is).  Every
// check prints one line; the exit status is 0 when all hold.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

// (the runtime's own, before its names are replaced)
static bool device_visible() {
    int n = 0;
    return cudaGetDeviceCount(&n) == cudaSuccess && n > 0;
}

static size_t g_size = 0, g_used = 0;
static std::map<void*, size_t> g_held;
static int32_t g_steps = 0;                     // what the counting launch says of every chunk's end
static cudaError_t t_malloc(void** p, size_t bytes) {
    if (bytes > g_size - g_used) return cudaErrorMemoryAllocation;
    *p = aligned_alloc(256, (bytes + 255) / 256 * 256);
    g_held[*p] = bytes;
    g_used += bytes;
    return cudaSuccess;
}
template <class T>
static cudaError_t t_malloc(T** p, size_t bytes) { return t_malloc(reinterpret_cast<void**>(p), bytes); }
static cudaError_t t_free(void* p) {
    if (!p) return cudaSuccess;
    if (!g_held.count(p)) { printf("freed twice\n"); exit(1); }
    g_used -= g_held[p];
    g_held.erase(p);
    free(p);
    return cudaSuccess;
}
static bool held(const void* p, size_t bytes) {  // [p, p + bytes) lies in one allocation
    auto it = g_held.upper_bound(const_cast<void*>(p));
    if (it == g_held.begin()) return false;
    --it;
    return (const char*)p + bytes <= (const char*)it->first + it->second;
}
static cudaError_t t_copy(void* d, const void* s, size_t bytes, cudaMemcpyKind kind, cudaStream_t) {
    if (kind == cudaMemcpyDeviceToHost) {
        for (size_t i = 0; i < bytes / 4; ++i) static_cast<int32_t*>(d)[i] = g_steps;
        return cudaSuccess;
    }
    if (!held(d, bytes)) { printf("copied outside an allocation\n"); exit(1); }
    memcpy(d, s, bytes);
    return cudaSuccess;
}
static cudaError_t t_set(void* d, int v, size_t bytes, cudaStream_t) {
    if (!held(d, bytes)) { printf("set outside an allocation\n"); exit(1); }
    memset(d, v, bytes);
    return cudaSuccess;
}
static cudaError_t t_info(size_t* free_bytes, size_t* total) {
    *free_bytes = g_size - g_used;
    *total = g_size;
    return cudaSuccess;
}
static cudaError_t t_attribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
static cudaError_t t_clusters(int* n) { *n = 16; return cudaSuccess; }
static cudaError_t t_occupancy(int* n) { *n = 2; return cudaSuccess; }

#define cudaMalloc(p, n) t_malloc(p, n)
#define cudaFree(p) t_free(p)
#define cudaMemcpyAsync(d, s, n, k, st) t_copy(d, s, n, k, st)
#define cudaMemsetAsync(d, v, n, st) t_set(d, v, n, st)
#define cudaMemGetInfo(f, t) t_info(f, t)
#define cudaSetDevice(d) cudaSuccess
#define cudaGetLastError() cudaSuccess
#define cudaStreamSynchronize(s) cudaSuccess
#define cudaDeviceGetAttribute(v, a, d) t_attribute(v, a, d)
#define cudaFuncSetAttribute(...) cudaSuccess
#define cudaOccupancyMaxActiveClusters(n, ...) t_clusters(n)
#define cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, ...) t_occupancy(n)
#include "batch.cu"

// what the other translation units have: an engine that needs g_engine bytes
static size_t g_engine = 0;
static int g_creates = 0;
extern "C" {
int sps_options_init(sps_options*) { return SPS_OK; }
int sps_create(const sps_problem_desc*, const sps_options*, sps_handle**) {
    ++g_creates;
    return g_engine > g_size - g_used ? SPS_ERR_OOM : SPS_OK;
}
int sps_set_warm_start(sps_handle*, const double*, const double*, double) { return SPS_OK; }
int sps_solve(sps_handle*, sps_result* r) { *r = sps_result{}; return SPS_OK; }
int sps_get_solution(sps_handle*, double*, double*) { return SPS_OK; }
const char* sps_last_error(const sps_handle*) { return "out of memory"; }
void sps_destroy(sps_handle*) {}
const char* sps_gnn_last_error(const sps_gnn*) { return ""; }
}
namespace sps {
void set_create_error(const std::string&) {}
namespace gnn {
int device_io(sps_gnn*, DeviceIO*) { return -1; }
int forward_in_place(sps_gnn*, int) { return -1; }
int check_device_error(sps_gnn*) { return -1; }
}  // namespace gnn
}  // namespace sps

constexpr int kCount = 3, kN = 2000, kM = 1000, kNnz = 8192, kSteps = 100;
constexpr size_t kSliceBytes = size_t(2 * kCount * kSteps) * 1024 + size_t(kCount * (kN + kM)) * 16;
constexpr size_t kWarmBytes = size_t(kCount * (kN + kM) + kCount) * 8;
constexpr size_t kTables = 64 << 10;             // more than the slices' tables take

static void fill(sps_batch& b) {
    b.count = kCount;
    b.G = b.Gr = 8;
    b.blocks = kCount;
    b.opt.mode = SPS_MODE_ADAPTIVE;
    b.sum_n = kCount * kN;
    b.sum_m = kCount * kM;
    b.inst.resize(kCount);
    for (Inst& I : b.inst) {
        I = Inst{};
        I.n = kN;
        I.m = I.m_ub = kM;
        I.nnz = kNnz;
    }
    g_steps = kSteps;
}
static bool check(const char* name, bool ok) {
    printf("%s %s\n", name, ok ? "ok" : "FAILED");
    return ok;
}

int main() {
    setenv("CUDA_VISIBLE_DEVICES", "", 1);
    if (device_visible()) {
        printf("a device is visible: its kernels would be given host memory\n");
        return 1;
    }
    bool all = true;
    const std::vector<double> x(kCount * kN, 0.5), y(kCount * kM, 0.5);
    {   // room for the slices, then none for the warm starts beside them
        sps_batch b;
        fill(b);
        g_size = 2 * kSliceBytes + kTables;
        all &= check("slices made", build_slices(&b) == SPS_OK && b.arr.slice && held(b.arr.pts, 16 * (b.sum_n + b.sum_m)));
        g_size = g_used + kWarmBytes / 2;
        all &= check("warm starts take the slices' memory",
                     sps_batch_set_warm_starts(&b, x.data(), y.data(), nullptr) == SPS_OK && !b.arr.slice && !b.arr.steps &&
                         !b.arr.pts && !b.arr.soff && b.warm == 1 && g_used == kWarmBytes);
        all &= check("nothing left to release", !b.release_slices());
    }
    {   // slices that would take more than half of what is free are not made, and leave nothing behind
        sps_batch b;
        fill(b);
        g_size = kSliceBytes + kTables;
        all &= check("half of the free memory", build_slices(&b) == SPS_OK && !b.arr.slice && g_used == 0);
        g_size = kTables / 1024;
        all &= check("no memory for the tables", build_slices(&b) == SPS_OK && !b.arr.slice && g_used == 0);
    }
    {   // no room for the warm starts at all: refused each time, and nothing is half there
        sps_batch b;
        fill(b);
        g_size = kWarmBytes - 8;
        for (int k = 0; k < 2; ++k)
            all &= check("warm starts refused", sps_batch_set_warm_starts(&b, x.data(), y.data(), nullptr) == SPS_ERR_OOM &&
                                                    !b.d_wx && !b.d_wy && b.warm == 0 && g_used == 0);
    }
    {   // a continuation that does not fit beside the slices
        sps_batch b;
        fill(b);
        g_size = 2 * kSliceBytes + kTables;
        all &= build_slices(&b) == SPS_OK && b.arr.slice;
        b.out.assign(kCount, Ctl{});
        b.opt.max_iters = 10;
        b.h_rptr = HostBuf<int32_t>(kM + 1);
        std::memset(b.h_rptr.data(), 0, sizeof(int32_t) * (kM + 1));
        b.escalated.assign(kCount, 0);
        b.handed_off.assign(kCount, 0);
        b.xo.resize(b.sum_n);
        b.yo.resize(b.sum_m);
        g_engine = g_size - g_used + 1;
        std::string why;
        all &= check("continuation takes the slices' memory",
                     continue_single(&b, 0, 0.0, &why) == SPS_OK && g_creates == 2 && !b.arr.slice && g_used == 0);
    }
    all &= check("all freed", g_held.empty() && g_used == 0);
    return all ? 0 : 1;
}
