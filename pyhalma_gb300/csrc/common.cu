// Status strings, per-thread error text, cached workspace and launch accounting.
#include <stdarg.h>
#include <stdio.h>
#include <unistd.h>

#include <atomic>
#include <map>

#include "common.cuh"

namespace halma {

static thread_local char g_last_error[512] = "";
static thread_local int64_t g_group_members = 0;

void set_group_members(int64_t n) { g_group_members = n; }
static std::atomic<int64_t> g_launches{0};

int fail(int status, const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
    va_end(ap);
    return status;
}

int cuda_fail(cudaError_t e, const char *what, const char *file, int line) {
    int st = (e == cudaErrorMemoryAllocation) ? HALMA_ERR_NOMEM
             : (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) ? HALMA_ERR_NO_DEVICE
                                                                             : HALMA_ERR_CUDA;
    return fail(st, "%s failed: %s (%s:%d)", what, cudaGetErrorString(e), file, line);
}

void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
void add_launches(int64_t k) { g_launches.fetch_add(k, std::memory_order_relaxed); }

std::mutex &api_mutex() {
    static std::mutex m;
    return m;
}

int current_device() {
    int d = 0;
    cudaGetDevice(&d);
    return d;
}

int device_sm_count() {
    static std::mutex m;
    static std::map<int, int> cache;
    int d = current_device();
    std::lock_guard<std::mutex> g(m);
    auto it = cache.find(d);
    if (it != cache.end()) return it->second;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d) != cudaSuccess || sms <= 0)
        sms = 148;
    cache[d] = sms;
    return sms;
}

struct WsEntry {
    void *ptr = nullptr;
    size_t bytes = 0;
};
static std::map<std::pair<int, int>, WsEntry> &ws_map() {   // (device, slot)
    static std::map<std::pair<int, int>, WsEntry> m;
    return m;
}

int workspace(size_t bytes, void **ptr, cudaStream_t stream, int slot) {
    int d = current_device();
    WsEntry &e = ws_map()[{d, slot}];
    if (bytes == 0) bytes = 256;
    if (e.bytes < bytes) {
        if (e.ptr) {
            // earlier work on any stream may still read the old buffer
            HALMA_CUDA(cudaDeviceSynchronize());
            HALMA_CUDA(cudaFree(e.ptr));
            e.ptr = nullptr;
            e.bytes = 0;
        }
        size_t want = bytes + bytes / 8;
        void *p = nullptr;
        cudaError_t err = cudaMalloc(&p, want);
        if (err != cudaSuccess) {
            cudaGetLastError();
            return fail(HALMA_ERR_NOMEM, "workspace allocation of %zu bytes failed: %s", want,
                        cudaGetErrorString(err));
        }
        e.ptr = p;
        e.bytes = want;
    }
    (void)stream;
    *ptr = e.ptr;
    return HALMA_OK;
}

MemoryKind memory_kind(const void *p) {
    if (!p) return MemoryKind::kUnknown;
    cudaPointerAttributes a;
    cudaError_t e = cudaPointerGetAttributes(&a, p);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return MemoryKind::kUnknown;
    }
    if (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) return MemoryKind::kDevice;
    return a.type == cudaMemoryTypeHost ? MemoryKind::kPinned : MemoryKind::kPageable;
}

bool is_device_pointer(const void *p) { return memory_kind(p) == MemoryKind::kDevice; }

bool host_page_tables() {
    static std::map<int, bool> m;   // a property of the device
    static std::mutex mu;
    std::lock_guard<std::mutex> guard(mu);
    const int d = current_device();
    auto it = m.find(d);
    if (it == m.end()) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrPageableMemoryAccessUsesHostPageTables, d) != cudaSuccess) {
            cudaGetLastError();
            v = 0;
        }
        it = m.emplace(d, v != 0).first;
    }
    return it->second;
}

void touch_pages(const void *p, size_t bytes) {
    static const size_t page = (size_t)std::max(sysconf(_SC_PAGESIZE), 1l);
    if (bytes == 0) return;
    const volatile unsigned char *c = static_cast<const unsigned char *>(p);
    (void)c[0];
    for (size_t k = page - reinterpret_cast<uintptr_t>(p) % page; k < bytes; k += page) (void)c[k];
}

namespace {

// Array blockIdx.y, in the widest words its address allows (the destination is 256-byte aligned), then the bytes left over.
template <class W>
__device__ __forceinline__ size_t upload_words(const void *src, void *dst, size_t bytes) {
    const W *from = static_cast<const W *>(src);
    W *to = static_cast<W *>(dst);
    const size_t n = bytes / sizeof(W), step = (size_t)gridDim.x * blockDim.x;
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    for (; i + 3 * step < n; i += 4 * step) {
        W v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = from[i + k * step];
#pragma unroll
        for (int k = 0; k < 4; ++k) to[i + k * step] = v[k];
    }
    for (; i < n; i += step) to[i] = from[i];
    return n * sizeof(W);
}

__global__ void __launch_bounds__(512) upload_kernel(Uploads u) {
    const void *src = u.src[blockIdx.y];
    void *dst = u.dst[blockIdx.y];
    const size_t bytes = u.bytes[blockIdx.y];
    const unsigned at = (unsigned)(uintptr_t)src;
    const size_t done = at % 16 == 0  ? upload_words<uint4>(src, dst, bytes)
                        : at % 8 == 0 ? upload_words<uint2>(src, dst, bytes)
                        : at % 4 == 0 ? upload_words<unsigned>(src, dst, bytes)
                                      : upload_words<unsigned char>(src, dst, bytes);
    const size_t i = done + blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < bytes) static_cast<unsigned char *>(dst)[i] = static_cast<const unsigned char *>(src)[i];
}

}  // namespace

int upload(const Uploads &u, cudaStream_t s) {
    size_t most = 0;
    for (int k = 0; k < u.n; ++k) most = std::max(most, u.bytes[k]);
    HALMA_LAUNCH(upload_kernel, dim3((unsigned)grid_for((int64_t)(most / 16 + 1), 512, 64), (unsigned)u.n), 512, 0, s, u);
    return HALMA_OK;
}

}  // namespace halma

extern "C" {

int halma_abi_version(void) { return HALMA_ABI_VERSION; }

const char *halma_status_string(int s) {
    switch (s) {
        case HALMA_OK: return "ok";
        case HALMA_ERR_INVALID: return "invalid argument";
        case HALMA_ERR_NOMEM: return "out of memory";
        case HALMA_ERR_CUDA: return "CUDA error";
        case HALMA_ERR_NOT_CONVERGED: return "not converged";
        case HALMA_ERR_TIMEOUT: return "device wait timed out";
        case HALMA_ERR_CAPACITY: return "capacity exceeded";
        case HALMA_ERR_NO_DEVICE: return "no CUDA device";
        default: return "unknown status";
    }
}

const char *halma_last_error(void) { return halma::g_last_error; }

int64_t halma_last_group_members(void) { return halma::g_group_members; }

int64_t halma_kernel_launch_count(void) { return halma::g_launches.load(); }

int halma_release_workspace(void) {
    std::lock_guard<std::mutex> g(halma::api_mutex());
    for (auto &kv : halma::ws_map()) {
        if (kv.second.ptr) {
            cudaSetDevice(kv.first.first);
            cudaDeviceSynchronize();
            cudaFree(kv.second.ptr);
        }
    }
    halma::ws_map().clear();
    return HALMA_OK;
}

}  // extern "C"
