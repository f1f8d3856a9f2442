// A CUDA runtime without a GPU, for tests of the library's host code: device
// memory is address ranges, a device has a capacity and a context that can be
// replaced (as cudaDeviceReset does), streams hold work until somebody waits for
// the device.  Uses of memory that is gone are counted, not made.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {

struct Range {
    size_t bytes;
    int dev;
    bool busy;  // queued work uses it
};
struct State {
    std::map<char *, Range> device;          // live device memory
    std::map<char *, int> host;              // live pinned memory, the device of its context
    std::map<int, unsigned long long> ctx;   // a device's context id
    std::map<int, size_t> used;
    size_t capacity = ~size_t(0) >> 1;
    unsigned long long next_ctx = 1;
    char *next = reinterpret_cast<char *>(0x700000000000);
    long long mallocs = 0, frees = 0, bad = 0;
    bool no_ids = false;
} g;
std::recursive_mutex g_mu;
std::map<const void *, std::string> g_kernels;
thread_local int t_dev = 0;
thread_local std::map<int, bool> t_bound;  // a context is current on this thread
thread_local cudaError_t t_last = cudaSuccess;
thread_local struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t st;
} t_call;

using Lock = std::lock_guard<std::recursive_mutex>;

unsigned long long bind() {
    t_bound[t_dev] = true;
    unsigned long long &c = g.ctx[t_dev];
    if (!c) c = g.next_ctx++;
    return c;
}
cudaError_t ret(cudaError_t e) {
    if (e != cudaSuccess) t_last = e;
    return e;
}
bool live(const void *p) {
    auto it = g.device.upper_bound((char *)p);
    if (it == g.device.begin()) return false;
    --it;
    return (char *)p < it->first + it->second.bytes;
}
CUresult get_current(CUcontext *c) {
    Lock l(g_mu);
    *c = !g.no_ids && t_bound[t_dev] && g.ctx[t_dev] ? (CUcontext)(uintptr_t)g.ctx[t_dev] : nullptr;
    return CUDA_SUCCESS;
}
CUresult get_id(CUcontext c, unsigned long long *id) {
    *id = (unsigned long long)(uintptr_t)c;
    return CUDA_SUCCESS;
}

}  // namespace

// What the tested files take from the rest of the library, and what the test calls in them.
void fv_note_launch() {}
void fv_internal_set_cuda_error(cudaError_t, const char *) {}
void fv_internal_set_error_text(const char *) {}
cudaError_t fv_block_alloc_raw(void **p, size_t bytes);
cudaError_t fv_device_malloc_raw(void **p, size_t bytes);
cudaError_t fv_malloc_async_raw(void **p, size_t bytes, cudaStream_t st);
void fv_blocks_free(void *const *blocks, int n);
unsigned long long fv_bound_context_id();
int *fv_flag_take(unsigned long long ctx);
void fv_flag_return(unsigned long long ctx, int *flag, bool idle);

extern "C" {

// ------------------------------------------------------------------ the test's side
void *pool_alloc(size_t bytes) {
    void *p = nullptr;
    return fv_block_alloc_raw(&p, bytes) == cudaSuccess ? p : nullptr;
}
void *device_alloc(size_t bytes) {
    void *p = nullptr;
    return fv_device_malloc_raw(&p, bytes) == cudaSuccess ? p : nullptr;
}
void *stream_alloc(size_t bytes) {
    void *p = nullptr;
    return fv_malloc_async_raw(&p, bytes, nullptr) == cudaSuccess ? p : nullptr;
}
// Takes a flag, says whether its memory is there, and gives it back.
int flag_is_there(int idle) {
    const unsigned long long ctx = fv_bound_context_id();
    int *const f = fv_flag_take(ctx);
    Lock l(g_mu);
    const bool there = f && g.host.count((char *)f);
    fv_flag_return(ctx, f, idle != 0);
    return there;
}
size_t fake_pinned() { return g.host.size(); }
void pool_free(void *p) { fv_blocks_free(&p, 1); }
void fake_reset() {
    Lock l(g_mu);
    const unsigned long long c = g.next_ctx;
    char *const n = g.next;
    g = State();
    g.next_ctx = c;
    g.next = n;
}
void fake_device(int dev) { t_dev = dev; }
void fake_capacity(size_t bytes) { g.capacity = bytes; }
void fake_no_context_ids(int on) { g.no_ids = on != 0; }
// The context of the current device and all its memory are gone; addresses start again.
void fake_replace_context() {
    Lock l(g_mu);
    for (auto it = g.device.begin(); it != g.device.end();) it = it->second.dev == t_dev ? g.device.erase(it) : std::next(it);
    for (auto it = g.host.begin(); it != g.host.end();) it = it->second == t_dev ? g.host.erase(it) : std::next(it);
    g.used[t_dev] = 0;
    g.ctx[t_dev] = 0;
    if (g.device.empty()) g.next = reinterpret_cast<char *>(0x700000000000);
}
void fake_use(void *p) {  // work that uses p is queued on some stream
    Lock l(g_mu);
    auto it = g.device.find((char *)p);
    if (it == g.device.end())
        ++g.bad;
    else
        it->second.busy = true;
}
int fake_busy(void *p) {
    auto it = g.device.find((char *)p);
    return it != g.device.end() && it->second.busy;
}
long long fake_count(int what) {
    return what == 0 ? g.mallocs : what == 1 ? g.frees : g.bad;
}
size_t fake_used() { return g.used[t_dev]; }

// ------------------------------------------------------------------ the runtime's side
cudaError_t cudaGetDevice(int *d) {
    *d = t_dev;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = t_last;
    t_last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *name, void **f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *q) {
    *f = !strcmp(name, "cuCtxGetCurrent") ? (void *)get_current : !strcmp(name, "cuCtxGetId") ? (void *)get_id : nullptr;
    if (q) *q = *f ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t bytes) {
    Lock l(g_mu);
    bind();
    ++g.mallocs;
    if (g.used[t_dev] + bytes > g.capacity) return ret(cudaErrorMemoryAllocation);
    *p = g.next;
    g.device[g.next] = Range{bytes, t_dev, false};
    g.next += (bytes + 511) / 256 * 256;
    g.used[t_dev] += bytes;
    return cudaSuccess;
}
// As the runtime's does, it waits for the device.
cudaError_t cudaFree(void *p) {
    Lock l(g_mu);
    bind();
    if (!p) return cudaSuccess;
    ++g.frees;
    auto it = g.device.find((char *)p);
    if (it == g.device.end()) {
        ++g.bad;
        return ret(cudaErrorInvalidValue);
    }
    for (auto &d : g.device)
        if (d.second.dev == it->second.dev) d.second.busy = false;
    g.used[it->second.dev] -= it->second.bytes;
    g.device.erase(it);
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int) {
    *p = nullptr;
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMallocAsync(void **p, size_t bytes, cudaStream_t) { return cudaMalloc(p, bytes); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) {
    Lock l(g_mu);
    bind();
    *p = malloc(bytes);  // never given back: the test process reads it after it is gone
    g.host[(char *)*p] = t_dev;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    Lock l(g_mu);
    if (!p) return cudaSuccess;
    if (!g.host.erase((char *)p)) {
        ++g.bad;
        return ret(cudaErrorInvalidValue);
    }
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int, size_t, cudaStream_t) {
    Lock l(g_mu);
    if (!live(p)) {
        ++g.bad;
        return ret(cudaErrorInvalidValue);
    }
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }

// Kernels: the reductions leave the number of entries as their result.
void **__cudaRegisterFatBinary(void *) {
    static void *h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
    g_kernels[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t st) {
    t_call = {grid, block, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *st) {
    *grid = t_call.grid;
    *block = t_call.block;
    *smem = t_call.smem;
    *(cudaStream_t *)st = t_call.st;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **args, size_t, cudaStream_t) {
    Lock l(g_mu);
    bind();
    if (g_kernels[f].find("k_vec_reduce") != std::string::npos) {
        char *partial = *(char **)args[3], *out = *(char **)args[4];
        auto it = g.host.find(out);
        if (!live(partial) || it == g.host.end())
            ++g.bad;
        else
            *(double *)out = (double)*(int64_t *)args[0];
    }
    return cudaSuccess;
}

}  // extern "C"
