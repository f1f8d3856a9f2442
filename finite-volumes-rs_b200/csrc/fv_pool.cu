// Device memory of matrices and preconditioners: freed blocks are kept for the
// next object.
//
// A program that assembles, factorises and solves once per problem spent more
// on cudaMalloc / cudaFree than on the factorisation: a block of a megabyte or
// less costs 2-4 us each way, one of several megabytes 1-4 ms, because it is
// mapped and unmapped every time (24,576 rows: 3-5 ms of an 8 ms solve).
//
// A block is handed out again only after the device has finished all work
// submitted before it was freed: fv_blocks_free first allocates and frees 256
// bytes, and cudaFree synchronises across all streams of the device (the CUDA
// programming guide says so of cudaMalloc and cudaFree where it introduces the
// stream-ordered allocator; measured: it returns when a kernel in flight on
// another, non-blocking stream ends).  So a block from here may be used on any
// stream at once, like memory from cudaMalloc.  cudaDeviceSynchronize would wait
// as well, but a stream capture on any other host thread is invalidated by it, in
// every capture mode; dropping an object leaves thread-local and relaxed captures
// alone, as cudaFree of its blocks does.
//
// Kept memory is bounded (kKeepBytes per context, blocks of at most kKeepBlock;
// the oldest make room for the next) and given back when an allocation of this
// library fails or fv_release_kept_memory is called.  Blocks belong to the
// context they were made in and are handed out, kept and freed in that one only:
// when it has been replaced (cudaDeviceReset), its addresses mean nothing any
// more, or something else.
#include <cuda.h>  // CUcontext / CUresult types only; the driver calls are reached through the runtime

#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "fv_internal.cuh"

// Unique id of the calling thread's current context (cuCtxGetId, unique over
// the process's life), or 0 when the driver does not provide it.
unsigned long long fv_current_context_id() {
    using GetCurrent = CUresult (*)(CUcontext *);
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = (GetCurrent)f;
        f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = (GetId)f;
        cudaGetLastError();
    });
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS)
        return 0;
    return id;
}

// The same, once the current device's context is current on this thread: a
// thread that has made no call yet which needs one has none.
unsigned long long fv_bound_context_id() {
    const unsigned long long id = fv_current_context_id();
    return id != 0 || cudaFree(nullptr) != cudaSuccess ? id : fv_current_context_id();
}

namespace {

constexpr size_t kKeepBytes = 512u << 20, kKeepBlock = 64u << 20;

struct Block {
    size_t bytes;
    unsigned long long ctx;
};
struct Kept {
    struct Entry {
        void *p;
        unsigned long long age;
    };
    using BySize = std::multimap<size_t, Entry>;
    BySize by_size;
    std::map<unsigned long long, BySize::iterator> by_age;  // the oldest first
    unsigned long long next_age = 0;
    size_t bytes = 0;

    void put(size_t size, void *p) {
        const auto it = by_size.emplace(size, Entry{p, next_age});
        try {
            by_age.emplace(next_age++, it);
        } catch (...) {
            by_size.erase(it);
            throw;
        }
        bytes += size;
    }
    void take(BySize::iterator it) {
        bytes -= it->first;
        by_age.erase(it->second.age);
        by_size.erase(it);
    }
};
std::mutex g_mu;
std::unordered_map<void *, Block> g_live;     // blocks handed out that may be kept when freed
std::map<unsigned long long, Kept> g_kept;    // by context

}  // namespace

// Everything kept in the current context goes back to the driver; whether that was anything.
static bool give_back() {
    std::lock_guard<std::mutex> g(g_mu);
    auto it = g_kept.find(fv_bound_context_id());
    if (it == g_kept.end() || it->second.by_size.empty()) return false;
    for (auto &b : it->second.by_size) cudaFree(b.second.p);
    g_kept.erase(it);
    return true;
}

extern "C" fv_status fv_release_kept_memory(void) {
    return fv_host_guard([] {
        give_back();
        return FV_OK;
    });
}

// An allocation, made again after kept memory was given back when there is none left.
template <class F>
static cudaError_t with_kept_memory(F alloc) {
    cudaError_t e = alloc();
    if (e == cudaErrorMemoryAllocation && give_back()) {
        cudaGetLastError();
        e = alloc();
    }
    return e;
}

cudaError_t fv_device_malloc_raw(void **p, size_t bytes) {
    return with_kept_memory([&] { return cudaMalloc(p, bytes); });
}

cudaError_t fv_malloc_async_raw(void **p, size_t bytes, cudaStream_t st) {
    static std::atomic<bool> configured[64];
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && !configured[dev].load()) {
        std::lock_guard<std::mutex> g(mu);
        if (!configured[dev].load()) {
            cudaMemPool_t pool;
            if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
                uint64_t keep = UINT64_MAX;
                cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
            }
            configured[dev].store(true);
        }
    }
    return with_kept_memory([&] { return cudaMallocAsync(p, bytes, st); });
}

cudaError_t fv_block_alloc_raw(void **p, size_t bytes) {
    *p = nullptr;
    const unsigned long long ctx = fv_bound_context_id();  // 0 (unknown): nothing is taken or kept
    const bool keep = ctx != 0 && bytes <= kKeepBlock;
    try {
        if (keep) {
            std::lock_guard<std::mutex> g(g_mu);
            Kept &k = g_kept[ctx];
            auto it = k.by_size.lower_bound(bytes);
            if (it != k.by_size.end() && it->first <= bytes + bytes / 4 + 4096) {
                void *const block = it->second.p;
                g_live[block] = Block{it->first, ctx};
                k.take(it);
                *p = block;
                return cudaSuccess;
            }
        }
        const cudaError_t e = fv_device_malloc_raw(p, bytes);
        if (e == cudaSuccess && keep) {
            std::lock_guard<std::mutex> g(g_mu);
            g_live[*p] = Block{bytes, ctx};
        }
        return e;
    } catch (...) {  // host memory for the bookkeeping: plain memory then
        return *p ? cudaSuccess : cudaMalloc(p, bytes);
    }
}

void fv_block_free(void *p) {
    if (!p) return;
    {
        std::lock_guard<std::mutex> g(g_mu);
        g_live.erase(p);
    }
    cudaFree(p);
}

void fv_blocks_free(void *const *blocks, int n) {
    if (std::all_of(blocks, blocks + n, [](void *p) { return !p; })) return;
    const unsigned long long ctx = fv_bound_context_id();
    void *fence = nullptr;
    const bool idle = ctx != 0 && cudaMalloc(&fence, 256) == cudaSuccess &&
                      cudaFree(fence) == cudaSuccess;  // waits for the device
    if (!idle) cudaGetLastError();
    for (int i = 0; i < n; ++i) {
        if (!blocks[i]) continue;
        bool kept = false;
        if (idle) {
            try {
                std::lock_guard<std::mutex> g(g_mu);
                auto it = g_live.find(blocks[i]);
                if (it != g_live.end() && it->second.ctx == ctx) {
                    const size_t bytes = it->second.bytes;
                    Kept &k = g_kept[ctx];
                    while (k.bytes + bytes > kKeepBytes) {  // the oldest make room
                        const auto oldest = k.by_age.begin()->second;
                        cudaFree(oldest->second.p);
                        k.take(oldest);
                    }
                    k.put(bytes, blocks[i]);
                    g_live.erase(it);
                    kept = true;
                }
            } catch (...) {  // host memory for the bookkeeping: freed then
            }
        }
        if (!kept) fv_block_free(blocks[i]);
    }
}

// Flags wait under their context's id: replacing a context frees its pinned
// memory.  At most as many as were taken at once (freeing pinned memory may
// synchronise the device, so a solve does not).
static std::map<unsigned long long, std::vector<int *>> g_flags;

int *fv_flag_take(unsigned long long ctx) {
    if (ctx != 0) {
        std::lock_guard<std::mutex> g(g_mu);
        const auto it = g_flags.find(ctx);
        if (it != g_flags.end() && !it->second.empty()) {
            int *const flag = it->second.back();
            it->second.pop_back();
            return flag;
        }
    }
    int *flag = nullptr;
    if (cudaHostAlloc((void **)&flag, sizeof(int), cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        flag = nullptr;
    }
    return flag;
}

void fv_flag_return(unsigned long long ctx, int *flag, bool idle) {
    if (!flag) return;
    if (idle && ctx != 0) {
        try {
            std::lock_guard<std::mutex> g(g_mu);
            g_flags[ctx].push_back(flag);
            return;
        } catch (...) {  // host memory for the list: freed then
        }
    }
    cudaFreeHost(flag);
}
