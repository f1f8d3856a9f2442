// DistributedVector operations (linalg/dvector.rs:46-160): dot / dot_smaller
// and sum with a fixed reduction order (each thread sums a fixed strided set
// of entries, then a fixed shuffle tree, then the block partials in block
// order, so a result depends only on n and the data), and the elementwise
// updates +=, -=, *= (scalar), inv and set, which are exact.
#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

#include "fv_internal.cuh"

namespace {

constexpr int kVB = 256;

inline int vec_grid(int64_t n) {
    const int64_t b = (n + kVB - 1) / kVB;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, 148 * 4));
}

constexpr int kMaxBlocks = 148 * 4;

// The workspace of a reduction: the block partials and the ticket (0 between
// uses), and the result in pinned host memory, which the kernel writes.  Both
// belong to the context they were made in (cudaDeviceReset frees them), so free
// ones wait under its id: at most as many as reductions ran at once.  A reduction
// returns its workspace after its stream has finished, so no two meet in one.
struct Workspace {
    double *partial = nullptr;  // kMaxBlocks values, then the ticket
    double *result = nullptr;
};
std::mutex g_mu;
std::map<unsigned long long, std::vector<Workspace>> g_free;

void destroy(Workspace &w) {
    cudaFree(w.partial);
    cudaFreeHost(w.result);
}

cudaError_t take_workspace(unsigned long long ctx, cudaStream_t st, Workspace &w) {
    if (ctx != 0) {
        std::lock_guard<std::mutex> g(g_mu);
        auto it = g_free.find(ctx);
        if (it != g_free.end() && !it->second.empty()) {
            w = it->second.back();
            it->second.pop_back();
            return cudaSuccess;
        }
    }
    cudaError_t e = fv_device_malloc(&w.partial, sizeof(double) * (kMaxBlocks + 1));
    if (e == cudaSuccess) e = cudaHostAlloc((void **)&w.result, sizeof(double), cudaHostAllocPortable);
    if (e == cudaSuccess) e = cudaMemsetAsync(w.partial, 0, sizeof(double) * (kMaxBlocks + 1), st);
    if (e != cudaSuccess) destroy(w);
    return e;
}

void return_workspace(unsigned long long ctx, Workspace &w) {
    if (ctx != 0) {
        try {
            std::lock_guard<std::mutex> g(g_mu);
            g_free[ctx].push_back(w);
            return;
        } catch (...) {  // host memory for the list: freed then
        }
    }
    destroy(w);
}

__device__ __forceinline__ double block_sum(double v, double *sm) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kVB / 32; ++w) t += sm[w];
    return t;
}

// DOT: sum x_i y_i, else sum x_i.  One kernel: the last block to finish loads
// the block partials together and adds them in block order (a second kernel's
// single thread read them from L2 one after the other), and the result goes
// straight to the host.  Bound by memory above some 10^6 entries, below by the
// launch and the host's wait: dot of 10,007 entries 34 -> 22 us per call from
// Python, of 1,000,003 entries 56 -> 24, of 8,000,000 entries 69 -> 41.
template <bool DOT>
__global__ void __launch_bounds__(kVB) k_vec_reduce(int64_t n, const double *__restrict__ x,
                                                    const double *__restrict__ y, double *partial,
                                                    double *__restrict__ out) {
    __shared__ double sm[kVB / 32], all[kMaxBlocks];
    __shared__ bool last;
    unsigned *ticket = reinterpret_cast<unsigned *>(partial + kMaxBlocks);
    double acc = 0.0;
#pragma unroll 4
    for (int64_t i = (int64_t)blockIdx.x * kVB + threadIdx.x; i < n; i += (int64_t)gridDim.x * kVB)
        acc += DOT ? x[i] * y[i] : x[i];
    const double t = block_sum(acc, sm);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = t;
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    for (int b = threadIdx.x; b < gridDim.x; b += kVB) all[b] = __ldcg(&partial[b]);
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int b = 0; b < gridDim.x; ++b) s += all[b];
        *ticket = 0;
        *out = s;
        __threadfence_system();
    }
}

// op 0: y += x; 1: y -= x; 2: y *= a; 3: y = 1 / y; 4: y = x
__global__ void k_vec_update(int64_t n, double *__restrict__ y, const double *__restrict__ x, double a, int op) {
    for (int64_t i = (int64_t)blockIdx.x * kVB + threadIdx.x; i < n; i += (int64_t)gridDim.x * kVB) {
        switch (op) {
        case 0: y[i] = y[i] + x[i]; break;
        case 1: y[i] = y[i] - x[i]; break;
        case 2: y[i] = y[i] * a; break;
        case 3: y[i] = 1.0 / y[i]; break;
        default: y[i] = x[i]; break;
        }
    }
}

fv_status reduce(int64_t n, const double *x, const double *y, int mode, void *stream, double *out) {
    if (n < 0 || !out) return FV_ERR_INVALID;
    if (n == 0) {  // empty vectors: no data pointer is needed
        *out = 0.0;
        return FV_OK;
    }
    if (!x || (mode == 0 && !y)) return FV_ERR_INVALID;
    cudaStream_t st = fv_stream(stream);
    const unsigned long long ctx = fv_bound_context_id();
    Workspace w;
    FV_CUDA_TRY(take_workspace(ctx, st, w));
    fv_note_launch();
    if (mode == 0)
        k_vec_reduce<true><<<vec_grid(n), kVB, 0, st>>>(n, x, y, w.partial, w.result);
    else
        k_vec_reduce<false><<<vec_grid(n), kVB, 0, st>>>(n, x, y, w.partial, w.result);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        destroy(w);
        FV_CUDA_TRY(e);
    }
    *out = *(volatile double *)w.result;
    return_workspace(ctx, w);
    return FV_OK;
}

}  // namespace

extern "C" fv_status fv_vec_dot(int64_t n, const double *x, const double *y, void *stream, double *out) {
    return reduce(n, x, y, 0, stream, out);
}

extern "C" fv_status fv_vec_sum(int64_t n, const double *x, void *stream, double *out) {
    return reduce(n, x, nullptr, 1, stream, out);
}

extern "C" fv_status fv_vec_update(int64_t n, double *y, const double *x, double a, int32_t op, void *stream) {
    if (n < 0 || op < 0 || op > 4) return FV_ERR_INVALID;
    if (n == 0) return FV_OK;
    if (!y || ((op == 0 || op == 1 || op == 4) && !x)) return FV_ERR_INVALID;
    cudaStream_t st = fv_stream(stream);
    fv_note_launch();
    k_vec_update<<<vec_grid(n), kVB, 0, st>>>(n, y, x, a, op);
    FV_CUDA_TRY(cudaGetLastError());
    return FV_OK;
}
