// One cluster of one CTA runs the sweeps of a factor without off-diagonal entries
// (z = d_backward * d_forward * r), twice, as a solve does; on request its copies
// never count as landed, or an error is raised before.
#define FV_WAIT_LIMIT_NS 20000000ULL
#include "fv_resident.cuh"

namespace {

constexpr int kMl = 2, kSets = 8, kWidth = 32;
using Rec = fv_res_rec<double, kMl>;
constexpr int kPl = sizeof(Rec) / 16;

__global__ void __cluster_dims__(1) __launch_bounds__(kResThreads, 1)
    k_run(const __grid_constant__ fv_res_args a, const double *r, double *z, int never, int *err) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ unsigned long long bars[kResBars];
    fv_res_cta<double, kMl, kSets> cta(a, smem, bars);
    fv_cluster_arrive();
    fv_cluster_wait();
    if (never && threadIdx.x == 0)  // two arrivals complete a phase, a copy makes one
        for (int b = 0; b < kResBuffers; ++b) {
            const unsigned m = (unsigned)__cvta_generic_to_shared(&bars[b]);
            asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(m) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(m) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    __syncthreads();
    cta.load(r);
    cta.sweeps(err);
    cta.sweeps(err);
    cta.store(z, fv_row_skip{});
}

}  // namespace

// rows: rows of the CTA, `levels` of kWidth rows each; returns milliseconds, < 0: a CUDA error.
extern "C" float run(int levels, int never, int raise, const double *r, const double *d, double *z, int *err_out) {
    const int rows = levels * kWidth, steps = 2 * levels, pad = (kSets - steps % kSets) % kSets, ns = steps + pad;
    std::vector<Rec> rec((size_t)ns * kWidth);
    std::vector<uint4> planes((size_t)ns * kWidth * kPl);
    std::vector<int32_t> ids(rows);
    for (int i = 0; i < rows; ++i) ids[i] = i;
    for (int s = 0; s < ns; ++s)
        for (int l = 0; l < kWidth; ++l) {
            Rec &q = rec[(size_t)s * kWidth + l];
            memset(&q, 0, sizeof(q));
            for (int e = 0; e < kMl; ++e) q.dep[e] = (uint16_t)rows;
            const int row = (s < levels ? s : s - levels) * kWidth + l;
            q.self = (uint16_t)(s < steps ? row : rows + 1);
            q.d = s < steps ? d[row] : 1.0;
            for (int p = 0; p < kPl; ++p)
                planes[((size_t)s * kPl + p) * kWidth + l] = reinterpret_cast<const uint4 *>(&q)[p];
        }
    const int32_t ends[2] = {0, rows}, steps_of[2] = {0, ns};
    uint4 *d_rec;
    int32_t *d_ids, *d_ends, *d_steps;
    double *d_r, *d_z;
    int *d_err;
    cudaMalloc(&d_rec, planes.size() * 16);
    cudaMalloc(&d_ids, 4 * rows);
    cudaMalloc(&d_ends, 8);
    cudaMalloc(&d_steps, 8);
    cudaMalloc(&d_r, 8 * rows);
    cudaMalloc(&d_z, 8 * rows);
    cudaMalloc(&d_err, 4);
    cudaMemcpy(d_rec, planes.data(), planes.size() * 16, cudaMemcpyHostToDevice);
    cudaMemcpy(d_ids, ids.data(), 4 * rows, cudaMemcpyHostToDevice);
    cudaMemcpy(d_ends, ends, 8, cudaMemcpyHostToDevice);
    cudaMemcpy(d_steps, steps_of, 8, cudaMemcpyHostToDevice);
    cudaMemcpy(d_r, r, 8 * rows, cudaMemcpyHostToDevice);
    cudaMemcpy(d_err, &raise, 4, cudaMemcpyHostToDevice);
    const fv_res_args a{d_rec, nullptr, d_steps, d_ends, d_ids, 1, rows, 0, kWidth, kSets};
    const size_t smem = (size_t)kResBuffers * kSets * kWidth * sizeof(Rec) + (size_t)(rows + 2) * 8;
    cudaFuncSetAttribute(k_run, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmem);
    cudaEvent_t e[2];
    for (cudaEvent_t &v : e) cudaEventCreate(&v);
    cudaDeviceSynchronize();
    cudaEventRecord(e[0]);
    if (smem <= kResSmem) k_run<<<1, kResThreads, smem>>>(a, d_r, d_z, never, d_err);
    cudaEventRecord(e[1]);
    float ms = -1.f;
    if (smem > kResSmem || cudaDeviceSynchronize() != cudaSuccess || cudaEventElapsedTime(&ms, e[0], e[1]) != cudaSuccess)
        ms = -1.f;
    cudaMemcpy(z, d_z, 8 * rows, cudaMemcpyDeviceToHost);
    cudaMemcpy(err_out, d_err, 4, cudaMemcpyDeviceToHost);
    for (void *p : {(void *)d_rec, (void *)d_ids, (void *)d_ends, (void *)d_steps, (void *)d_r, (void *)d_z, (void *)d_err})
        cudaFree(p);
    for (cudaEvent_t v : e) cudaEventDestroy(v);
    return ms;
}
