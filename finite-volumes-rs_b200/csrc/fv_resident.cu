// Plans, records and launch of the resident sweeps (fv_resident.cuh).
#include <algorithm>
#include <cub/cub.cuh>
#include <cstdint>
#include <new>
#include <vector>

#include "fv_resident.cuh"

namespace {

// ------------------------------------------------------------------ plan kernels
// first[k] = first position p with key(p) >= k (keys ascending), for k = 0 .. nk
template <class Key>
__device__ __forceinline__ void res_bounds(int64_t p, int64_t n, int32_t nk, Key key, int32_t *__restrict__ first) {
    if (p > n) return;
    const int64_t a = p == 0 ? 0 : (int64_t)key(p - 1) + 1, b = p == n ? nk : (int64_t)key(p);
    for (int64_t k = a; k <= b; ++k) first[k] = (int32_t)p;
}
__global__ void k_res_bounds(int64_t n, int32_t nk, const uint32_t *__restrict__ key, int32_t *__restrict__ first) {
    res_bounds((int64_t)blockIdx.x * blockDim.x + threadIdx.x, n, nk, [=](int64_t p) { return key[p]; }, first);
}
__global__ void k_res_level_start(int64_t n, int32_t nlev, const int32_t *__restrict__ order,
                                  const int32_t *__restrict__ level, int32_t *__restrict__ first) {
    res_bounds((int64_t)blockIdx.x * blockDim.x + threadIdx.x, n, nlev, [=](int64_t p) { return level[order[p]]; },
               first);
}

// The CTA of every row.
//
// Rows sorted by level (k_res_owner_sorted): a row goes where its last
// dependency goes, down to a row of level 0, and those are dealt in equal
// ranges -- with the box-colour order the rows of a box follow each other along
// their dependencies, so a box stays with one CTA.
//
// Narrow levels (res_build): bands of levels.
//
// Any other order: each level's rows are dealt in equal ranges (balanced, but a
// CTA's share moves through the mesh from level to level), or, where the rows'
// cell centres are known and every level stays balanced, the mesh is cut into
// slabs along one axis (k_res_choose).  Then a lexicographic mesh sends values
// to other CTAs only at the slabs' faces and only downstream, so a CTA lags its
// neighbour instead of waiting on every level (24,576-row ILU(0) on 8 CTAs:
// 1,024 halo slots per CTA instead of 9,065).
//
// A batch's problems (k_res_owner_batch): the same within each problem, over the
// CTAs of the problem's cluster.
__global__ void k_res_root_count(int64_t n, const int32_t *__restrict__ lstart, const int32_t *__restrict__ perm,
                                 const int32_t *__restrict__ of_row, int32_t *__restrict__ root0,
                                 int32_t *__restrict__ nroot) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= lstart[1]) return;
    const int32_t q = of_row[perm ? perm[i] : i];
    atomicMin(&root0[q], (int32_t)i);
    atomicAdd(&nroot[q], 1);
}
__global__ void k_res_owner_batch(int64_t n, int C, const int32_t *__restrict__ perm,
                                  const int32_t *__restrict__ of_row, const int32_t *__restrict__ cluster,
                                  const int32_t *__restrict__ root0, const int32_t *__restrict__ nroot,
                                  const int32_t *__restrict__ lp, const int32_t *__restrict__ lc,
                                  uint32_t *__restrict__ owner) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int32_t q = of_row[perm ? perm[p] : p];
    int r = (int)p;
    for (int e = lp[r + 1]; e > lp[r]; e = lp[r + 1]) r = lc[e - 1];
    const int64_t at = (int64_t)(r - root0[q]) * C / max(1, nroot[q]);
    owner[p] = (uint32_t)(cluster[q] * C + (int)max((int64_t)0, min((int64_t)C - 1, at)));
}
__global__ void k_res_owner_sorted(int64_t n, int C, const int32_t *__restrict__ lstart,
                                   const int32_t *__restrict__ lp, const int32_t *__restrict__ lc,
                                   uint32_t *__restrict__ owner) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    int r = (int)p;
    for (int e = lp[r + 1]; e > lp[r]; e = lp[r + 1]) r = lc[e - 1];  // a dependency is a lower row: ends at a root
    owner[p] = (uint32_t)((int64_t)r * C / lstart[1]);
}

constexpr int kResBins = 256;  // bins of an axis
struct ResAxes {
    unsigned long long lo[3], hi[3];        // extent, as ordered integers
    int32_t bin[3][kResBins];               // rows per bin, then the CTA of a bin
    unsigned int cross[4];                  // dependencies on another CTA: slabs of each axis, balanced
    int32_t axis;                           // the chosen axis, -1: none
};
__device__ __forceinline__ unsigned long long res_ordered(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    return b >> 63 ? ~b : b | 0x8000000000000000ULL;
}
__device__ __forceinline__ double res_from_ordered(unsigned long long b) {
    return __longlong_as_double((long long)(b >> 63 ? b & 0x7FFFFFFFFFFFFFFFULL : ~b));
}
__device__ __forceinline__ int res_bin(const ResAxes *a, int d, double x) {
    const double lo = res_from_ordered(a->lo[d]), hi = res_from_ordered(a->hi[d]);
    const double t = hi > lo ? (x - lo) / (hi - lo) * kResBins : 0.0;
    return min(kResBins - 1, max(0, (int)t));
}
__device__ __forceinline__ double res_coord(const double4 &c, int d) { return d == 0 ? c.x : d == 1 ? c.y : c.z; }

__global__ void k_res_axes_init(ResAxes *a) {
    for (int k = threadIdx.x; k < 3 * kResBins; k += blockDim.x) a->bin[k / kResBins][k % kResBins] = 0;
    if (threadIdx.x < 3) {
        a->lo[threadIdx.x] = ~0ULL;
        a->hi[threadIdx.x] = 0;
    }
    if (threadIdx.x < 4) a->cross[threadIdx.x] = 0;
    if (threadIdx.x == 0) a->axis = -1;
}
__global__ void k_res_extent(int64_t n, const double4 *__restrict__ cell, ResAxes *a) {
    double lo[3], hi[3];
    for (int d = 0; d < 3; ++d) lo[d] = INFINITY, hi[d] = -INFINITY;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double4 c = cell[i];
        for (int d = 0; d < 3; ++d) lo[d] = fmin(lo[d], res_coord(c, d)), hi[d] = fmax(hi[d], res_coord(c, d));
    }
    for (int d = 0; d < 3; ++d) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[d] = fmin(lo[d], __shfl_down_sync(0xffffffffu, lo[d], o));
            hi[d] = fmax(hi[d], __shfl_down_sync(0xffffffffu, hi[d], o));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&a->lo[d], res_ordered(lo[d]));
            atomicMax(&a->hi[d], res_ordered(hi[d]));
        }
    }
}
__global__ void k_res_bins(int64_t n, const double4 *__restrict__ cell, ResAxes *a) {
    __shared__ int32_t cnt[3 * kResBins];
    for (int k = threadIdx.x; k < 3 * kResBins; k += blockDim.x) cnt[k] = 0;
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double4 c = cell[i];
        for (int d = 0; d < 3; ++d) atomicAdd(&cnt[d * kResBins + res_bin(a, d, res_coord(c, d))], 1);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 3 * kResBins; k += blockDim.x)
        if (cnt[k]) atomicAdd(&a->bin[k / kResBins][k % kResBins], cnt[k]);
}
// Equal numbers of rows per CTA along every axis (whole bins).  One warp per axis.
__global__ void k_res_cuts(int64_t n, int C, ResAxes *a) {
    const int d = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int per = kResBins / 32;
    int32_t w[per], sum = 0;
#pragma unroll
    for (int k = 0; k < per; ++k) sum += w[k] = a->bin[d][lane * per + k];
    int32_t before = sum;
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
        const int32_t t = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += t;
    }
    before -= sum;
#pragma unroll
    for (int k = 0; k < per; ++k) {
        a->bin[d][lane * per + k] = (int32_t)min((int64_t)C - 1, (2 * (int64_t)before + w[k]) * C / (2 * n));
        before += w[k];
    }
}
// Bands of levels, or the balanced candidate and the rows of every (axis, CTA, level) of the slabs.
__global__ void k_res_owner(int64_t n, int C, bool bands, int32_t nlev, const int32_t *__restrict__ order,
                            const int32_t *__restrict__ level, const int32_t *__restrict__ lstart,
                            const double4 *__restrict__ cell, const ResAxes *__restrict__ a,
                            uint32_t *__restrict__ owner, int32_t *__restrict__ hist) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int32_t i = order[p], l = level[i], s = lstart[l];
    owner[i] = bands ? (uint32_t)(p * C / n) : (uint32_t)((p - s) * C / (lstart[l + 1] - s));
    if (!cell) return;
    const double4 c = cell[i];
    for (int d = 0; d < 3; ++d)
        atomicAdd(&hist[((int64_t)d * C + a->bin[d][res_bin(a, d, res_coord(c, d))]) * nlev + l], 1);
}
__global__ void k_res_cross(int64_t n, const int32_t *__restrict__ lp, const int32_t *__restrict__ lc,
                            const double4 *__restrict__ cell, const uint32_t *__restrict__ owner, ResAxes *a) {
    unsigned int cnt[4] = {0, 0, 0, 0};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double4 c = cell[i];
        for (int e = lp[i]; e < lp[i + 1]; ++e) {
            const int32_t j = lc[e];
            const double4 q = cell[j];
            for (int d = 0; d < 3; ++d)
                cnt[d] += a->bin[d][res_bin(a, d, res_coord(c, d))] != a->bin[d][res_bin(a, d, res_coord(q, d))];
            cnt[3] += owner[i] != owner[j];
        }
    }
    for (int d = 0; d < 4; ++d) {
        const unsigned int t = __reduce_add_sync(0xffffffffu, cnt[d]);
        if ((threadIdx.x & 31) == 0 && t) atomicAdd(&a->cross[d], t);
    }
}
// The axis whose slabs need the fewest steps (steps of a level = those of its
// fullest CTA), when that is at most a quarter more than the balanced number
// and the slabs at least halve the dependencies between CTAs (they do on 3D
// meshes; on the 2D ones the balanced ranges move little from level to level
// and the slabs were slower: 65,522-row IC(0) 195 us per apply against 108, where
// 24,576-row ILU(0) takes 51 in slabs and 115 dealt).
// One block.
__global__ void k_res_choose(int C, int width, int32_t nlev, const int32_t *__restrict__ lstart,
                             const int32_t *__restrict__ hist, ResAxes *a) {
    __shared__ int sums[4];
    if (threadIdx.x < 4) sums[threadIdx.x] = 0;
    __syncthreads();
    for (int l = threadIdx.x; l < nlev; l += blockDim.x) {
        for (int d = 0; d < 3; ++d) {
            int m = 0;
            for (int c = 0; c < C; ++c) m = max(m, hist[((int64_t)d * C + c) * nlev + l]);
            atomicAdd(&sums[d], (m + width - 1) / width);
        }
        atomicAdd(&sums[3], ((lstart[l + 1] - lstart[l] + C - 1) / C + width - 1) / width);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int best = 0;
        for (int d = 1; d < 3; ++d)
            if (sums[d] < sums[best]) best = d;
        a->axis = 4 * (int64_t)sums[best] <= 5 * (int64_t)sums[3] && 2ULL * a->cross[best] <= a->cross[3] ? best : -1;
    }
}
__global__ void k_res_pick(int64_t n, const double4 *__restrict__ cell, const ResAxes *__restrict__ a,
                           uint32_t *__restrict__ owner) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || a->axis < 0) return;
    owner[i] = (uint32_t)a->bin[a->axis][res_bin(a, a->axis, res_coord(cell[i], a->axis))];
}
__global__ void k_res_iota(int64_t m, int32_t *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < m) out[i] = (int32_t)i;
}

__global__ void k_res_slots(int64_t n, const int32_t *__restrict__ rows, const uint32_t *__restrict__ owner,
                            const int32_t *__restrict__ cta_ptr, const int32_t *__restrict__ perm,
                            uint16_t *__restrict__ slot_of, int32_t *__restrict__ nat) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int32_t i = rows[p];
    slot_of[i] = (uint16_t)(p - cta_ptr[owner[i]]);
    if (nat) nat[p] = perm[i];
}

// An item is a row's forward (row) or backward (n + row) computation.  Its sort
// key is (CTA, level), a CTA's backward levels after its forward ones and one
// more key at its end; mask: the other CTAs that read its value.
struct ResPattern {
    int64_t n;
    const int32_t *ptr[2], *col[2], *level[2];
    int32_t nlev[2];
    __host__ __device__ int32_t keys() const { return nlev[0] + nlev[1] + 1; }
};
// *bad: a dependency on another cluster (the plan does not apply).
__global__ void k_res_keys(ResPattern a, int C, const uint32_t *__restrict__ owner, uint32_t *__restrict__ key,
                           uint32_t *__restrict__ mask, int32_t *__restrict__ bad) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 2 * a.n) return;
    const int d = t >= a.n ? 1 : 0;
    const int64_t i = t - d * a.n;
    const uint32_t o = owner[i];
    key[t] = o * (uint32_t)a.keys() + (uint32_t)(a.level[d][i] + (d ? a.nlev[0] : 0));
    for (int e = a.ptr[d][i]; e < a.ptr[d][i + 1]; ++e) {
        const int32_t j = a.col[d][e];
        if (owner[j] == o) continue;
        atomicOr(&mask[d * a.n + j], 1u << (o % C));
        if (owner[j] / C != o / C) *bad = 1;
    }
}

// Readers of every item, steps of every key (but a CTA's last one, k_res_pad).
__global__ void k_res_counts(int64_t items, const uint32_t *__restrict__ mask, int32_t *__restrict__ nread, int32_t nk,
                             int32_t per_cta, const int32_t *__restrict__ first, int width,
                             int32_t *__restrict__ nstep) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= items) nread[i] = i < items ? __popc(mask[i]) : 0;
    if (i > nk) return;
    if (i == nk) nstep[i] = 0;
    else if ((i + 1) % per_cta != 0) nstep[i] = (first[i + 1] - first[i] + width - 1) / width;
}
// A CTA's last key holds the empty steps that make its number of steps a
// multiple of `sets`.  One warp per CTA.
__global__ void k_res_pad(int32_t per_cta, int sets, int32_t *__restrict__ nstep) {
    const int64_t k0 = (int64_t)blockIdx.x * per_cta;
    int sum = 0;
    for (int k = threadIdx.x; k < per_cta - 1; k += 32) sum += nstep[k0 + k];
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (threadIdx.x == 0) nstep[k0 + per_cta - 1] = (sets - sum % sets) % sets;
}

// Halo slots: an item read by CTA c takes the next free slot of c.
__global__ void k_res_halo(int64_t n, const uint32_t *__restrict__ owner, const uint32_t *__restrict__ mask,
                           const int32_t *__restrict__ poff, int32_t *__restrict__ hcount,
                           uint16_t *__restrict__ hslot, int32_t per_cta, int C, int ctas,
                           const int32_t *__restrict__ soff, int32_t *__restrict__ step_ptr) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= ctas) step_ptr[i] = soff[i * per_cta];
    if (i >= 2 * n) return;
    const uint32_t first = owner[i >= n ? i - n : i] / C * C;  // its cluster's first CTA
    int k = poff[i];
    for (uint32_t m = mask[i]; m; m &= m - 1) {
        const int h = atomicAdd(&hcount[first + __ffs(m) - 1], 1);
        hslot[k++] = (uint16_t)min(h, 65535);  // a count past the limit makes the plan inapplicable
    }
}

// The slot of the p-th item in key order, its dependencies and readers.
__global__ void k_res_compose(ResPattern a, int C, int ml, int width, int zero, const uint32_t *__restrict__ key,
                              const int32_t *__restrict__ item, const int32_t *__restrict__ first,
                              const int32_t *__restrict__ soff, const uint32_t *__restrict__ owner,
                              const uint16_t *__restrict__ slot_of, const uint32_t *__restrict__ mask,
                              const int32_t *__restrict__ poff, const uint16_t *__restrict__ hslot,
                              int32_t *__restrict__ slot_item, uint16_t *__restrict__ slot_dep,
                              uint32_t *__restrict__ slot_push, uint32_t *__restrict__ push) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= 2 * a.n) return;
    const int32_t t = item[p];
    const int d = t >= a.n ? 1 : 0;
    const int64_t i = t - d * a.n;
    const uint32_t o = owner[i];
    const int64_t s = (int64_t)soff[key[p]] * width + (p - first[key[p]]);
    const int e0 = a.ptr[d][i], m = a.ptr[d][i + 1] - e0;
    const int hbase = zero + 2;
    uint32_t meta = 0;
    slot_item[s] = t;
    for (int q = 0; q < ml; ++q) {
        uint16_t c = (uint16_t)zero;
        if (q < m) {
            const int32_t j = a.col[d][e0 + q];
            if (owner[j] == o) {
                c = slot_of[j];
            } else {
                const int64_t u = d * a.n + j;
                c = (uint16_t)(hbase + hslot[poff[u] + __popc(mask[u] & ((1u << (o % C)) - 1u))]);
            }
        }
        slot_dep[s * ml + q] = c;
    }
    uint32_t p0 = 0;
    int k = poff[t];
    const int nr = __popc(mask[t]);
    for (uint32_t b = mask[t]; b; b &= b - 1, ++k) {
        const uint32_t code = ((uint32_t)(__ffs(b) - 1) << 16) | (uint32_t)(hbase + hslot[k]);
        if (k == poff[t])
            p0 = code;
        else
            push[k] = code;
    }
    if (nr) meta |= kResPush | ((uint32_t)(poff[t] + 1) << 8) | ((uint32_t)(nr - 1) << 4);
    slot_push[2 * s] = p0;
    slot_push[2 * s + 1] = meta;
}

template <typename T, int ML>
__global__ void k_res_records(fv_resident p, int64_t n, bool unit_fwd, const int32_t *__restrict__ lp,
                              const int32_t *__restrict__ up, const T *__restrict__ lv, const T *__restrict__ uv,
                              const T *__restrict__ dinv, uint4 *__restrict__ rec) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= p.nslots) return;
    constexpr int PL = (int)(sizeof(fv_res_rec<T, ML>) / 16);
    union U {
        fv_res_rec<T, ML> r;
        uint4 q[PL];
        __device__ U() {}
    } u;
#pragma unroll
    for (int k = 0; k < PL; ++k) u.q[k] = make_uint4(0, 0, 0, 0);
    const int32_t t = p.slot_item[s];
    const bool live = t >= 0, bwd = t >= n;
    const int64_t i = live ? t - (bwd ? n : 0) : 0;
    const int32_t *ptr = bwd ? up : lp;
    const T *val = bwd ? uv : lv;
    const int e0 = live ? ptr[i] : 0, m = live ? ptr[i + 1] - e0 : 0;
#pragma unroll
    for (int q = 0; q < ML; ++q) {
        u.r.val[q] = q < m ? val[e0 + q] : T(0);
        u.r.dep[q] = live ? p.slot_dep[s * ML + q] : (uint16_t)p.cap;
    }
    u.r.d = live && (bwd || !unit_fwd) ? dinv[i] : T(1);
    u.r.self = live ? p.slot_of[i] : (uint16_t)(p.cap + 1);
    u.r.push0 = live ? p.slot_push[2 * s] : 0;
    u.r.meta = live ? p.slot_push[2 * s + 1] : 0;
    const int64_t step = s / p.width;
#pragma unroll
    for (int k = 0; k < PL; ++k) rec[(step * PL + k) * p.width + (s - step * p.width)] = u.q[k];
}

// ------------------------------------------------------------------ the apply
template <typename T, int ML, int S>
__global__ void __launch_bounds__(kResThreads, 1) k_resident_apply(const __grid_constant__ fv_res_args a, const T *__restrict__ r,
                                                                   T *__restrict__ z, const int *skip, fv_row_skip rs,
                                                                   int *err) {
    if (skip && *(volatile const int *)skip) return;  // the same answer in every CTA of the cluster
    extern __shared__ __align__(128) unsigned char res_smem[];
    __shared__ unsigned long long bars[kResBars];
    fv_res_cta<T, ML, S> cta(a, res_smem, bars);
    fv_cluster_arrive();  // no push before every CTA's halo is reset
    cta.load(r);
    fv_cluster_wait();
    cta.sweeps(err);
    fv_cluster_arrive();  // a CTA leaves only when no other can still push into its halo
    cta.store(z, rs);
    fv_cluster_wait();
}

// Bytes of a record, steps per copy.
size_t res_rec_bytes(int ml, size_t tb) {
    return fv_res_dispatch(ml, 2, [&](auto M, auto) {
        return tb == 8 ? sizeof(fv_res_rec<double, M()>) : sizeof(fv_res_rec<float, M()>);
    });
}
int res_group(const fv_resident *p, size_t tb) {
    int g = p->sets;  // a multiple of the thread sets
    while (g < 16 && (size_t)(2 * g * p->width) * res_rec_bytes(p->ml, tb) <= (size_t)kResGroupBytes) g *= 2;
    return g;
}

template <typename T>
int res_launchable(const fv_resident *p) {
    return fv_res_dispatch(p->ml, p->sets, [&](auto M, auto S) {
        return fv_res_launchable(k_resident_apply<T, M(), S()>, p->C, fv_resident_smem(p, sizeof(T)));
    });
}

constexpr int kResMaxCtas = 160;  // CTAs of all clusters
constexpr size_t kResSparseBytes = 64u << 20;  // records of a plan of mostly idle slots, at most

// Shares the problems out over clusters: the cluster size whose fullest CTA has
// the fewest rows, problems to the emptiest cluster in descending size.
fv_status res_share_problems(const fv_resident_problems &q, int levels, int &C, int &width, int &clusters,
                             std::vector<int32_t> &cluster) {
    try {
        std::vector<int> order(q.n);
        for (int k = 0; k < q.n; ++k) order[k] = k;
        auto rows = [&](int k) { return q.offsets[k + 1] - q.offsets[k]; };
        std::sort(order.begin(), order.end(), [&](int x, int y) { return rows(x) != rows(y) ? rows(x) > rows(y) : x < y; });
        int64_t best = INT64_MAX;
        for (int c = 1; c <= kResMaxCta; c *= 2) {
            // clusters resident at once with one CTA per SM (148 SMs; a cluster stays within a GPC)
            const int most = c == 1 ? 148 : c == 2 ? 74 : c == 4 ? 33 : c == 8 ? 15 : 7;
            const int k = std::min(most, q.n);
            std::vector<int64_t> load(k, 0);
            std::vector<int32_t> to(q.n);
            for (int t : order) {
                const int at = (int)(std::min_element(load.begin(), load.end()) - load.begin());
                load[at] += rows(t);
                to[t] = at;
            }
            const int64_t full = (*std::max_element(load.begin(), load.end()) + c - 1) / c;
            if (full < best - best / 8) {  // larger clusters hand more values over
                best = full;
                C = c;
                clusters = k;
                cluster = to;
            }
        }
        width = 32;
        const int64_t lw = best / std::max(1, levels);
        while (width < 256 && 2 * lw > width) width *= 2;
        return FV_OK;
    } catch (const std::bad_alloc &) {
        return FV_ERR_ALLOC;
    }
}

// Arrays laid out in one allocation.
struct Layout {
    size_t bytes = 0;
    size_t take(size_t b) {
        const size_t o = bytes;
        bytes += (b + 255) / 256 * 256;
        return o;
    }
};

}  // namespace

size_t fv_resident_smem(const fv_resident *p, size_t tb) {
    return (size_t)kResBuffers * res_group(p, tb) * p->width * res_rec_bytes(p->ml, tb) +
           (size_t)(p->cap + 2 + p->halo) * tb;
}

fv_res_args fv_resident_args(const fv_resident *p, const void *rec, size_t tb) {
    fv_res_args a;
    a.rec = (const uint4 *)rec;
    a.push = p->push;
    a.step_ptr = p->step_ptr;
    a.cta_ptr = p->cta_ptr;
    a.rows = p->nat ? p->nat : p->rows;
    a.C = p->C * p->clusters;
    a.cap = p->cap;
    a.halo = p->halo;
    a.width = p->width;
    a.group = res_group(p, tb);
    return a;
}

void fv_resident_free(fv_resident *p) {
    if (!p) return;
    fv_blocks_free(p->arena, 2);
    delete p;
}

size_t fv_resident_record_bytes(const fv_resident *p, size_t tb) { return (size_t)p->nslots * res_rec_bytes(p->ml, tb); }

// How to go on when the shared memory of the buffers and the rows does not fit:
// the rows over twice the CTAs (65,522-row IC(0), 362 levels, on 4 CTAs with half the
// sets and on 8: 170 -> 111 us per apply), then half the thread sets and with them
// half the buffers (105,456-row ILU(0): 204 us per apply with level chunks, 122 this
// way).
struct ResTry {
    bool more_ctas = false;
    int half_sets = 0;
    // found by the last try: shared memory was all that it lacked; its CTAs, the bytes of their rows and halos
    bool full = false;
    int C = 0;
    size_t rows = 0;
};

static fv_status res_build(const fv_resident_src &s, cudaStream_t st, fv_resident **out,
                           const fv_resident_problems *problems, ResTry &t) {
    *out = nullptr;
    const bool again = t.full;
    t.full = false;
    const int64_t n = s.n;
    if (n <= 0 || n > (problems ? 148 : kResMaxCta) * 20000LL || s.max_side > 6 || !s.fwd_level || !s.bwd_level)
        return FV_OK;
    if (problems && !s.sorted) return FV_OK;
    const int64_t lw = n / std::max(1, s.n_fwd_levels);  // rows per level
    int C = 1, width = 32;
    while (C < kResMaxCta && n > (int64_t)C * 18000) C *= 2;  // shared memory for the rows
    // Narrow levels (long chains, channels): one step holds a level, so the rows go
    // to the CTAs in bands of levels.  Dealt over the CTAs each level would be
    // handed over and every row fill a step of its own (4 KB of records per row
    // with 16 rows per level on 16 CTAs).  us per apply, dealt / in bands / level
    // chunks: 100,000-row IC(0) 16 rows per level 1,662 / 998 / 11,749, 64 rows 494 /
    // 301 / 2,940; 30,000 rows, 32 per level 249 / 187 / 1,851.  Above 64 rows a band's
    // steps are 128 wide with four thread sets, and a 2D mesh (24,200 rows, 110 per
    // level: 77 / 99) is better dealt, unless that leaves four slots to a row.  Rows
    // sorted by level have their own rule below; chains among them do not.
    const bool narrow = !problems && (s.sorted ? lw <= 32 && n > 12000 : lw <= 64 || (lw <= 128 && lw < 8 * C));
    const bool wide = s.sorted && !narrow;
    // Rows sorted by level in one cluster: few wide levels, which more than 5,000
    // rows a CTA take longer than consecutive rows on all SMs.  us per apply with
    // 23 of launch and check, resident against consecutive: 32,768-row IC(0) 41 47,
    // 80,000 rows 48 49, 131,072 rows 59 50; ILU(0) 24,576 rows 47 62, 82,944 62 62.
    if (wide && !problems && n > kResMaxCta * 5000LL) return FV_OK;
    // CTAs: enough shared memory for the rows, and as few as keep a level of a
    // CTA within 128 rows (natural order: more CTAs only add hand-offs) or as
    // many as leave it 32 (rows sorted by level: few, wide levels).  Measured as
    // us per apply, the launch and its status check (23 us) included:
    // 48,000-row ILU(0), natural, C x width: 4x128 79, 8x128 87, 16x64 100, 16x32
    // 105; 32,768-row IC(0), sorted: 16x256 40, 16x128 41, 8x128 50, 8x64 49
    // (consecutive rows 47).
    while (C < kResMaxCta && lw > (int64_t)C * (wide ? 32 : 128)) C *= 2;
    if (t.more_ctas && !problems) C = std::min(2 * C, kResMaxCta);
    while (width < (wide ? 256 : 128) && lw * (wide ? 2 : 1) > (int64_t)(narrow ? 1 : C) * width) width *= 2;
    std::vector<int32_t> cluster;  // of every problem
    int clusters = 1;
    if (problems) FV_TRY(res_share_problems(*problems, s.n_fwd_levels, C, width, clusters, cluster));
    // entries per record: a padded one costs a dependent subtraction and its bytes
    // (131,072-row IC(0) in natural order with 3 and 2 per side: 146 and 145 us per
    // apply; the whole solve 94.2 and 92.7 ms)
    const int ml = s.max_side <= 2 ? 2 : s.max_side <= 3 ? 3 : s.max_side <= 4 ? 4 : 6, ctas = C * clusters;
    // Thread sets: with four, the unpacking of a record (some 500 cycles) sets the
    // pace of a 100-cycle step; eight of up to 64 threads hide it.  Four -> eight,
    // us per apply in natural order: 8,192-row IC(0), 128 levels, 59 -> 48;
    // 131,072 rows, 512 levels, 149 -> 145.
    const int sets = (width > 64 ? 512 / width : 8) >> t.half_sets;
    if (sets < 2) return FV_OK;
    fv_resident *p = new (std::nothrow) fv_resident();
    if (!p) return FV_ERR_ALLOC;
    p->C = C;
    p->clusters = clusters;
    p->width = width;
    p->sets = sets;
    p->ml = ml;
    p->cap = (int32_t)((n + ctas - 1) / ctas);  // at least
    const size_t buffers = fv_resident_smem(p, sizeof(double)) - (size_t)(p->cap + 2) * sizeof(double);
    const size_t rows = again && t.C == C ? t.rows : (size_t)(p->cap + 2) * sizeof(double);
    if (buffers + rows > kResSmem) {
        t.full = true;
        t.C = C;
        t.rows = rows;
        delete p;
        return FV_OK;
    }
    ResPattern a;
    a.n = n;
    a.ptr[0] = s.l_ptr, a.ptr[1] = s.u_ptr;
    a.col[0] = s.l_col, a.col[1] = s.u_col;
    a.level[0] = s.fwd_level, a.level[1] = s.bwd_level;
    a.nlev[0] = s.n_fwd_levels, a.nlev[1] = s.n_bwd_levels;
    const double4 *cell = narrow || wide || problems || ctas == 1 ? nullptr : s.cell;
    const int64_t items = 2 * n, nk = (int64_t)ctas * a.keys(), nnz = s.nnz_l + s.nnz_u;
    const int64_t cm = std::max(items, nk) + 2;
    Layout pl, tl;
    const size_t o_cta = pl.take(4 * (ctas + 1)), o_rows = pl.take(4 * n), o_nat = pl.take(s.perm ? 4 * n : 0),
                 o_slot = pl.take(2 * n), o_sptr = pl.take(4 * (ctas + 1)), o_push = pl.take(4 * (nnz + 1));
    const size_t t_owner = tl.take(4 * n), t_iota = tl.take(4 * items), t_key = tl.take(4 * items),
                 t_sorted = tl.take(4 * items), t_item = tl.take(4 * items), t_cnt = tl.take(4 * cm),
                 t_cnt2 = tl.take(4 * cm), t_hc = tl.take(4 * (ctas + 1)), t_prob = tl.take(problems ? 12 * (size_t)problems->n : 0), t_axes = tl.take(sizeof(ResAxes)),
                 t_hist = tl.take(cell ? 12 * (size_t)C * a.nlev[0] : 0), t_lst = tl.take(4 * (a.nlev[0] + 2)),
                 t_mask = tl.take(4 * items), t_poff = tl.take(4 * (items + 1)), t_hslot = tl.take(2 * (nnz + 1)),
                 t_first = tl.take(4 * (nk + 1)), t_soff = tl.take(4 * (nk + 1));
    size_t sort_bytes = 0, scan_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, (const uint32_t *)nullptr, (uint32_t *)nullptr,
                                    (const int32_t *)nullptr, (int32_t *)nullptr, (int)items, 0, 32, st);
    cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (const int32_t *)nullptr, (int32_t *)nullptr, (int)cm, st);
    size_t cub_bytes = std::max(sort_bytes, scan_bytes);
    const size_t t_cub = tl.take(cub_bytes);
    char *plan = nullptr, *tmp = nullptr;
    cudaError_t e = fv_block_alloc(&plan, pl.bytes);
    p->arena[0] = plan;
    if (e == cudaSuccess) e = fv_malloc_async(&tmp, tl.bytes, st);
    auto fail = [&]() {
        fv_internal_set_cuda_error(e, "resident sweep plan");
        if (tmp) cudaFreeAsync(tmp, st);
        fv_resident_free(p);
        return e == cudaErrorMemoryAllocation ? FV_ERR_ALLOC : FV_ERR_CUDA;
    };
    if (e != cudaSuccess) return fail();
    p->cta_ptr = (int32_t *)(plan + o_cta);
    p->rows = (int32_t *)(plan + o_rows);
    p->nat = s.perm ? (int32_t *)(plan + o_nat) : nullptr;
    p->slot_of = (uint16_t *)(plan + o_slot);
    p->step_ptr = (int32_t *)(plan + o_sptr);
    p->push = (uint32_t *)(plan + o_push);
    auto i32 = [&](size_t o) { return (int32_t *)(tmp + o); };
    auto u32 = [&](size_t o) { return (uint32_t *)(tmp + o); };
    uint32_t *owner = u32(t_owner), *key = u32(t_key), *sorted = u32(t_sorted), *mask = u32(t_mask);
    int32_t *iota = i32(t_iota), *hc = i32(t_hc), *lst = i32(t_lst), *first = i32(t_first), *soff = i32(t_soff);
    int32_t *item = i32(t_item), *poff = i32(t_poff), *cnt = i32(t_cnt), *cnt2 = i32(t_cnt2);
    uint16_t *hslot = (uint16_t *)(tmp + t_hslot);
    void *cubt = tmp + t_cub;
    auto grid = [](int64_t m) { return (unsigned)((m + 255) / 256); };
    auto bits_of = [](int64_t keys) {
        int b = 1;
        while (b < 31 && (1LL << b) < keys) ++b;
        return b;
    };
    auto sort = [&](const uint32_t *k, int32_t *v, int64_t m, int64_t keys) {
        if (e == cudaSuccess)
            e = cub::DeviceRadixSort::SortPairs(cubt, cub_bytes, k, sorted, iota, v, (int)m, 0, bits_of(keys), st);
    };
    e = cudaMemsetAsync(hc, 0, 4 * (ctas + 1), st);  // the last entry: a dependency between clusters
    if (e == cudaSuccess) e = cudaMemsetAsync(mask, 0, 4 * items, st);
    fv_note_launch(), k_res_level_start<<<grid(n + 1), 256, 0, st>>>(n, a.nlev[0], s.fwd_order, s.fwd_level, lst);
    fv_note_launch(), k_res_iota<<<grid(items), 256, 0, st>>>(items, iota);
    if (problems) {
        const int np = problems->n;
        int32_t *root0 = i32(t_prob), *nroot = root0 + np, *dcl = root0 + 2 * np;
        if (e == cudaSuccess) e = cudaMemsetAsync(root0, 0x7F, 4 * (size_t)np, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(nroot, 0, 4 * (size_t)np, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(dcl, cluster.data(), 4 * (size_t)np, cudaMemcpyHostToDevice, st);
        fv_note_launch(), k_res_root_count<<<grid(n), 256, 0, st>>>(n, lst, s.perm, problems->of_row, root0, nroot);
        fv_note_launch(), k_res_owner_batch<<<grid(n), 256, 0, st>>>(n, C, s.perm, problems->of_row, dcl, root0, nroot,
                                                                     s.l_ptr, s.l_col, owner);
    } else if (ctas == 1) {
        if (e == cudaSuccess) e = cudaMemsetAsync(owner, 0, 4 * n, st);
    } else if (wide) {
        fv_note_launch(), k_res_owner_sorted<<<grid(n), 256, 0, st>>>(n, C, lst, s.l_ptr, s.l_col, owner);
    } else {
        int32_t *hist = i32(t_hist);
        ResAxes *ax = (ResAxes *)(tmp + t_axes);
        const unsigned gs = std::min(grid(n), 296u);
        if (cell) {
            if (e == cudaSuccess) e = cudaMemsetAsync(hist, 0, 12 * (size_t)C * a.nlev[0], st);
            fv_note_launch(), k_res_axes_init<<<1, 256, 0, st>>>(ax);
            fv_note_launch(), k_res_extent<<<gs, 256, 0, st>>>(n, cell, ax);
            fv_note_launch(), k_res_bins<<<gs, 256, 0, st>>>(n, cell, ax);
            fv_note_launch(), k_res_cuts<<<1, 96, 0, st>>>(n, C, ax);
        }
        fv_note_launch(), k_res_owner<<<grid(n), 256, 0, st>>>(n, C, narrow, a.nlev[0], s.fwd_order, s.fwd_level, lst,
                                                               cell, ax, owner, hist);
        if (cell) {
            fv_note_launch(), k_res_cross<<<gs, 256, 0, st>>>(n, s.l_ptr, s.l_col, cell, owner, ax);
            fv_note_launch(), k_res_choose<<<1, 256, 0, st>>>(C, width, a.nlev[0], lst, hist, ax);
            fv_note_launch(), k_res_pick<<<grid(n), 256, 0, st>>>(n, cell, ax, owner);
        }
    }
    sort(owner, p->rows, n, ctas);
    fv_note_launch(), k_res_bounds<<<grid(n + 1), 256, 0, st>>>(n, ctas, sorted, p->cta_ptr);
    fv_note_launch(), k_res_slots<<<grid(n), 256, 0, st>>>(n, p->rows, owner, p->cta_ptr, s.perm, p->slot_of, p->nat);
    fv_note_launch(), k_res_keys<<<grid(items), 256, 0, st>>>(a, C, owner, key, mask, hc + ctas);
    sort(key, item, items, nk);
    fv_note_launch(), k_res_bounds<<<grid(items + 1), 256, 0, st>>>(items, (int32_t)nk, sorted, first);
    fv_note_launch(), k_res_counts<<<grid(cm), 256, 0, st>>>(items, mask, cnt, (int32_t)nk, a.keys(), first, width,
                                                             cnt2);
    fv_note_launch(), k_res_pad<<<ctas, 32, 0, st>>>(a.keys(), sets, cnt2);
    if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(cubt, cub_bytes, cnt, poff, (int)(items + 1), st);
    if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(cubt, cub_bytes, cnt2, soff, (int)(nk + 1), st);
    fv_note_launch(), k_res_halo<<<grid(std::max<int64_t>(items, ctas + 1)), 256, 0, st>>>(
                          n, owner, mask, poff, hc, hslot, a.keys(), C, ctas, soff, p->step_ptr);
    int32_t h_cta[kResMaxCtas + 1], h_hc[kResMaxCtas + 1], h_sptr[kResMaxCtas + 1];
    if (e == cudaSuccess) e = cudaMemcpyAsync(h_sptr, p->step_ptr, 4 * (ctas + 1), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h_cta, p->cta_ptr, 4 * (ctas + 1), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h_hc, hc, 4 * (ctas + 1), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail();
    for (int c = 0; c < ctas; ++c) {
        p->cap = std::max(p->cap, h_cta[c + 1] - h_cta[c]);
        p->halo = std::max(p->halo, h_hc[c]);
    }
    p->nslots = (int64_t)h_sptr[ctas] * width;
    const bool small = fv_resident_smem(p, sizeof(double)) <= kResSmem;
    const bool fits = !h_hc[ctas] && p->cap + p->halo + 2 < 65536 && small && res_launchable<double>(p) > 0 &&
                      res_launchable<float>(p) > 0;
    if (!fits) {
        t.full = !h_hc[ctas] && !small;
        t.C = C;
        t.rows = (size_t)(p->cap + 2 + p->halo) * sizeof(double);
        cudaFreeAsync(tmp, st);
        fv_resident_free(p);
        return FV_OK;
    }
    // A step is filled by a level of 32 rows or more.  Below 7 rows per level the
    // idle slots are most of what the plan holds (64 bytes a slot and more, where
    // the factor has some 100 a row), so only small plans are let be that sparse;
    // the others' rows are swept by level chunks.
    if (p->nslots > 5 * items && fv_resident_record_bytes(p, sizeof(double)) > kResSparseBytes) {
        cudaFreeAsync(tmp, st);
        fv_resident_free(p);
        return FV_OK;
    }
    // Orders without locality (a random numbering, an unstructured mesh's own): the
    // levels are few and wide and most rows' values go to other CTAs, so a step
    // waits on hand-offs.  Fitted over 2D and 3D meshes of 8,000-180,000 rows in
    // random and block-wise random orders (within 7 % in the median): an apply takes
    // 33 us + (0.114 + 0.193 h) per step with h halo slots per row, level chunks 33 us +
    // 1.0-3 per level.  us per apply, resident / level chunks: 64,800-row IC(0) random
    // 85 / 54 (h 2.7, 80 steps, 22 levels), 63,888-row ILU(0) 100 / 63, 180,000 rows in
    // random blocks of 512 110 / 89 (h 1.0, 190 steps, 24 levels); kept: 105,800 rows in
    // such blocks 62 / 87 (h 1.0, 120 steps, 24 levels), 48,000 75 / 87.  Up to 30,000
    // rows whole iterations in the cluster win with any order (24,200 rows random, CG:
    // 44 / 68 us each).
    if (!problems && n > 30000) {
        int steps = 0;
        for (int c = 0; c < ctas; ++c) steps = std::max(steps, h_sptr[c + 1] - h_sptr[c]);
        const double h = (double)p->halo / p->cap;
        if (h > 0.95 && steps * (0.114 + 0.193 * h) > (h > 1.05 ? 1.0 : 2.2) * (a.nlev[0] + a.nlev[1])) {
            cudaFreeAsync(tmp, st);
            fv_resident_free(p);
            return FV_OK;
        }
    }
    Layout sl;
    const size_t s_item = sl.take(4 * p->nslots), s_dep = sl.take(2 * (size_t)p->ml * p->nslots),
                 s_push = sl.take(8 * p->nslots);
    e = fv_block_alloc(&p->arena[1], sl.bytes);
    if (e != cudaSuccess) return fail();
    p->slot_item = (int32_t *)((char *)p->arena[1] + s_item);
    p->slot_dep = (uint16_t *)((char *)p->arena[1] + s_dep);
    p->slot_push = (uint32_t *)((char *)p->arena[1] + s_push);
    e = cudaMemsetAsync(p->slot_item, 0xFF, 4 * p->nslots, st);
    fv_note_launch(), k_res_compose<<<grid(items), 256, 0, st>>>(a, C, p->ml, width, p->cap, sorted, item, first, soff,
                                                                 owner, p->slot_of, mask, poff, hslot, p->slot_item,
                                                                 p->slot_dep, p->slot_push, p->push);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return fail();
    cudaFreeAsync(tmp, st);
    *out = p;
    return FV_OK;
}

fv_status fv_resident_build(const fv_resident_src &s, cudaStream_t st, fv_resident **out,
                            const fv_resident_problems *problems) {
    ResTry t;
    FV_TRY(res_build(s, st, out, problems, t));
    if (t.full && !problems) {
        t.more_ctas = true;
        FV_TRY(res_build(s, st, out, problems, t));
    }
    while (t.full) {  // ends with less than two sets
        ++t.half_sets;
        FV_TRY(res_build(s, st, out, problems, t));
    }
    return FV_OK;
}

template <typename T>
cudaError_t fv_resident_records(const fv_resident *p, const fv_resident_src &s, bool unit_fwd, const T *l_val,
                                const T *u_val, const T *dinv, void *rec, cudaStream_t st) {
    fv_res_dispatch(p->ml, 2, [&](auto M, auto) {
        fv_note_launch(), k_res_records<T, M()><<<(unsigned)((p->nslots + 255) / 256), 256, 0, st>>>(
                              *p, s.n, unit_fwd, s.l_ptr, s.u_ptr, l_val, u_val, dinv, (uint4 *)rec);
        return 0;
    });
    return cudaGetLastError();
}

template <typename T>
cudaError_t fv_resident_apply(const fv_resident *p, const void *rec, const T *r, T *z, const int *skip,
                              const fv_row_skip &rs, int *err, cudaStream_t st) {
    return fv_res_dispatch(p->ml, p->sets, [&](auto M, auto S) {
        cudaLaunchAttribute at;
        const cudaLaunchConfig_t cfg = fv_res_config(p->C, fv_resident_smem(p, sizeof(T)), st, &at, p->clusters);
        fv_note_launch();
        const cudaError_t e = cudaLaunchKernelEx(&cfg, k_resident_apply<T, M(), S()>,
                                                 fv_resident_args(p, rec, sizeof(T)), r, z, skip, rs, err);
        return e == cudaSuccess ? cudaGetLastError() : e;
    });
}

template cudaError_t fv_resident_records<double>(const fv_resident *, const fv_resident_src &, bool, const double *,
                                                 const double *, const double *, void *, cudaStream_t);
template cudaError_t fv_resident_records<float>(const fv_resident *, const fv_resident_src &, bool, const float *,
                                                const float *, const float *, void *, cudaStream_t);
template cudaError_t fv_resident_apply<double>(const fv_resident *, const void *, const double *, double *,
                                               const int *, const fv_row_skip &, int *, cudaStream_t);
template cudaError_t fv_resident_apply<float>(const fv_resident *, const void *, const float *, float *, const int *,
                                              const fv_row_skip &, int *, cudaStream_t);
