// Resident triangular sweeps: one thread-block cluster applies M^-1 with the
// whole vector in (distributed) shared memory.
//
// What bounds the level-chunk sweeps on small systems is the hand-off of a
// level through L2 (0.8-1.1 us per level, whatever its width).  Here every
// CTA of a cluster owns a set of rows and keeps their slots of the vector in
// its shared memory; it walks its rows level by level, each step one row per
// thread, and the few values that other CTAs need are pushed into halo slots
// of their shared memory (st.shared::cluster), where the consumer polls its own
// copy.  The vector is updated in place: right-hand side, forward result and
// backward result occupy the same slot, so nothing but the factor's records
// streams from memory.  A level costs 0.11-0.13 us: operands from shared
// memory (30 cycles), the row's FP64 chain (40), one store and one barrier.
//
// Measured per apply (both sweeps; level chunks -> resident): 131,072-row IC(0)
// in natural order (512 levels) 569 -> 122 us, 24,576-row ILU(0) (64 levels)
// 98 -> 28 us, 196,608-row ILU(0) (128 levels) 189 -> 52 us; 24,576-row ILU(0) in box
// order (28 wide levels; consecutive rows -> resident) 39 -> 24 us, 65,522-row IC(0)
// (18 levels) 26 -> 25 us.
//
// Rows are computed with the operations of k_sweep in the same order, so the
// results are the same bits.
//
// Forward progress: the CTAs of a cluster are co-resident.  A CTA at level L
// waits only for values of lower levels, so the CTA at the lowest level never
// waits on anything unfinished.  Every wait is bounded in time.
#pragma once

#include <type_traits>

#include "fv_internal.cuh"

// One row of a sweep: factor values, 1/diagonal (1 where the diagonal is a
// unit), the shared-memory slots of its dependencies and its own, the first
// remote reader of its value (rank << 16 | slot) and
//   meta = offset of further readers in the push table << 8 | their number << 4
//          | kResPush
// Unused entries have value 0 and read the slot that holds 0 (x - 0 * 0 keeps
// every x, signed zeros included); idle lanes of a step write the slot after it.
enum : uint32_t { kResPush = 1 };
template <typename T, int ML>
struct __align__(16) fv_res_rec {
    T val[ML];
    T d;
    uint16_t dep[ML];
    uint16_t self;
    uint32_t push0, meta;
};
static_assert(sizeof(fv_res_rec<double, 2>) == 48 && sizeof(fv_res_rec<double, 3>) == 48 && sizeof(fv_res_rec<double, 4>) == 64 &&
                  sizeof(fv_res_rec<double, 6>) == 80 && sizeof(fv_res_rec<float, 3>) == 32,
              "record sizes are multiples of 16");

constexpr int kResMaxCta = 16;  // largest cluster
constexpr size_t kResSmem = 226 * 1024;  // dynamic shared memory of a CTA (1 KB is left for static use)
// The records stream into shared memory as bulk copies of whole groups of
// steps (about 16 KB, one copy by one thread), kResBuffers groups deep: a copy
// takes about a microsecond from L2, a group of steps as long.  (Loading them
// into registers ahead of use was slower: a ring of loads per step runs out of
// the six scoreboards a warp tracks its loads with, and the unrolled code out
// of the instruction cache.)
constexpr int kResBuffers = 4;
constexpr int kResGroupBytes = 16 * 1024;
constexpr int kResBars = kResBuffers + 1;  // an mbarrier per buffer, then the word that says a copy was given up

// The plan of an apply: one cluster for a system, or several clusters, each with
// some of the independent problems of a batch.  Every CTA has one list of steps, the levels of its
// rows forward and then backward; a level is one or more steps of `width`
// slots, one row per thread, and every step ends with a barrier.
struct fv_resident {
    int C = 0, clusters = 1;       // CTAs per cluster, clusters
    int width = 0, sets = 0, ml = 0;  // rows per step, thread sets (below), entries per record
    int32_t cap = 0;               // most rows of a CTA
    int32_t halo = 0;              // most halo slots of a CTA
    int64_t nslots = 0;            // slots of all steps
    int32_t *cta_ptr = nullptr;    // [clusters * C + 1] first entry of a CTA in `rows`
    int32_t *rows = nullptr;       // slot k of CTA c holds row rows[cta_ptr[c] + k]
    int32_t *nat = nullptr;        // the same rows in the caller's numbering (null: no permutation)
    uint16_t *slot_of = nullptr;   // the slot of every row in its CTA
    int32_t *step_ptr = nullptr;   // [clusters * C + 1] first step of every CTA
    uint32_t *push = nullptr;      // further push targets, rank << 16 | slot
    int32_t *slot_item = nullptr;  // row (forward) or n + row (backward) of every slot, -1: idle
    uint16_t *slot_dep = nullptr;  // [ml] per slot
    uint32_t *slot_push = nullptr; // push0, meta per slot
    void *arena[2] = {nullptr, nullptr};  // the allocations the arrays lie in
};

__device__ __forceinline__ unsigned fv_cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void fv_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void fv_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ unsigned fv_mapa(unsigned addr, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void fv_push(unsigned addr, double v) {
    asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(fv_pack_value(v)) : "memory");
}
__device__ __forceinline__ void fv_push(unsigned addr, float v) {
    asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(fv_pack_value(v)) : "memory");
}
__device__ __forceinline__ bool fv_halo_ready(unsigned addr, double &v) {
    unsigned long long b;
    asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];" : "=l"(b) : "r"(addr) : "memory");
    v = __longlong_as_double((long long)b);
    return b != FV_SENTINEL_U64;
}
__device__ __forceinline__ bool fv_halo_ready(unsigned addr, float &v) {
    unsigned b;
    asm volatile("ld.relaxed.cluster.shared::cta.u32 %0, [%1];" : "=r"(b) : "r"(addr) : "memory");
    v = __uint_as_float(b);
    return b != FV_SENTINEL_U32;
}

// A dependency's slot.  Where it is a halo slot another CTA may write it
// meanwhile, so the load is a relaxed one for every warp: a branch to weak loads
// for the warps without halo slots cost 131,072-row IC(0) 4 % of a solve.
__device__ __forceinline__ void fv_lds_relaxed(unsigned a, double &v) {
    asm volatile("ld.relaxed.cluster.shared::cta.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void fv_lds_relaxed(unsigned a, float &v) {
    asm volatile("ld.relaxed.cluster.shared::cta.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
}

// The value of a halo slot, waited for (bounded like fv_wait_value).
template <typename T>
__device__ __noinline__ T fv_halo_value(unsigned addr, int *err) {
    T v;
    if (fv_halo_ready(addr, v)) return v;
    const unsigned long long t0 = fv_globaltimer();
    for (unsigned it = 1; !fv_halo_ready(addr, v); ++it)
        if ((it & 255u) == 0 && (*(volatile int *)err || fv_globaltimer() - t0 > FV_WAIT_LIMIT_NS)) {
            if (!*(volatile int *)err) atomicOr(err, FV_DEV_TIMEOUT);
            return T(NAN);
        }
    return v;
}

__device__ __forceinline__ uint4 fv_lds16(unsigned a) {
    uint4 v;
    asm volatile("ld.shared::cta.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void fv_lds(unsigned a, double &v) {
    asm volatile("ld.shared::cta.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void fv_lds(unsigned a, float &v) {
    asm volatile("ld.shared::cta.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void fv_sts(unsigned a, double v) {
    asm volatile("st.shared::cta.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void fv_sts(unsigned a, float v) {
    asm volatile("st.shared::cta.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// Both sweeps over this CTA's rows, in place in xs, by the first S * width
// threads of the block (the others skip it; the caller synchronises the block
// before and after).  rec: the CTA's first step, a step being `PL` planes of
// `width` 16-byte pieces (conflict-free reads); nsteps steps, `group` of them
// per copy (both multiples of S).  The S sets of threads take the steps in
// turn, and a set waits only for the step before its own (arrive / sync on the
// steps' named barriers; what lies further back is ordered through it).  While
// the others compute, a set unpacks the record of its next step, so from one
// step to the next lie only the operands' loads, the row's arithmetic and one
// store: with all threads at one barrier per step the unpacking (about 400
// cycles) set the pace.  buf: kResBuffers
// groups of records; bars: kResBars words, the mbarriers initialised with count 1;
// groups: copies made through them before, kept across calls.  A copy that does
// not land in time, or while an error is raised, ends the work: only the steps'
// barriers go on, bars[kResBuffers] is set, and the copies in flight are waited
// for (bounded) before the return.  No further call may then use the mbarriers.  halo0: first
// halo slot (the slots before it are the constant 0 and the idle lanes' slot).
template <typename T, int ML, int S>
__device__ __forceinline__ void fv_resident_sweeps(const uint4 *__restrict__ rec, int nsteps, int width, int group,
                                                   T *xs, unsigned halo0, uint4 *buf, unsigned long long *bars,
                                                   unsigned &groups, const uint32_t *__restrict__ push, int *err) {
    using R = fv_res_rec<T, ML>;
    constexpr int PL = (int)(sizeof(R) / 16);
    static_assert(S > 1, "a set waits for the one before it");
    const int set = (int)threadIdx.x / width, lane = (int)threadIdx.x - set * width;
    const int ng = (nsteps + group - 1) / group;
    const unsigned xbase = (unsigned)__cvta_generic_to_shared(xs);
    const unsigned bbase = (unsigned)__cvta_generic_to_shared(buf) + (unsigned)lane * 16u;
    const unsigned mbase = (unsigned)__cvta_generic_to_shared(bars);
    const unsigned step_bytes = (unsigned)(width * PL) * 16u;
    const unsigned g0 = groups;
    auto copy = [&](int g) {  // one thread
        if (g >= ng) return;
        const unsigned b = (g0 + g) % kResBuffers, bytes = (unsigned)min(group, nsteps - g * group) * step_bytes;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbase + 8 * b), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         bbase + b * group * step_bytes),
                     "l"(rec + (int64_t)g * group * width * PL), "r"(bytes), "r"(mbase + 8 * b)
                     : "memory");
    };
    // step k ends with barrier 1 + k % S: its set arrives, the next step's set waits
    const int after_prev = 1 + (set + S - 1) % S, after_own = 1 + set, two = 2 * width;
    auto wait_prev = [&]() {
        __syncwarp();
        asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(after_prev), "r"(two) : "memory");
    };
    auto end_own = [&]() {
        __syncwarp();
        asm volatile("barrier.cta.arrive.aligned %0, %1;" ::"r"(after_own), "r"(two) : "memory");
    };
    // whether the copy of group g lands within the limit (t0: when the wait began); heed: an error ends it too
    auto landed = [&](int g, unsigned long long &t0, bool heed) {
        const unsigned b = (g0 + g) % kResBuffers, parity = ((g0 + g) / kResBuffers) & 1u;
        unsigned done = 0;
        for (unsigned it = 0; !done; ++it) {
            asm volatile(
                "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                : "=r"(done)
                : "r"(mbase + 8 * b), "r"(parity)
                : "memory");
            if (!done && (it & 63u) == 63u) {
                if (!t0) t0 = fv_globaltimer();
                if ((heed && *(volatile int *)err) || fv_globaltimer() - t0 > FV_WAIT_LIMIT_NS) return false;
            }
        }
        return true;
    };
    union Stage {
        uint4 q[PL];
        R r;
        __device__ Stage() {}
    };
    Stage u;
    unsigned a_self = 0, a_push = 0, a_dep[ML], halo_deps = 0, slow = 0;
    // the set's next step: steps left of its group, that group's successor, its record's address
    int left = 0, g = 0, todo = nsteps / S;
    unsigned src = 0;
    bool gone = false;  // (the same in a warp) a copy was given up
    auto fetch = [&]() {
        if (todo == 0) return;
        --todo;
        if (left == 0) {  // the set's first step of group g: its copy has landed
            // the step computed last lies in group g - 1: every record of group g - 2 has been read
            if (threadIdx.x == 0 && g > 1) copy(g - 2 + kResBuffers);
            unsigned long long t0 = 0;
            gone = __any_sync(0xffffffffu, !landed(g, t0, true));
            left = group / S;
            src = bbase + ((g0 + g) % kResBuffers * group + set) * step_bytes;
            ++g;
            if (gone) {
                if (!*(volatile int *)err) atomicOr(err, FV_DEV_TIMEOUT);
                *(volatile unsigned long long *)&bars[kResBuffers] = 1;
                return;
            }
        }
        --left;
#pragma unroll
        for (int p = 0; p < PL; ++p) u.q[p] = fv_lds16(src + (unsigned)(p * width) * 16u);
        src += S * step_bytes;
        a_self = xbase + u.r.self * (unsigned)sizeof(T);
#pragma unroll
        for (int q = 0; q < ML; ++q) a_dep[q] = xbase + u.r.dep[q] * (unsigned)sizeof(T);
        // formed here for every row: a branch around them costs a level 0.015 us
        a_push = fv_mapa(xbase + (u.r.push0 & 0xFFFFu) * (unsigned)sizeof(T), u.r.push0 >> 16);
        halo_deps = 0;
#pragma unroll
        for (int q = 0; q < ML; ++q) halo_deps |= u.r.dep[q] >= halo0 ? 1u << q : 0u;
        slow = __any_sync(0xffffffffu, halo_deps != 0);
    };
    if (threadIdx.x == 0)
        for (int g = 0; g < kResBuffers; ++g) copy(g);
    fetch();
    int st = set;
    for (; st < nsteps && !gone; st += S) {
        if (st > 0) wait_prev();
        T x, xv[ML];
#pragma unroll
        for (int q = 0; q < ML; ++q) fv_lds_relaxed(a_dep[q], xv[q]);
        fv_lds(a_self, x);
        if (slow) {  // a row of this warp reads another CTA's values
            unsigned wait = 0;
#pragma unroll
            for (int q = 0; q < ML; ++q) wait |= (fv_is_sentinel(xv[q]) ? halo_deps : 0u) & (1u << q);
            if (wait) {
#pragma unroll
                for (int q = 0; q < ML; ++q)
                    if ((wait >> q) & 1u) xv[q] = fv_halo_value<T>(a_dep[q], err);
            }
        }
#pragma unroll
        for (int q = 0; q < ML; ++q) x = x - u.r.val[q] * xv[q];
        x = u.r.d * x;
        fv_sts(a_self, x);
        if (u.r.meta & kResPush) {
            fv_push(a_push, x);
            if (u.r.meta & 0xF0u) {
                for (uint32_t e = u.r.meta >> 8, last = e + ((u.r.meta >> 4) & 15u); e < last; ++e) {
                    const uint32_t t = __ldg(&push[e]);
                    fv_push(fv_mapa(xbase + (t & 0xFFFFu) * (unsigned)sizeof(T), t >> 16), x);
                }
            }
        }
        end_own();
        fetch();
    }
    for (; st < nsteps; st += S) {  // the barriers go on
        if (st > 0) wait_prev();
        end_own();
    }
    if (set == 0 && nsteps > 0) wait_prev();  // the last step's arrivals are met
    if (gone && threadIdx.x == 0) {  // it gave up group g - 1; the last copy it made is that of group g + 1
        unsigned long long t0 = 0;
        const int made = min(ng, max(kResBuffers, g - 2 + kResBuffers));
        for (int q = g - 1; q < made && landed(q, t0, false);) ++q;
    }
    groups = g0 + ng;
}

// What the kernels of a plan take.
struct fv_res_args {
    const uint4 *rec;
    const uint32_t *push;
    const int32_t *step_ptr, *cta_ptr, *rows;  // rows: in the caller's numbering
    int C, cap, halo, width, group;            // C: CTAs of all clusters
};
fv_res_args fv_resident_args(const fv_resident *p, const void *rec, size_t value_bytes);
// Dynamic shared memory of a CTA for values of this size; the kernels run
// kResThreads threads per CTA (enough to load and store the vector; the sweeps
// use sets * width of them) as one cluster of at least p->C CTAs; further CTAs
// hold no rows.
size_t fv_resident_smem(const fv_resident *p, size_t value_bytes);
constexpr int kResThreads = 512;

// A CTA's part of a plan: its shared memory and its rows.
template <typename T, int ML, int S>
struct fv_res_cta {
    static constexpr int PL = (int)(sizeof(fv_res_rec<T, ML>) / 16);
    const fv_res_args &a;
    uint4 *buf;
    T *xs;
    unsigned long long *bars;
    const int32_t *rows;
    const uint4 *rec;
    int nr, ns;
    unsigned groups = 0;

    // smem: fv_resident_smem bytes; mbar: kResBars words.  A cluster barrier has
    // to follow before the first sweeps.
    __device__ __forceinline__ fv_res_cta(const fv_res_args &args, unsigned char *smem, unsigned long long *mbar)
        : a(args), buf(reinterpret_cast<uint4 *>(smem)), bars(mbar) {
        xs = reinterpret_cast<T *>(buf + kResBuffers * a.group * a.width * PL);
        const unsigned c = blockIdx.x;  // cluster * C + rank
        const bool mine = c < (unsigned)a.C;
        const int r0 = mine ? a.cta_ptr[c] : 0, s0 = mine ? a.step_ptr[c] : 0;
        nr = mine ? a.cta_ptr[c + 1] - r0 : 0;
        ns = mine ? a.step_ptr[c + 1] - s0 : 0;
        rows = a.rows + r0;
        rec = a.rec + (int64_t)s0 * a.width * PL;
        if (threadIdx.x == 0) {
            for (int b = 0; b < kResBuffers; ++b)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(&bars[b])));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            bars[kResBuffers] = 0;
        }
        if (threadIdx.x < 2) xs[a.cap + threadIdx.x] = T(0);
        reset_halo();
    }
    // The halo's slots wait for values again: after the sweeps have read them,
    // and with a cluster barrier before the next ones push.
    __device__ __forceinline__ void reset_halo() {
        for (int k = threadIdx.x; k < a.halo; k += kResThreads) xs[a.cap + 2 + k] = fv_sentinel(T(0));
    }
    // (k0: addresses are formed at each call; hoisted out of a solver's loop they would spill)
    __device__ __forceinline__ void load(const T *r) {
        int k0 = threadIdx.x;
        asm volatile("" : "+r"(k0));
#pragma unroll 8
        for (int k = k0; k < nr; k += kResThreads) xs[k] = __ldcg(&r[__ldg(&rows[k])]);
    }
    __device__ __forceinline__ void store(T *z, const fv_row_skip &rs) {
        int k0 = threadIdx.x;
        asm volatile("" : "+r"(k0));
        if (!rs.group) {
#pragma unroll 8
            for (int k = k0; k < nr; k += kResThreads) z[__ldg(&rows[k])] = xs[k];
        } else {  // rows of a batch's converged problems keep their value
            for (int k = k0; k < nr; k += kResThreads) {
                const int32_t i = __ldg(&rows[k]);
                if (!rs.done[(int64_t)__ldg(&rs.group[i]) * rs.stride]) z[i] = xs[k];
            }
        }
    }
    // Between load and store: the block is synchronised before and after.  Once a
    // copy has been given up (err is raised then) the rows become NaN.
    __device__ __forceinline__ void sweeps(int *err) {
        const bool ended = gave_up();  // read before the barrier, written after it
        __syncthreads();
        if (!ended && (int)threadIdx.x < S * a.width)
            fv_resident_sweeps<T, ML, S>(rec, ns, a.width, a.group, xs, a.cap + 2, buf, bars, groups, a.push, err);
        __syncthreads();
        if (gave_up())
            for (int k = threadIdx.x; k < nr; k += kResThreads) xs[k] = T(NAN);
    }
    __device__ __forceinline__ bool gave_up() const { return *(volatile unsigned long long *)&bars[kResBuffers] != 0; }
};

template <typename F>
auto fv_res_dispatch(int ml, int sets, F &&f) {
    auto by_sets = [&](auto M) {
        if (sets == 8) return f(M, std::integral_constant<int, 8>());
        if (sets == 4) return f(M, std::integral_constant<int, 4>());
        return f(M, std::integral_constant<int, 2>());
    };
    if (ml == 2) return by_sets(std::integral_constant<int, 2>());
    if (ml == 3) return by_sets(std::integral_constant<int, 3>());
    if (ml == 4) return by_sets(std::integral_constant<int, 4>());
    return by_sets(std::integral_constant<int, 6>());
}

// Launch configuration of a plan's kernels on clusters of C CTAs (at: storage for its attribute).
inline cudaLaunchConfig_t fv_res_config(int C, size_t smem, cudaStream_t st, cudaLaunchAttribute *at,
                                        int clusters = 1) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(C * clusters);
    cfg.blockDim = dim3(kResThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = C;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// Sets a kernel's launch attributes; how many such clusters of it the GPU runs at once.
template <class K>
int fv_res_launchable(K *k, int C, size_t smem) {
    if (smem > kResSmem) return 0;
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = fv_res_config(C, smem, nullptr, &at);
    int nc = 0;
    const bool ok =
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmem) == cudaSuccess &&
        cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&nc, k, &cfg) == cudaSuccess;
    if (!ok) cudaGetLastError();
    return ok ? nc : 0;
}

// The symbolic side of a factor a plan is built from (all arrays on the device).
struct fv_resident_src {
    int64_t n = 0, nnz_l = 0, nnz_u = 0;
    const int32_t *l_ptr = nullptr, *l_col = nullptr, *u_ptr = nullptr, *u_col = nullptr;
    const int32_t *fwd_level = nullptr, *bwd_level = nullptr;
    const int32_t *fwd_order = nullptr;  // rows by forward level
    int32_t n_fwd_levels = 0, n_bwd_levels = 0, max_side = 0;  // max_side: longest strict-lower / strict-upper row
    bool sorted = false;                                       // rows sorted by forward level
    const int32_t *perm = nullptr;                             // caller's row of every row (null: the same)
    const double4 *cell = nullptr;                             // the rows' cell centres (null: unknown)
};

// The plan for a factor, or null when the resident sweeps do not apply (too
// many rows or entries per row, or a shape the level-chunk sweeps serve better).
// Problems of a batch: nothing couples rows of different ones.
struct fv_resident_problems {
    int n = 0;
    const int64_t *offsets = nullptr;  // host, [n + 1]: the caller's rows of every problem
    const int32_t *of_row = nullptr;   // device: the problem of every row, in the caller's numbering
};
// problems (optional): several clusters, each with whole problems; rows sorted by level only.
fv_status fv_resident_build(const fv_resident_src &s, cudaStream_t st, fv_resident **out,
                            const fv_resident_problems *problems = nullptr);
void fv_resident_free(fv_resident *p);

// Records of the factor's current values (rec: fv_resident_record_bytes of
// device memory).  unit_fwd: the forward sweep has a unit diagonal.
size_t fv_resident_record_bytes(const fv_resident *p, size_t value_bytes);
template <typename T>
cudaError_t fv_resident_records(const fv_resident *p, const fv_resident_src &s, bool unit_fwd, const T *l_val,
                                const T *u_val, const T *dinv, void *rec, cudaStream_t st);

// z = M^-1 r (one kernel); rows that rs skips keep their z.
template <typename T>
cudaError_t fv_resident_apply(const fv_resident *p, const void *rec, const T *r, T *z, const int *skip,
                              const fv_row_skip &rs, int *err, cudaStream_t st);
