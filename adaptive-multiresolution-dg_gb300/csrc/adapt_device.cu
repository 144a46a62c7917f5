// Element-set changes on the device: the adaptive loop's refine and coarsen
// (DGAdapt::refine DGAdapt.cpp:371-404, coarsen :675-688 and :982-1016,
// check_hole :1351-1385, update_leaf :1036-1063) and the neighbour lists of
// the fast transforms (DGSolution::find_ptr_vol/flx_alpt, DGSolution.cpp:675-728,
// with the predicates of Element.cpp:265-348) built from the sorted packed keys
// without a round trip through the host.
//
// The element set lives on the device as sorted packed keys (1D orders, nmax
// bits per dimension, first dimension most significant).  A key -> element
// open-addressing hash answers "is this multi-index present" in O(1); it is
// rebuilt after every change.  A refinement marks the missing children of the
// refined leaves into the hash and a list (atomic append), fills holes in one
// CTA (rounds of "every parent of a new key must exist"), and the new sorted
// key set is the merge of the old keys and the sorted new ones.  A coarsening
// decides removal by passes over the level sums from the finest down (an
// element goes when its indicator is below eta, it is not the root, and all its
// present children went), then compacts by a scan.  Each change synchronises the stream once to
// learn the new element count; everything else stays on the device.  The
// results are the host implementation's (csrc/adapt.cpp, csrc/grid.cpp): the
// same element sets, the same neighbour lists in the same order.
#include <cuda_runtime.h>

#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "amdg_internal.hpp"
#include "kernels.cuh"
#include "kernels_plan.cuh"
#include "device_alloc.cuh"
#include "launch.cuh"

using namespace amdg;

#define AMDG_CK(...)                                                                                    \
    do {                                                                                                \
        cudaError_t amdg_err_ = (__VA_ARGS__);                                                          \
        if (amdg_err_ != cudaSuccess)                                                                   \
            return fail(AMDG_ERR_CUDA, std::string(#__VA_ARGS__) + ": " + cudaGetErrorString(amdg_err_)); \
    } while (0)

namespace {

constexpr unsigned long long kEmptyKey = ~0ull;
constexpr size_t kHashSlot = sizeof(unsigned long long) + sizeof(int32_t);  // a key and its value
constexpr int kMaxLevels = 17;  // nmax <= 16

cudaStream_t stream_of(const amdg_grid* g) { return static_cast<cudaStream_t>(g->ctx->stream); }

// Statistics of one element-set change, read back by the host in one copy.
struct AdaptStats {
    unsigned long long count;     // refine: keys added; coarsen: elements kept
    unsigned long long lev_sum[kMaxDim];
    int lev_max[kMaxDim];
    int levsum_max;
    int err;                      // bit 0: a list overflowed; bit 1: hole filling did not finish
    unsigned long long missed;    // coarsen: missed refinements recorded
    int nonfinite;                // set by the indicator kernel (cleared with the indicators only)
    int topo_err;                 // set by the neighbour-list kernels (cleared when reported)
};
// refine / coarsen restart everything before `nonfinite`
constexpr size_t kStatsReset = offsetof(AdaptStats, nonfinite);

template <class T>
amdg_status grow(T** p, int64_t* cap, int64_t need, int64_t want) {
    if (need <= *cap) return AMDG_OK;
    cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    if (amdg::device_malloc(reinterpret_cast<void**>(p), size_t(want) * sizeof(T)) != cudaSuccess) {
        *p = nullptr;
        return fail(AMDG_ERR_NOMEM, "cudaMalloc failed (device adaptivity buffers)");
    }
    *cap = want;
    return AMDG_OK;
}

amdg_status grow_temp(GridDevice& d, size_t bytes) {
    if (bytes <= d.temp_bytes) return AMDG_OK;
    cudaFree(d.temp);
    d.temp = nullptr;
    d.temp_bytes = 0;
    const size_t want = bytes + bytes / 2 + 4096;
    if (amdg::device_malloc(&d.temp, want) != cudaSuccess) {
        d.temp = nullptr;
        return fail(AMDG_ERR_NOMEM, "cudaMalloc failed (sort / scan scratch)");
    }
    d.temp_bytes = want;
    return AMDG_OK;
}

amdg_status ensure_stats(GridDevice& d) {
    if (d.stats && d.host_stats) return AMDG_OK;
    if (!d.host_stats && cudaMallocHost(&d.host_stats, sizeof(AdaptStats)) != cudaSuccess) {
        d.host_stats = nullptr;
        return fail(AMDG_ERR_NOMEM, "cudaMallocHost failed (adaptivity statistics)");
    }
    if (!d.stats && amdg::device_malloc(&d.stats, sizeof(AdaptStats)) != cudaSuccess) {
        d.stats = nullptr;
        return fail(AMDG_ERR_NOMEM, "cudaMalloc failed (adaptivity statistics)");
    }
    // every field starts at zero (the error flags are only ever set, and cleared when reported)
    if (cudaMemset(d.stats, 0, sizeof(AdaptStats)) != cudaSuccess)
        return fail(AMDG_ERR_CUDA, "cudaMemset failed (adaptivity statistics)");
    std::memset(d.host_stats, 0, sizeof(AdaptStats));
    return AMDG_OK;
}

// ---- packed keys and 1D orders ------------------------------------------------
struct KeyShape {
    int dim, nmax;
    __host__ __device__ int field(uint64_t key, int d) const {
        return int((key >> (uint64_t(nmax) * (dim - 1 - d))) & ((uint64_t(1) << nmax) - 1));
    }
    __host__ __device__ uint64_t with(uint64_t key, int d, int o) const {
        const uint64_t shift = uint64_t(nmax) * (dim - 1 - d);
        const uint64_t mask = ((uint64_t(1) << nmax) - 1) << shift;
        return (key & ~mask) | (uint64_t(o) << shift);
    }
};

__host__ __device__ __forceinline__ int level_of(int o) {
#ifdef __CUDA_ARCH__
    return o == 0 ? 0 : 32 - __clz(o);
#else
    int l = 0;
    while ((1 << l) <= o) ++l;
    return l;
#endif
}
__device__ __forceinline__ int parent_of(int o) { return o == 1 ? 0 : o / 2; }
// children of 1D order o below level nmax: {1} for o = 0, {2o, 2o+1} otherwise
__device__ __forceinline__ int children_of(int o, int nmax, int* ch) {
    const int n = level_of(o);
    if (n >= nmax) return 0;
    if (o == 0) { ch[0] = 1; return 1; }
    ch[0] = 2 * o;
    ch[1] = 2 * o + 1;
    return 2;
}

// ---- key -> element hash ---------------------------------------------------------
struct KeyHash {
    unsigned long long* key;
    int32_t* val;
    uint64_t mask;
    int bits;
};

__device__ __forceinline__ uint64_t hslot(uint64_t k, int bits) { return (k * 0x9E3779B97F4A7C15ull) >> (64 - bits); }

// element index of key k (>= 0), -1 when absent or added by the current refinement; the value is
// read beside the key, not after it (a lookup is one trip to the L2 cache instead of two)
__device__ __forceinline__ int32_t hfind(const KeyHash& h, uint64_t k) {
    uint64_t s = hslot(k, h.bits);
    for (uint64_t i = 0; i <= h.mask; ++i, s = (s + 1) & h.mask) {
        const unsigned long long v = h.key[s];
        const int32_t w = h.val[s];
        if (v == kEmptyKey) return -1;
        if (v == k) return w;
    }
    return -1;
}
__device__ __forceinline__ bool hcontains(const KeyHash& h, uint64_t k) {
    uint64_t s = hslot(k, h.bits);
    for (uint64_t i = 0; i <= h.mask; ++i, s = (s + 1) & h.mask) {
        const unsigned long long v = *(volatile unsigned long long*)&h.key[s];
        if (v == kEmptyKey) return false;
        if (v == k) return true;
    }
    return false;
}
// inserts k; true when this call inserted it (slot in *slot), false when it was there
__device__ __forceinline__ bool hinsert(const KeyHash& h, uint64_t k, uint64_t* slot) {
    uint64_t s = hslot(k, h.bits);
    for (uint64_t i = 0; i <= h.mask; ++i, s = (s + 1) & h.mask) {
        const unsigned long long prev = atomicCAS(&h.key[s], kEmptyKey, (unsigned long long)k);
        if (prev == kEmptyKey) { *slot = s; return true; }
        if (prev == k) return false;
    }
    return false;  // the table is sized at least twice the keys it can receive: not reached
}

__global__ void hash_build_kernel(const uint64_t* __restrict__ keys, int64_t E, KeyHash h) {
    const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= E) return;
    uint64_t s;
    if (hinsert(h, keys[e], &s)) h.val[s] = int32_t(e);
}

// ---- indicators ----------------------------------------------------------------
// sqrt of the block's sum of squares in block order (as element_norm_kernel), plus the second
// vector's when given, added in that order (DGAdapt::indicator_norm, DGAdapt.cpp:1018-1030)
__global__ void norms_kernel(const double* __restrict__ u, const double* __restrict__ u2, int B, int64_t E,
                             double* __restrict__ out, AdaptStats* st) {
    const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= E) return;
    const double* x = u + e * B;
    double s = 0.0;
    for (int q = 0; q < B; ++q) s = __dadd_rn(s, __dmul_rn(x[q], x[q]));
    double v = sqrt(s);
    if (u2) {
        const double* y = u2 + e * B;
        double s2 = 0.0;
        for (int q = 0; q < B; ++q) s2 = __dadd_rn(s2, __dmul_rn(y[q], y[q]));
        v = __dadd_rn(v, sqrt(s2));
    }
    out[e] = v;
    if (!isfinite(v)) st->nonfinite = 1;
}

// Level statistics of the warp's keys (those with `in`): one atomic per warp and value.  One per
// element made every element of the set queue at the same few addresses.
__device__ __forceinline__ void add_level_stats(const KeyShape& ks, uint64_t key, bool in, AdaptStats* st) {
    if (!__ballot_sync(0xffffffffu, in)) return;
    const bool first = (threadIdx.x & 31) == 0;
    int sum = 0;
    for (int d = 0; d < ks.dim; ++d) {
        const int l = in ? level_of(ks.field(key, d)) : 0;
        sum += l;
        const int s = __reduce_add_sync(0xffffffffu, l), m = __reduce_max_sync(0xffffffffu, l);
        if (first) {
            atomicAdd(&st->lev_sum[d], (unsigned long long)s);
            atomicMax(&st->lev_max[d], m);
        }
    }
    sum = __reduce_max_sync(0xffffffffu, sum);
    if (first) atomicMax(&st->levsum_max, sum);
}

// ---- refinement ------------------------------------------------------------------
// Leaves (fewer present children than possible, DGAdapt::update_leaf) that want refinement get
// every missing child in every dimension (DGAdapt::refine), appended once to newk.
// `width` lanes (a power of two, 2 dim or more) share an element, one child each: the lookups of an
// element are one trip to memory, not 2 dim in a row.
__global__ void refine_mark_kernel(const uint64_t* keys, int64_t E, KeyShape ks, const double* norms, double eps,
                                   const uint8_t* force, KeyHash h, uint64_t* newk, AdaptStats* st, int64_t cap,
                                   uint8_t* refined, int width) {
    const int64_t gid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, j = lane & (width - 1);
    const int64_t e = gid / width;
    wait_for_previous();
    const bool want = e < E && (force ? force[e] != 0 : (norms[e] > eps));
    uint64_t ck = 0;
    bool child = false, there = false;
    if (want && j < 2 * ks.dim) {
        const uint64_t key = keys[e];
        int ch[2];
        const int d = j >> 1, nc = children_of(ks.field(key, d), ks.nmax, ch);
        child = (j & 1) < nc;
        if (child) {
            ck = ks.with(key, d, ch[j & 1]);
            there = hfind(h, ck) >= 0;
        }
    }
    const unsigned group = (width == 32 ? 0xffffffffu : ((1u << width) - 1u)) << (lane - j);
    const bool leaf = (__ballot_sync(0xffffffffu, child && !there) & group) != 0;
    if (e < E && j == 0) refined[e] = leaf ? 1 : 0;
    uint64_t slot;
    if (child && !there && hinsert(h, ck, &slot)) {
        const long long i = (long long)atomicAdd(&st->count, 1ull);
        if (i < cap) newk[i] = ck;
        else atomicOr(&st->err, 1);
    }
}

// Hole filling (DGAdapt::check_hole) in one CTA: every parent of a new key must be present;
// rounds over the keys the previous round added, until a round adds none.  Then the level
// statistics of the added keys.
__global__ void __launch_bounds__(1024) hole_fill_kernel(KeyShape ks, KeyHash h, uint64_t* newk, AdaptStats* st,
                                                         int64_t cap) {
    __shared__ long long s_hi;
    wait_for_previous();
    long long lo = 0;
    int round = 0;
    for (;; ++round) {
        __syncthreads();
        if (threadIdx.x == 0) s_hi = (long long)*(volatile unsigned long long*)&st->count;
        __syncthreads();
        const long long hi = s_hi < cap ? s_hi : cap;
        if (lo >= hi) break;
        if (round >= 4 * kMaxDim * kMaxLevels) {  // a hole-free closure needs at most dim * nmax rounds
            if (threadIdx.x == 0) atomicOr(&st->err, 2);
            break;
        }
        for (long long i = lo + threadIdx.x; i < hi; i += blockDim.x) {
            const uint64_t key = newk[i];
            for (int d = 0; d < ks.dim; ++d) {
                const int o = ks.field(key, d);
                if (o == 0) continue;
                const uint64_t p = ks.with(key, d, parent_of(o));
                if (hcontains(h, p)) continue;
                uint64_t slot;
                if (!hinsert(h, p, &slot)) continue;
                const long long j = (long long)atomicAdd(&st->count, 1ull);
                if (j < cap) newk[j] = p;
                else atomicOr(&st->err, 1);
            }
        }
        lo = hi;
    }
    __syncthreads();
    const long long n = s_hi < cap ? s_hi : cap;
    for (long long i0 = 0; i0 < n; i0 += blockDim.x) {  // whole warps: the sums are taken per warp
        const long long i = i0 + threadIdx.x;
        add_level_stats(ks, i < n ? newk[i] : 0, i < n, st);
    }
}

// The new element set: old and added keys, both sorted and without common keys, merged by rank (a
// key's place is its own index plus the number of the other list's keys below it).  Writes the
// keys, their 1D orders and the old element of each (-1: added).
__global__ void merge_keys_kernel(const uint64_t* old, int64_t E, const uint64_t* added, int64_t n, KeyShape ks,
                                  uint64_t* out, int32_t* map, int32_t* order) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    wait_for_previous();
    if (i >= E + n) return;
    const bool is_old = i < E;
    const uint64_t key = is_old ? old[i] : added[i - E];
    const uint64_t* other = is_old ? added : old;
    int64_t lo = 0, hi = is_old ? n : E;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (other[mid] < key) lo = mid + 1;
        else hi = mid;
    }
    const int64_t r = lo + (is_old ? i : i - E);
    out[r] = key;
    map[r] = is_old ? int32_t(i) : -1;
    for (int d = 0; d < ks.dim; ++d) order[r * ks.dim + d] = ks.field(key, d);
}

// ---- coarsening ------------------------------------------------------------------
// Elements of level sum L: removed when the indicator is below eta, some level is above 0, and
// every present child (level sum L + 1, decided by the previous pass) is removed -- the fixed
// point of DGAdapt::coarsen's repeated sweeps over childless elements.
__global__ void coarsen_pass_kernel(const uint64_t* __restrict__ keys, int64_t E, KeyShape ks,
                                    const double* __restrict__ norms, double eta, int L, KeyHash h,
                                    uint8_t* __restrict__ removed) {
    const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= E) return;
    const uint64_t key = keys[e];
    int sum = 0, mx = 0;
    for (int d = 0; d < ks.dim; ++d) {
        const int l = level_of(ks.field(key, d));
        sum += l;
        mx = l > mx ? l : mx;
    }
    if (sum != L || mx == 0 || !(norms[e] < eta)) return;
    int ch[2];
    for (int d = 0; d < ks.dim; ++d) {
        const int nc = children_of(ks.field(key, d), ks.nmax, ch);
        for (int c = 0; c < nc; ++c) {
            const int32_t i = hfind(h, ks.with(key, d, ch[c]));
            if (i >= 0 && !removed[i]) return;
        }
    }
    removed[e] = 1;
}

__global__ void keep_flags_kernel(const uint8_t* __restrict__ removed, int64_t E, int32_t* __restrict__ keep) {
    const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e < E) keep[e] = removed[e] ? 0 : 1;
    else if (e == E) keep[e] = 0;
}

// statistics of the kept set; with missed_eps > 0 the kept leaves (leaf in the kept set) whose
// indicator exceeds missed_eps are appended to `missed`
__global__ void coarsen_stats_kernel(const uint64_t* __restrict__ keys, int64_t E, KeyShape ks,
                                     const uint8_t* __restrict__ removed, const int32_t* __restrict__ pos,
                                     const double* __restrict__ norms, double missed_eps, KeyHash h,
                                     uint64_t* __restrict__ missed, int64_t missed_cap, AdaptStats* st) {
    const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e == 0) st->count = pos[E];
    const bool kept = e < E && !removed[e];
    const uint64_t key = kept ? keys[e] : 0;
    add_level_stats(ks, key, kept, st);
    if (!kept) return;
    if (missed_eps > 0.0 && norms[e] > missed_eps) {
        int existing = 0, total = 0, ch[2];
        for (int d = 0; d < ks.dim; ++d) {
            const int nc = children_of(ks.field(key, d), ks.nmax, ch);
            total += nc;
            for (int c = 0; c < nc; ++c) {
                const int32_t i = hfind(h, ks.with(key, d, ch[c]));
                existing += (i >= 0 && !removed[i]) ? 1 : 0;
            }
        }
        if (existing < total) {
            const long long j = (long long)atomicAdd(&st->missed, 1ull);
            if (j < missed_cap) missed[j] = key;
        }
    }
}

// The whole coarsening of a small element set in one CTA: the same flags, positions and statistics
// as coarsen_pass_kernel + keep_flags_kernel + the device scan + coarsen_stats_kernel, without their
// launches.  "Some child is kept" is pushed up by the kept elements, not looked up by their parents:
// an element that the indicator keeps marks its parents (a byte of shared memory each) before the
// first pass, so a pass over a level sum only reads the marks of its candidates, and only a
// candidate that stays has lookups left to do.  With every element's key read and every candidate's
// children looked up in each pass, and one atomic per element and statistic, the kernel took
// 23 us at 1,168 elements and 86 us at 3,880; it takes 14 and 24 us.
constexpr int kSmallCoarsenThreads = 1024, kSmallCoarsenItems = 8;
constexpr int64_t kSmallCoarsenMax = int64_t(kSmallCoarsenThreads) * kSmallCoarsenItems;

// inclusive scan over the lanes of a warp
template <class T>
__device__ __forceinline__ T warp_scan(T v) {
#pragma unroll
    for (int q = 1; q < 32; q <<= 1) {
        const T u = __shfl_up_sync(0xffffffffu, v, q);
        if (int(threadIdx.x & 31) >= q) v += u;
    }
    return v;
}

// sum of `mine` over the warps below this one (32 warps, one value each) and over all of them
template <class T>
__device__ __forceinline__ T warps_before(T mine, T* totals, T* all) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) totals[warp] = mine;
    __syncthreads();
    const T t = totals[lane], upto = warp_scan(t);
    *all = __shfl_sync(0xffffffffu, upto, 31);
    return __shfl_sync(0xffffffffu, upto - t, warp);
}

__global__ void __launch_bounds__(kSmallCoarsenThreads, 1)
    coarsen_small_kernel(const uint64_t* keys, int64_t E, KeyShape ks, const double* norms, double eta, int levsum_max,
                         KeyHash h, uint8_t* removed, int32_t* pos, double missed_eps, uint64_t* missed,
                         int64_t missed_cap, AdaptStats* st) {
    __shared__ uint8_t held[kSmallCoarsenMax];  // some child of the element is kept
    __shared__ uint8_t gone[kSmallCoarsenMax];  // the element is removed
    const int tid = threadIdx.x;
    wait_for_previous();
    for (int e = tid; e < int(E); e += kSmallCoarsenThreads) held[e] = gone[e] = 0;
    __syncthreads();
    auto mark_parents = [&](uint64_t key) {
        for (int d = 0; d < ks.dim; ++d) {
            const int o = ks.field(key, d);
            if (o == 0) continue;
            const int32_t p = hfind(h, ks.with(key, d, parent_of(o)));
            if (p >= 0) held[p] = 1;
        }
    };
    int level[kSmallCoarsenItems];  // level sum of a candidate, 0: no candidate
#pragma unroll
    for (int i = 0; i < kSmallCoarsenItems; ++i) {
        const int e = tid + i * kSmallCoarsenThreads;
        level[i] = 0;
        if (e >= int(E)) continue;
        const uint64_t key = keys[e];
        if (norms[e] < eta)
            for (int d = 0; d < ks.dim; ++d) level[i] += level_of(ks.field(key, d));
        if (level[i] == 0) mark_parents(key);
    }
    __syncthreads();
    for (int L = levsum_max; L >= 1; --L) {
#pragma unroll
        for (int i = 0; i < kSmallCoarsenItems; ++i) {
            if (level[i] != L) continue;
            const int e = tid + i * kSmallCoarsenThreads;
            if (held[e]) mark_parents(keys[e]);
            else gone[e] = 1;
        }
        __syncthreads();  // pass L - 1 reads the marks of pass L
    }
    // kept positions: a warp's kSmallCoarsenItems x 32 elements by ballots, then the warps' totals
    __shared__ int totals[32];
    const int lane = tid & 31, warp = tid >> 5, first = warp * 32 * kSmallCoarsenItems + lane;
    int v[kSmallCoarsenItems], mine = 0;
#pragma unroll
    for (int i = 0; i < kSmallCoarsenItems; ++i) {
        const int e = first + 32 * i;
        const unsigned kept = __ballot_sync(0xffffffffu, e < int(E) && !gone[e]);
        v[i] = mine + __popc(kept & ((1u << lane) - 1u));
        mine += __popc(kept);
    }
    int total;
    const int base = warps_before(mine, totals, &total);
#pragma unroll
    for (int i = 0; i < kSmallCoarsenItems; ++i) {
        const int e = first + 32 * i;
        if (e < int(E)) pos[e] = base + v[i];
    }
    if (tid == 0) {
        pos[E] = total;
        st->count = (unsigned long long)total;
    }
    for (int e0 = 0; e0 < int(E); e0 += kSmallCoarsenThreads) {
        const int e = e0 + tid;
        const bool kept = e < int(E) && !gone[e];
        const uint64_t key = kept ? keys[e] : 0;
        add_level_stats(ks, key, kept, st);
        if (e < int(E)) removed[e] = kept ? 0 : 1;
        if (kept && missed_eps > 0.0 && norms[e] > missed_eps) {
            int existing = 0, tot = 0, ch[2];
            for (int d = 0; d < ks.dim; ++d) {
                const int nc = children_of(ks.field(key, d), ks.nmax, ch);
                tot += nc;
                for (int c = 0; c < nc; ++c) {
                    const int32_t i = hfind(h, ks.with(key, d, ch[c]));
                    existing += (i >= 0 && !gone[i]) ? 1 : 0;
                }
            }
            if (existing < tot) {
                const long long j = (long long)atomicAdd(&st->missed, 1ull);
                if (j < missed_cap) missed[j] = key;
            }
        }
    }
}

__global__ void compact_kernel(const uint64_t* __restrict__ keys, int64_t E, KeyShape ks, const uint8_t* __restrict__ removed,
                               const int32_t* __restrict__ pos, uint64_t* __restrict__ out_keys,
                               int32_t* __restrict__ map, int32_t* __restrict__ order) {
    const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= E || removed[e]) return;
    const int32_t p = pos[e];
    const uint64_t key = keys[e];
    out_keys[p] = key;
    map[p] = int32_t(e);
    for (int d = 0; d < ks.dim; ++d) order[int64_t(p) * ks.dim + d] = ks.field(key, d);
}

__global__ void mark_keys_kernel(const uint64_t* __restrict__ list, int64_t n, KeyHash h, uint8_t* __restrict__ flag) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t e = hfind(h, list[i]);
    if (e >= 0) flag[e] = 1;
}

// ---- neighbour lists of the fast transforms ----------------------------------------
// 1D support [a, b) of order o in units of 2^-nmax (levels 0 and 1 cover the domain)
__device__ __forceinline__ void support_of(int o, int nmax, int64_t* a, int64_t* b) {
    const int n = level_of(o);
    if (n <= 1) { *a = 0; *b = int64_t(1) << nmax; return; }
    const int64_t w = int64_t(1) << (nmax - n + 1);
    *a = int64_t(o - (1 << (n - 1))) * w;
    *b = *a + w;
}

// The candidates of level l >= 2 for element support [a0, b0) (Element.cpp:283-348 as index
// ranges): the intersecting intervals first..last (vol), widened to lo..hi where an interval
// ends or starts exactly at the boundary (flx), and the intervals across the periodic boundary.
struct LevelRange {
    int cnt, first, last, lo, hi;
    bool wrap_lo, wrap_hi;  // interval 0 (across x = 1) / interval cnt - 1 (across x = 0)
};
__device__ __forceinline__ LevelRange level_range(int l, int nmax, int64_t a0, int64_t b0) {
    LevelRange r;
    const int64_t one = int64_t(1) << nmax;
    r.cnt = 1 << (l - 1);
    const int sh = nmax - l + 1;  // intervals of 2^sh units
    const int64_t in = (int64_t(1) << sh) - 1;
    r.first = int(a0 >> sh);
    r.last = int((b0 - 1) >> sh);
    r.lo = r.first;
    r.hi = r.last;
    if ((a0 & in) == 0 && r.first >= 1) --r.lo;
    if ((b0 & in) == 0 && r.last + 1 < r.cnt) ++r.hi;
    r.wrap_lo = b0 == one && r.lo > 0;
    r.wrap_hi = a0 == 0 && r.hi < r.cnt - 1;
    return r;
}

struct TopoArgs {
    const uint64_t* keys;
    int64_t E;
    KeyShape ks;
    KeyHash h;
    const uint8_t* seen;  // [order][n1]
    int n1;
};

// The candidate 1D orders of level l for a row (element, dimension t) with 1D support [a0, b0),
// in increasing order: levels 0 and 1 are the single order l (intersecting every support); at
// level l >= 2 the interval across x = 1 (when it touches the support from the periodic side),
// the intervals lo .. hi (first .. last intersect the support: vol; the ones beside them touch
// it: flx only), and the interval across x = 0.  This is the host builder's sequence
// (csrc/grid.cpp, fibre_neighbours), so the lists come out in the same order.
struct LevelCands {
    int n;                 // candidates at this level
    int base, lo, wl;      // order of candidate i: cnt if i < wl (wrap), else base + lo + i - wl, ...
    int vfirst, vlast;     // vol range (orders)
    int wrap_hi_order;     // last candidate when >= 0
};
__device__ __forceinline__ LevelCands level_cands(int l, int nmax, int64_t a0, int64_t b0) {
    LevelCands c;
    if (l <= 1) {
        c.n = 1;
        c.base = l;
        c.lo = 0;
        c.wl = 0;
        c.vfirst = c.vlast = l;
        c.wrap_hi_order = -1;
        return c;
    }
    const LevelRange r = level_range(l, nmax, a0, b0);
    c.wl = r.wrap_lo ? 1 : 0;
    c.base = r.cnt;
    c.lo = r.lo;
    c.n = c.wl + (r.hi - r.lo + 1) + (r.wrap_hi ? 1 : 0);
    c.vfirst = r.cnt + r.first;
    c.vlast = r.cnt + r.last;
    c.wrap_hi_order = r.wrap_hi ? 2 * r.cnt - 1 : -1;
    return c;
}
__device__ __forceinline__ int cand_order(const LevelCands& c, int i) {
    if (i < c.wl) return c.base;  // the interval across x = 1 (order cnt)
    if (c.wrap_hi_order >= 0 && i == c.n - 1) return c.wrap_hi_order;
    return c.base + c.lo + (i - c.wl);
}

// One warp per row (element, dimension): the candidates of all levels in one sequence, looked up 32 at a
// time, the present ones counted (out == nullptr) or written in order (ballot prefix).  Returns the
// vol / flx counts and the counts at levels up to the element's own (the split between the "U" and
// "L" parts).  The finer vol neighbours without a point of the element are written from the end
// of the list down (RowRec in kernels_plan.cuh); *skip_out is their number.  Most rows have a few candidates on each level: taken level by level, a row waited
// for nmax + 1 lookups one after the other (the fill 32 us at 3,880 elements in two dimensions, cold
// caches, 14 us at 390; 22 and 10 us with the levels in one sequence).
struct RowOut {
    int2* vol;
    int2* flx;
    int64_t vmax, fmax;  // entries the row may write (fill)
};
__device__ __forceinline__ void row_lists(const TopoArgs& A, int64_t e, int t, const RowOut* out, int* nv_out,
                                          int* nf_out, int* sv_out, int* sf_out, int* skip_out) {
    const int lane = threadIdx.x & 31;
    const int nmax = A.ks.nmax;
    const uint64_t key = A.keys[e];
    const int oi = A.ks.field(key, t), own = level_of(oi);
    int64_t a0, b0;
    support_of(oi, nmax, &a0, &b0);
    int nv = 0, nf = 0, sv = 0, sf = 0, skip = 0;
    // lane l holds the number of candidates up to level l; those of the "U" part come first
    const int upto = warp_scan(lane <= nmax ? level_cands(lane, nmax, a0, b0).n : 0);
    const int total = __shfl_sync(0xffffffffu, upto, nmax), upper = __shfl_sync(0xffffffffu, upto, own);
    for (int base = 0; base < total; base += 32) {
        const int i = base + lane;
        int l = 0, before = 0;  // level of candidate i, candidates of the levels below
        for (int q = 0; q < nmax; ++q) {
            const int u = __shfl_sync(0xffffffffu, upto, q);
            if (u <= i) {
                l = q + 1;
                before = u;
            }
        }
        int s = -1, o = 0;
        bool inv = false;
        if (i < total) {
            const LevelCands c = level_cands(l, nmax, a0, b0);
            o = cand_order(c, i - before);
            s = hfind(A.h, A.ks.with(key, t, o));
            inv = s >= 0 && o >= c.vfirst && o <= c.vlast;
        }
        const unsigned bf = __ballot_sync(0xffffffffu, s >= 0);
        const unsigned bv = __ballot_sync(0xffffffffu, inv);
        if (out) {
            const unsigned below = (1u << lane) - 1u;
            if (s >= 0) {
                const int pf = nf + __popc(bf & below);
                if (pf < out->fmax) out->flx[pf] = make_int2(s, o);
            }
            const bool last = inv && i >= upper && !A.seen[int64_t(oi) * A.n1 + o];
            const unsigned bs = __ballot_sync(0xffffffffu, last);
            if (inv) {
                const int64_t pv = last ? out->vmax - 1 - (skip + __popc(bs & below)) : nv - skip + __popc(bv & ~bs & below);
                if (pv >= 0 && pv < out->vmax) out->vol[pv] = make_int2(s, o);
            }
            skip += __popc(bs);
        }
        nf += __popc(bf);
        nv += __popc(bv);
        const int left = upper - base;
        const unsigned um = left >= 32 ? 0xffffffffu : left > 0 ? (1u << left) - 1u : 0u;
        sf += __popc(bf & um);
        sv += __popc(bv & um);
    }
    *nv_out = nv;
    *nf_out = nf;
    *sv_out = sv;
    *sf_out = sf;
    *skip_out = skip;
}

__global__ void topo_count_kernel(TopoArgs A, int32_t* vcnt, int32_t* fcnt, int32_t* long_count) {
    const int64_t row = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int dim = A.ks.dim;
    wait_for_previous();
    if (row > A.E * dim) return;  // whole warps: the row test is uniform
    if (row == A.E * dim) {
        if ((threadIdx.x & 31) == 0) vcnt[row] = fcnt[row] = 0;
        if ((threadIdx.x & 31) < kMaxDim) long_count[threadIdx.x & 31] = 0;  // the fill kernel appends
        return;
    }
    const int64_t e = row / dim;
    int nv, nf, sv, sf, skip;
    row_lists(A, e, int(row - e * dim), nullptr, &nv, &nf, &sv, &sf, &skip);
    if ((threadIdx.x & 31) == 0) {
        vcnt[row] = nv;
        fcnt[row] = nf;
    }
}

__global__ void topo_fill_kernel(TopoArgs A, const int32_t* vol_ptr, const int32_t* flx_ptr,
                                 int2* vol_nbr, int2* flx_nbr, int32_t* vol_split,
                                 int32_t* flx_split, int64_t vol_cap, int64_t flx_cap, int* err,
                                 RowRec* rows, int32_t* long_count, int32_t* long_rows,
                                 int64_t long_stride) {
    const int64_t row = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int dim = A.ks.dim;
    wait_for_previous();
    if (row >= A.E * dim) return;
    const int64_t v0 = vol_ptr[row], f0 = flx_ptr[row];
    const int64_t v1 = vol_ptr[row + 1], f1 = flx_ptr[row + 1];
    if (v1 > vol_cap || f1 > flx_cap) {  // lists beyond the arrays: write nothing
        if ((threadIdx.x & 31) == 0) {
            atomicOr(err, 1);
            const int o = A.ks.field(A.keys[row / dim], int(row % dim));
            write_row_rec(rows, row, dim, 0, 0, 0, 0, 0, 0, o, 0, long_count, long_rows, long_stride);
        }
        return;
    }
    const RowOut out{vol_nbr + v0, flx_nbr + f0, v1 - v0, f1 - f0};
    const int64_t e = row / dim;
    int nv, nf, sv, sf, skip;
    row_lists(A, e, int(row - e * dim), &out, &nv, &nf, &sv, &sf, &skip);
    if ((threadIdx.x & 31) == 0) {
        if (nv != v1 - v0 || nf != f1 - f0) atomicOr(err, 1);
        vol_split[row] = int32_t(v0 + sv);
        flx_split[row] = int32_t(f0 + sf);
        write_row_rec(rows, row, dim, int(v0), int(v0 + sv), int(v1), int(f0), int(f0 + sf), int(f1),
                      A.ks.field(A.keys[e], int(row - e * dim)), skip, long_count, long_rows, long_stride);
    }
}

// surplus ancestors anc[e][d][ic]: the element owning surplus point ic of e along d
// (LagrInterpolation::eval_fp_to_coe_D_Lag, Interplation.cpp:1318-1376); -1 for level 0
__global__ void ancestors_kernel(TopoArgs A, const int32_t* anc_order, int p1, int32_t* anc, int* err) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int dim = A.ks.dim;
    wait_for_previous();
    if (i >= A.E * dim * p1) return;
    const int64_t row = i / p1, e = row / dim;
    const int ic = int(i - row * p1), d = int(row - e * dim);
    const uint64_t key = A.keys[e];
    const int o = A.ks.field(key, d);
    int32_t s = -1;
    if (o != 0) {
        s = hfind(A.h, A.ks.with(key, d, anc_order[o * p1 + ic]));
        if (s < 0) atomicOr(err, 2);
    }
    anc[i] = s;
}

__global__ void parent_table_kernel(TopoArgs A, int32_t* __restrict__ pg) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int dim = A.ks.dim;
    if (i >= A.E * dim) return;
    const int64_t e = i / dim;
    const int d = int(i - e * dim);
    uint64_t k = A.keys[e];
    int32_t* out = pg + i * 2;
    out[0] = out[1] = -1;
    for (int gen = 0; gen < 2; ++gen) {
        const int o = A.ks.field(k, d);
        if (o == 0) break;
        k = A.ks.with(k, d, parent_of(o));
        out[gen] = hfind(A.h, k);
    }
}

inline unsigned blocks_for(int64_t n, int threads) { return unsigned((n + threads - 1) / threads); }

KeyHash hash_of(const amdg_grid* g) {
    KeyHash h;
    h.key = g->dev.hkey;
    h.val = g->dev.hval;
    h.mask = uint64_t(g->dev.hcap) - 1;
    h.bits = g->dev.hbits;
    return h;
}

amdg_status read_stats(amdg_grid* g, AdaptStats* out) {
    cudaStream_t st = stream_of(g);
    AMDG_CK(cudaMemcpyAsync(g->dev.host_stats, g->dev.stats, sizeof(AdaptStats), cudaMemcpyDeviceToHost, st));
    AMDG_CK(cudaStreamSynchronize(st));
    std::memcpy(out, g->dev.host_stats, sizeof(AdaptStats));
    if (out->topo_err) {  // reported once
        AMDG_CK(cudaMemsetAsync(&static_cast<AdaptStats*>(g->dev.stats)->topo_err, 0, sizeof(int), st));
        return fail(AMDG_ERR_STATE, out->topo_err & 2 ? "element set has a hole: a surplus ancestor is missing"
                                                      : "device neighbour list overflow");
    }
    return AMDG_OK;
}

// Learned pre-adaptation flags (amdg_burgers_adaptive_step_learned): the classifier's "refine"
// (class 0) where its largest probability is at least tau, the surplus criterion where it is
// unsure (or everywhere without a classifier).  counts[0] += refined by the network,
// counts[1] += unsure.
__global__ void learned_flags_kernel(const float* __restrict__ prob, int64_t E, float tau,
                                     const double* __restrict__ norms, double eps, uint8_t* __restrict__ force,
                                     unsigned long long* counts) {
    const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= E) return;
    uint8_t f;
    if (!prob) {
        f = norms[e] > eps ? 1 : 0;
        atomicAdd(&counts[1], 1ull);
    } else {
        const float* p = prob + 3 * e;
        int arg = 0;
        for (int q = 1; q < 3; ++q)
            if (p[q] > p[arg]) arg = q;
        if (p[arg] < tau) {
            f = norms[e] > eps ? 1 : 0;
            atomicAdd(&counts[1], 1ull);
        } else if (arg == 0) {
            f = 1;
            atomicAdd(&counts[0], 1ull);
        } else {
            f = 0;
        }
    }
    force[e] = f;
}

amdg_status ensure_flags(amdg_grid* g, int64_t E) {
    GridDevice& d = g->dev;
    if (E + 1 <= d.flag_cap) return AMDG_OK;
    cudaFree(d.flag);
    cudaFree(d.force);
    cudaFree(d.pos);
    d.flag = d.force = nullptr;
    d.pos = nullptr;
    d.flag_cap = 0;
    const int64_t want = E + E / 2 + 64;
    if (amdg::device_malloc(&d.flag, size_t(want)) != cudaSuccess || amdg::device_malloc(&d.force, size_t(want)) != cudaSuccess ||
        amdg::device_malloc(&d.pos, size_t(want) * sizeof(int32_t)) != cudaSuccess)
        return fail(AMDG_ERR_NOMEM, "cudaMalloc failed (adaptivity flags)");
    d.flag_cap = want;
    return AMDG_OK;
}

}  // namespace

namespace amdg {

void grid_host_level_stats(amdg_grid* g) {
    const int dim = g->host.dim;
    for (int d = 0; d < kMaxDim; ++d) {
        g->lev_max[d] = 0;
        g->lev_sum[d] = 0;
    }
    g->levsum_max = 0;
    for (int64_t e = 0; e < g->host.num_elements; ++e) {
        int s = 0;
        for (int d = 0; d < dim; ++d) {
            const int l = level_of(g->host.order[size_t(e) * dim + d]);
            s += l;
            g->lev_sum[d] += l;
            g->lev_max[d] = std::max(g->lev_max[d], l);
        }
        g->levsum_max = std::max(g->levsum_max, s);
    }
}

// both key arrays hold at least E keys (the swaps keep them the same size); with `preserve` the
// current keys are carried over when they move
static amdg_status ensure_keys(amdg_grid* g, int64_t E, bool preserve) {
    GridDevice& d = g->dev;
    if (E <= d.key_cap && d.key && d.key_alt) return AMDG_OK;
    const int64_t want = std::max<int64_t>(E + E / 4 + 16, d.key_cap);
    uint64_t *k = nullptr, *a = nullptr;
    if (amdg::device_malloc(&k, size_t(want) * sizeof(uint64_t)) != cudaSuccess ||
        amdg::device_malloc(&a, size_t(want) * sizeof(uint64_t)) != cudaSuccess) {
        cudaFree(k);
        return fail(AMDG_ERR_NOMEM, "cudaMalloc failed (element keys)");
    }
    const int64_t n = g->host.num_elements;
    cudaStream_t st = stream_of(g);
    if (preserve && n > 0 && d.key) AMDG_CK(cudaMemcpyAsync(k, d.key, size_t(n) * sizeof(uint64_t), cudaMemcpyDeviceToDevice, st));
    AMDG_CK(cudaStreamSynchronize(st));
    cudaFree(d.key);
    cudaFree(d.key_alt);
    d.key = k;
    d.key_alt = a;
    d.key_cap = want;
    return AMDG_OK;
}

amdg_status grid_upload_keys(amdg_grid* g) {
    const int64_t E = g->host.num_elements;
    if (amdg_status s = ensure_keys(g, E, false); s != AMDG_OK) return s;
    if (E > 0)
        AMDG_CK(cudaMemcpyAsync(g->dev.key, g->host.key.data(), size_t(E) * sizeof(uint64_t), cudaMemcpyHostToDevice,
                                stream_of(g)));
    g->dev.hash_version = -1;
    g->host_stale = false;
    grid_host_level_stats(g);
    return AMDG_OK;
}

amdg_status grid_ensure_host(const amdg_grid* cg) {
    amdg_grid* g = const_cast<amdg_grid*>(cg);
    if (!g->host_stale) return AMDG_OK;
    const int64_t E = g->host.num_elements;
    std::vector<uint64_t> keys(static_cast<size_t>(E));
    cudaStream_t st = stream_of(g);
    if (E > 0) AMDG_CK(cudaMemcpyAsync(keys.data(), g->dev.key, size_t(E) * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    AMDG_CK(cudaStreamSynchronize(st));
    const int sparse = g->host.sparse;
    grid_from_keys(g->host.dim, g->host.nmax, g->host.k, std::move(keys), &g->host);
    g->host.sparse = sparse;
    g->host_stale = false;
    return AMDG_OK;
}

amdg_status grid_hash(amdg_grid* g) {
    GridDevice& d = g->dev;
    if (d.hash_version == g->version) return AMDG_OK;
    const int64_t E = g->host.num_elements;
    // room for the element set and everything one refinement can add (at most 2 dim children of
    // existing elements per element), at most half full
    const int64_t need = 2 * (1 + 2 * int64_t(g->host.dim)) * std::max<int64_t>(E, 1);
    if (need > d.hcap) {
        cudaFree(d.hkey);
        d.hkey = nullptr;
        d.hval = nullptr;
        d.hcap = 0;
        int bits = 6;
        while ((int64_t(1) << bits) < need + need / 2) ++bits;
        const int64_t cap = int64_t(1) << bits;
        // the values lie behind the keys: one fill empties both
        if (amdg::device_malloc(reinterpret_cast<void**>(&d.hkey), size_t(cap) * kHashSlot) != cudaSuccess)
            return fail(AMDG_ERR_NOMEM, "cudaMalloc failed (element hash)");
        d.hval = reinterpret_cast<int32_t*>(d.hkey + cap);
        d.hcap = cap;
        d.hbits = bits;
    }
    cudaStream_t st = stream_of(g);
    AMDG_CK(cudaMemsetAsync(d.hkey, 0xFF, size_t(d.hcap) * kHashSlot, st));
    if (E > 0) {
        hash_build_kernel<<<blocks_for(E, 256), 256, 0, st>>>(d.key, E, hash_of(g));
        AMDG_CK(cudaGetLastError());
        g->ctx->launches++;
    }
    d.hash_version = g->version;
    return AMDG_OK;
}

amdg_status grid_device_norms(amdg_grid* g, const double* d_u, const double* d_u2) {
    const int64_t E = g->host.num_elements;
    if (amdg_status s = ensure_stats(g->dev); s != AMDG_OK) return s;
    if (E > g->norms_capacity) {
        cudaFree(g->d_norms);
        g->d_norms = nullptr;
        g->norms_capacity = 0;
        const int64_t cap = E + E / 4 + 16;
        if (amdg::device_malloc(reinterpret_cast<void**>(&g->d_norms), size_t(cap) * sizeof(double)) != cudaSuccess)
            return fail(AMDG_ERR_NOMEM, "cudaMalloc failed (indicators)");
        g->norms_capacity = cap;
    }
    cudaStream_t st = stream_of(g);
    AMDG_CK(cudaMemsetAsync(g->dev.stats, 0, offsetof(AdaptStats, topo_err), st));
    if (E > 0) {
        norms_kernel<<<blocks_for(E, 128), 128, 0, st>>>(d_u, d_u2, g->block, E, g->d_norms,
                                                         static_cast<AdaptStats*>(g->dev.stats));
        AMDG_CK(cudaGetLastError());
        g->ctx->launches++;
    }
    return AMDG_OK;
}

amdg_status grid_reserve_remap(amdg_grid* g, int64_t E) {
    const int64_t grown = E + E / 4 + 16;
    auto regrow = [&](double** p, int64_t* cap) -> amdg_status {
        if (E <= *cap) return AMDG_OK;
        cudaFree(*p);
        *p = nullptr;
        *cap = 0;
        if (amdg::device_malloc(reinterpret_cast<void**>(p), size_t(grown) * g->block * sizeof(double)) != cudaSuccess)
            return fail(AMDG_ERR_NOMEM, "cudaMalloc failed (coefficient remap)");
        *cap = grown;
        return AMDG_OK;
    };
    amdg_status s;
    if ((s = regrow(&g->d_u_spare, &g->spare_capacity)) != AMDG_OK) return s;
    if (g->d_v && (s = regrow(&g->d_v_spare, &g->v_spare_capacity)) != AMDG_OK) return s;
    if (g->d_pred && (s = regrow(&g->d_pred_spare, &g->pred_spare_capacity)) != AMDG_OK) return s;
    if (g->d_pred_v && (s = regrow(&g->d_pred_v_spare, &g->pred_v_spare_capacity)) != AMDG_OK) return s;
    return AMDG_OK;
}

amdg_status grid_apply_remap(amdg_grid* g, int64_t E) {
    cudaStream_t st = stream_of(g);
    if (amdg_status s = grid_reserve_remap(g, E); s != AMDG_OK) return s;
    AMDG_CK(launch_remap(g->d_u, g->d_map, g->block, E, g->d_u_spare, st));
    g->ctx->launches++;
    if (g->d_v) {
        AMDG_CK(launch_remap(g->d_v, g->d_map, g->block, E, g->d_v_spare, st));
        g->ctx->launches++;
        std::swap(g->d_v, g->d_v_spare);
        std::swap(g->v_capacity, g->v_spare_capacity);
    }
    if (g->d_pred) {
        AMDG_CK(launch_remap(g->d_pred, g->d_map, g->block, E, g->d_pred_spare, st));
        g->ctx->launches++;
        std::swap(g->d_pred, g->d_pred_spare);
        std::swap(g->pred_capacity, g->pred_spare_capacity);
    }
    if (g->d_pred_v) {
        AMDG_CK(launch_remap(g->d_pred_v, g->d_map, g->block, E, g->d_pred_v_spare, st));
        g->ctx->launches++;
        std::swap(g->d_pred_v, g->d_pred_v_spare);
        std::swap(g->pred_v_capacity, g->pred_v_spare_capacity);
    }
    std::swap(g->d_u, g->d_u_spare);
    std::swap(g->capacity, g->spare_capacity);
    g->host.num_elements = E;
    g->dof = E * g->block;
    g->version++;
    return AMDG_OK;
}

// map, order and key arrays for E_new elements (grow-only)
static amdg_status ensure_set_arrays(amdg_grid* g, int64_t E) {
    const int64_t grown = E + E / 4 + 16;
    if (E > g->map_capacity) {
        cudaFree(g->d_map);
        g->d_map = nullptr;
        g->map_capacity = 0;
        if (amdg::device_malloc(reinterpret_cast<void**>(&g->d_map), size_t(grown) * sizeof(int32_t)) != cudaSuccess)
            return fail(AMDG_ERR_NOMEM, "cudaMalloc failed (element map)");
        g->map_capacity = grown;
    }
    if (E > g->order_capacity) {  // the current set's orders move along (a failure later leaves them intact)
        int32_t* p = nullptr;
        if (amdg::device_malloc(&p, size_t(grown) * g->host.dim * sizeof(int32_t)) != cudaSuccess)
            return fail(AMDG_ERR_NOMEM, "cudaMalloc failed (element orders)");
        const int64_t n = g->host.num_elements * g->host.dim;
        cudaStream_t st = stream_of(g);
        if (n > 0) AMDG_CK(cudaMemcpyAsync(p, g->d_order, size_t(n) * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
        AMDG_CK(cudaStreamSynchronize(st));
        cudaFree(g->d_order);
        g->d_order = p;
        g->order_capacity = grown;
    }
    return AMDG_OK;
}

amdg_status grid_device_refine(amdg_grid* g, double eps, const uint8_t* d_force, int8_t* refined, int64_t* added) {
    const KeyShape ks{g->host.dim, g->host.nmax};
    const int64_t E = g->host.num_elements;
    GridDevice& d = g->dev;
    amdg_status s;
    if ((s = ensure_stats(d)) != AMDG_OK || (s = grid_hash(g)) != AMDG_OK || (s = ensure_flags(g, E)) != AMDG_OK)
        return s;
    // added keys are children of existing elements: at most 2 dim per element
    const int64_t cap = 2 * int64_t(ks.dim) * E + 16;
    if ((s = grow(&d.newk, &d.new_cap, cap, cap + cap / 4)) != AMDG_OK) return s;
    cudaStream_t st = stream_of(g);
    AdaptStats* dst = static_cast<AdaptStats*>(d.stats);
    AMDG_CK(cudaMemsetAsync(dst, 0, kStatsReset, st));
    // the marks put the added keys into the hash: it no longer holds the element set alone, and a call that
    // fails below must not leave it for the next one, which would take those keys for already marked
    d.hash_version = -1;
    if (E > 0) {
        int width = 2;  // lanes per element: 12 -> 6 us at 2,104 elements in three dimensions
        while (width < 2 * ks.dim) width *= 2;
        AMDG_CK(launch_after(refine_mark_kernel, dim3(blocks_for(E * width, 128)), 128, 0, st, d.key, E, ks,
                             d_force ? nullptr : g->d_norms, eps, d_force, hash_of(g), d.newk, dst, d.new_cap, d.flag,
                             width));
        AMDG_CK(launch_after(hole_fill_kernel, dim3(1), 1024, 0, st, ks, hash_of(g), d.newk, dst, d.new_cap));
        g->ctx->launches += 2;
    }
    AdaptStats hs;
    if ((s = read_stats(g, &hs)) != AMDG_OK) return s;
    if (hs.nonfinite) return fail(AMDG_ERR_NONFINITE, "element indicator is not finite");
    if (hs.err) return fail(AMDG_ERR_STATE, "device refinement: key list overflow or unfinished hole filling");
    if (refined && E > 0) {
        AMDG_CK(cudaMemcpyAsync(refined, d.flag, size_t(E), cudaMemcpyDeviceToHost, st));
        AMDG_CK(cudaStreamSynchronize(st));
    }
    const int64_t n_new = hs.count;
    if (added) *added = n_new;
    if (n_new == 0) {
        d.hash_version = g->version;
        return AMDG_OK;
    }
    const int64_t En = E + n_new;
    if (En > (int64_t(1) << 31) - 1) return fail(AMDG_ERR_CAPACITY, "more than 2^31-1 elements");
    // every allocation before the first change, so a failure leaves the element set as it was
    if ((s = ensure_keys(g, En, true)) != AMDG_OK || (s = ensure_set_arrays(g, En)) != AMDG_OK ||
        (s = grid_reserve_remap(g, En)) != AMDG_OK)
        return s;
    // only the added keys are sorted (keys use dim * nmax bits), into the scratch behind the sort's own
    const int bits = ks.dim * ks.nmax;
    const size_t list = (size_t(n_new) * sizeof(uint64_t) + 255) / 256 * 256;
    size_t temp = 0;
    AMDG_CK(cub::DeviceRadixSort::SortKeys(nullptr, temp, d.newk, d.newk, int(n_new), 0, bits, st));
    if ((s = grow_temp(d, list + temp)) != AMDG_OK) return s;
    uint64_t* sorted = static_cast<uint64_t*>(d.temp);
    AMDG_CK(cub::DeviceRadixSort::SortKeys(static_cast<char*>(d.temp) + list, temp, d.newk, sorted, int(n_new), 0, bits, st));
    AMDG_CK(launch_after(merge_keys_kernel, dim3(blocks_for(En, 128)), 128, 0, st, d.key, E, sorted, n_new, ks, d.key_alt,
                         g->d_map, g->d_order));
    g->ctx->launches += 2;
    std::swap(d.key, d.key_alt);
    if ((s = grid_apply_remap(g, En)) != AMDG_OK) return s;
    for (int k = 0; k < ks.dim; ++k) {
        g->lev_sum[k] += hs.lev_sum[k];
        g->lev_max[k] = std::max(g->lev_max[k], hs.lev_max[k]);
    }
    g->levsum_max = std::max(g->levsum_max, hs.levsum_max);
    g->host_stale = true;
    return AMDG_OK;
}

amdg_status grid_device_coarsen(amdg_grid* g, double eta, double missed_eps, int64_t* removed_out) {
    const KeyShape ks{g->host.dim, g->host.nmax};
    const int64_t E = g->host.num_elements;
    GridDevice& d = g->dev;
    amdg_status s;
    if ((s = ensure_stats(d)) != AMDG_OK || (s = grid_hash(g)) != AMDG_OK || (s = ensure_flags(g, E)) != AMDG_OK)
        return s;
    if (missed_eps > 0 && (s = grow(&d.missed, &d.missed_cap, E, E + E / 4 + 16)) != AMDG_OK) return s;
    cudaStream_t st = stream_of(g);
    AdaptStats* dst = static_cast<AdaptStats*>(d.stats);
    AMDG_CK(cudaMemsetAsync(dst, 0, kStatsReset, st));
    if (E == 0) {
        if (removed_out) *removed_out = 0;
        return AMDG_OK;
    }
    if (E <= kSmallCoarsenMax) {  // one CTA does it all
        AMDG_CK(launch_after(coarsen_small_kernel, dim3(1), kSmallCoarsenThreads, 0, st, d.key, E, ks, g->d_norms, eta,
                             g->levsum_max, hash_of(g), d.flag, d.pos, missed_eps, d.missed, d.missed_cap, dst));
        g->ctx->launches++;
    } else {
        AMDG_CK(cudaMemsetAsync(d.flag, 0, size_t(E), st));
        for (int L = g->levsum_max; L >= 1; --L) {
            coarsen_pass_kernel<<<blocks_for(E, 128), 128, 0, st>>>(d.key, E, ks, g->d_norms, eta, L, hash_of(g),
                                                                    d.flag);
            AMDG_CK(cudaGetLastError());
            g->ctx->launches++;
        }
        // kept positions: exclusive scan of keep flags (E + 1 entries, the last one 0 -> total)
        keep_flags_kernel<<<blocks_for(E + 1, 256), 256, 0, st>>>(d.flag, E, d.pos);
        AMDG_CK(cudaGetLastError());
        size_t temp = 0;
        AMDG_CK(cub::DeviceScan::ExclusiveSum(nullptr, temp, d.pos, d.pos, int(E + 1), st));
        if ((s = grow_temp(d, temp)) != AMDG_OK) return s;
        size_t tb = d.temp_bytes;
        AMDG_CK(cub::DeviceScan::ExclusiveSum(d.temp, tb, d.pos, d.pos, int(E + 1), st));
        coarsen_stats_kernel<<<blocks_for(E, 128), 128, 0, st>>>(d.key, E, ks, d.flag, d.pos, g->d_norms, missed_eps,
                                                                 hash_of(g), d.missed, d.missed_cap, dst);
        AMDG_CK(cudaGetLastError());
        g->ctx->launches += 3;
    }
    AdaptStats hs;
    if ((s = read_stats(g, &hs)) != AMDG_OK) return s;
    if (hs.nonfinite) return fail(AMDG_ERR_NONFINITE, "element indicator is not finite");
    const int64_t En = hs.count;
    if (missed_eps > 0) d.n_missed = std::min<int64_t>(hs.missed, d.missed_cap);
    if (removed_out) *removed_out = E - En;
    if (En == E) return AMDG_OK;
    if ((s = ensure_keys(g, En, true)) != AMDG_OK || (s = ensure_set_arrays(g, En)) != AMDG_OK ||
        (s = grid_reserve_remap(g, En)) != AMDG_OK)
        return s;
    compact_kernel<<<blocks_for(E, 256), 256, 0, st>>>(d.key, E, ks, d.flag, d.pos, d.key_alt, g->d_map, g->d_order);
    AMDG_CK(cudaGetLastError());
    g->ctx->launches++;
    std::swap(d.key, d.key_alt);
    if ((s = grid_apply_remap(g, En)) != AMDG_OK) return s;
    for (int k = 0; k < ks.dim; ++k) {
        g->lev_sum[k] = hs.lev_sum[k];
        g->lev_max[k] = hs.lev_max[k];
    }
    g->levsum_max = hs.levsum_max;
    g->host_stale = true;
    return AMDG_OK;
}

amdg_status grid_learned_flags(amdg_grid* g, const float* d_prob, double tau, double eps, uint8_t** d_force,
                               unsigned long long* d_counts) {
    const int64_t E = g->host.num_elements;
    if (amdg_status s = ensure_flags(g, E); s != AMDG_OK) return s;
    *d_force = g->dev.force;
    if (E == 0) return AMDG_OK;
    learned_flags_kernel<<<blocks_for(E, 128), 128, 0, stream_of(g)>>>(d_prob, E, float(tau), g->d_norms, eps,
                                                                      g->dev.force, d_counts);
    AMDG_CK(cudaGetLastError());
    g->ctx->launches++;
    return AMDG_OK;
}

int* grid_topology_error_flag(amdg_grid* g) {
    if (ensure_stats(g->dev) != AMDG_OK) return nullptr;
    return &static_cast<AdaptStats*>(g->dev.stats)->topo_err;
}

amdg_status grid_check_topology(amdg_grid* g) {
    if (amdg_status s = ensure_stats(g->dev); s != AMDG_OK) return s;
    AdaptStats hs;
    return read_stats(g, &hs);
}

amdg_status grid_mark_missed(amdg_grid* g, uint8_t* d_force) {
    if (g->dev.n_missed == 0) return AMDG_OK;
    if (amdg_status s = grid_hash(g); s != AMDG_OK) return s;
    mark_keys_kernel<<<blocks_for(g->dev.n_missed, 128), 128, 0, stream_of(g)>>>(g->dev.missed, g->dev.n_missed,
                                                                                hash_of(g), d_force);
    AMDG_CK(cudaGetLastError());
    g->ctx->launches++;
    return AMDG_OK;
}

void transform_topology_bounds(const amdg_grid* g, int64_t* vol_pairs, int64_t* flx_pairs) {
    // |vol(e, t)| = level_t(e) + 1 ancestors (itself included) + its present descendants; over a
    // hole-free set every ancestor relation is counted from both ends: E + 2 sum_e level_t(e).
    // flx adds at most 4 touching intervals per level >= 2.
    const int64_t E = g->host.num_elements;
    int64_t v = 0;
    for (int t = 0; t < g->host.dim; ++t) v += E + 2 * g->lev_sum[t];
    *vol_pairs = v;
    *flx_pairs = v + 4 * int64_t(std::max(g->host.nmax - 1, 0)) * E * g->host.dim;
}

// Exclusive scans of the vol and flx row counts (n entries each) in one CTA, for small element
// sets: the results of the two device-wide scans without their launches.  Both counts of a row in
// one 64-bit sum (the lists hold fewer than 2^31 entries each); a warp scans consecutive rows, 32
// side by side, so that its loads and stores are whole lines (eight consecutive rows per thread and
// one scan per array: 11 us at 7,761 rows, cold caches; 8 us this way).
__global__ void __launch_bounds__(kSmallCoarsenThreads, 1)
    scan_pair_small_kernel(const int32_t* a, const int32_t* b, int64_t n, int32_t* sa, int32_t* sb) {
    __shared__ unsigned long long totals[32];
    const int items = int((n + kSmallCoarsenThreads - 1) / kSmallCoarsenThreads);  // rows per thread
    const int first = (threadIdx.x >> 5) * 32 * items + (threadIdx.x & 31);
    unsigned long long v[kSmallCoarsenItems], mine = 0;
    wait_for_previous();
#pragma unroll
    for (int i = 0; i < kSmallCoarsenItems; ++i) {
        const int r = first + 32 * i;
        v[i] = i < items && r < int(n) ? (unsigned long long)(unsigned(b[r])) << 32 | unsigned(a[r]) : 0ull;
    }
#pragma unroll
    for (int i = 0; i < kSmallCoarsenItems; ++i) {
        if (i >= items) break;
        const unsigned long long upto = warp_scan(v[i]);
        v[i] = mine + upto - v[i];
        mine += __shfl_sync(0xffffffffu, upto, 31);
    }
    unsigned long long total;
    const unsigned long long base = warps_before(mine, totals, &total);
#pragma unroll
    for (int i = 0; i < kSmallCoarsenItems; ++i) {
        const int r = first + 32 * i;
        if (i < items && r < int(n)) {
            sa[r] = int32_t(unsigned(base + v[i]));
            sb[r] = int32_t((base + v[i]) >> 32);
        }
    }
}

amdg_status device_transform_topology(amdg_grid* g, const DeviceTopoOut& out, int32_t* d_cnt, void* stream) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (amdg_status s = grid_hash(g); s != AMDG_OK) return s;
    const int64_t E = g->host.num_elements;
    const int dim = g->host.dim;
    const int64_t rows = E * dim;
    TopoArgs A{g->dev.key, E, KeyShape{dim, g->host.nmax}, hash_of(g), out.seen, out.n1};
    // counts of the vol rows in d_cnt[0 .. rows], of the flx rows in d_cnt[rows + 1 ..]
    int32_t* vcnt = d_cnt;
    int32_t* fcnt = d_cnt + rows + 1;
    AMDG_CK(launch_after(topo_count_kernel, dim3(blocks_for(32 * (rows + 1), 256)), 256, 0, st, A, vcnt, fcnt,
                         out.long_count));
    if (rows + 1 <= kSmallCoarsenMax) {
        AMDG_CK(launch_after(scan_pair_small_kernel, dim3(1), kSmallCoarsenThreads, 0, st, vcnt, fcnt, rows + 1,
                             out.vol_ptr, out.flx_ptr));
    } else {
        size_t temp = 0;
        AMDG_CK(cub::DeviceScan::ExclusiveSum(nullptr, temp, vcnt, out.vol_ptr, int(rows + 1), st));
        if (amdg_status s = grow_temp(g->dev, temp); s != AMDG_OK) return s;
        size_t tb = g->dev.temp_bytes;
        AMDG_CK(cub::DeviceScan::ExclusiveSum(g->dev.temp, tb, vcnt, out.vol_ptr, int(rows + 1), st));
        tb = g->dev.temp_bytes;
        AMDG_CK(cub::DeviceScan::ExclusiveSum(g->dev.temp, tb, fcnt, out.flx_ptr, int(rows + 1), st));
    }
    AMDG_CK(launch_after(topo_fill_kernel, dim3(blocks_for(32 * rows, 256)), 256, 0, st, A, out.vol_ptr, out.flx_ptr,
                         reinterpret_cast<int2*>(out.vol_nbr), reinterpret_cast<int2*>(out.flx_nbr), out.vol_split,
                         out.flx_split, out.vol_cap, out.flx_cap, out.err, static_cast<RowRec*>(out.rows),
                         out.long_count, out.long_rows, out.long_stride));
    AMDG_CK(launch_after(ancestors_kernel, dim3(blocks_for(rows * out.p1, 128)), 128, 0, st, A, out.anc_order, out.p1,
                         out.anc, out.err));
    g->ctx->launches += 6;
    return AMDG_OK;
}

amdg_status device_parent_table(amdg_grid* g, int32_t* d_pg, void* stream) {
    if (amdg_status s = grid_hash(g); s != AMDG_OK) return s;
    const int64_t E = g->host.num_elements;
    const int dim = g->host.dim;
    if (E == 0) return AMDG_OK;
    TopoArgs A{g->dev.key, E, KeyShape{dim, g->host.nmax}, hash_of(g), nullptr, 0};
    parent_table_kernel<<<blocks_for(E * dim, 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(A, d_pg);
    AMDG_CK(cudaGetLastError());
    g->ctx->launches++;
    return AMDG_OK;
}

}  // namespace amdg
