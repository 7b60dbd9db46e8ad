// rs_prep.cu -- the query path's input preparation on the GPU: the unique-edge payload of
// EdgePreprocessor::extractEdges (preprocess/src/EdgePreprocessor.cpp:41-119), byte for
// byte.
//
// Every edge of every valid triangle (triangle order; edges v0v1, v1v2, v2v0) is a record
// r = 3 t + e.  Its key is the ordered pair (k0 <= k1) of its endpoints quantised with
// llround(double(x) * 1e5), and the reference's std::map orders keys lexicographically.
// Each run of equal keys is one unique edge: its first record gives the endpoints in that
// record's own orientation, and the run's objects, deduplicated in first-seen order, are the
// sources -- the reference's first-occurrence rules.
//
// The vertices are sorted, not the records: there are a sixth as many, and a record's key is
// then the pair of its endpoints' ranks (equal quantised positions share one).  The records
// are listed by their lower rank -- a counting pass, a scan and a fill, a handful of records
// a list -- and each list is sorted by (higher rank, record) on its own, so the runs come out
// in the map's order.  Lists of up to kBucketSmall records take a thread, up to kBucketBig a
// block; an input with a longer one is left to the records path, which sorts all records, by
// the two ranks in one word, and then by (run, object).  An input with more vertices than
// records goes there at once, by packed quantised keys in wide words.  3.2 M triangles of 1.6 M
// vertices: 6.1 ms by wide words, 1.2 by vertices.
#include <algorithm>
#include <climits>

#include "rs_engine.h"
#include "rs_prims.cuh"

namespace rs {
namespace {

constexpr int kPT = 256;

__device__ __forceinline__ void quantise(const float* __restrict__ V, uint32_t v, long long q[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) q[k] = llround((double)V[3 * (uint64_t)v + k] * 1e5);
}

__device__ __forceinline__ bool less3(const long long* a, const long long* b) {
    return a[0] < b[0] || (a[0] == b[0] && (a[1] < b[1] || (a[1] == b[1] && a[2] < b[2])));
}

// Key endpoints of record r; false when its triangle has an index >= nV (the reference
// skips such triangles, EdgePreprocessor.cpp:64-66).
__device__ __forceinline__ bool record_key(const float* __restrict__ V, uint64_t nV, const uint32_t* __restrict__ I,
                                           uint32_t r, long long k0[3], long long k1[3]) {
    const uint64_t t = r / 3;
    const int e = (int)(r % 3);
    const uint32_t v[3] = {I[3 * t], I[3 * t + 1], I[3 * t + 2]};
    if (v[0] >= nV || v[1] >= nV || v[2] >= nV) return false;
    long long q0[3], q1[3];
    quantise(V, v[e], q0);
    quantise(V, v[e == 2 ? 0 : e + 1], q1);
    const bool sw = less3(q1, q0);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        k0[k] = sw ? q1[k] : q0[k];
        k1[k] = sw ? q0[k] : q1[k];
    }
    return true;
}

// Per-axis range of the quantised coordinates over valid records, and their number.
__global__ void k_q_bounds(const float* __restrict__ V, uint64_t nV, const uint32_t* __restrict__ I, uint64_t m,
                           long long* __restrict__ b, unsigned long long* __restrict__ n_valid) {
    long long mn[3] = {LLONG_MAX, LLONG_MAX, LLONG_MAX}, mx[3] = {LLONG_MIN, LLONG_MIN, LLONG_MIN};
    unsigned long long cnt = 0;
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < m; r += (uint64_t)gridDim.x * blockDim.x) {
        long long k0[3], k1[3];
        if (!record_key(V, nV, I, (uint32_t)r, k0, k1)) continue;
        ++cnt;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            mn[k] = min(mn[k], min(k0[k], k1[k]));
            mx[k] = max(mx[k], max(k0[k], k1[k]));
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        atomicMin(&b[k], mn[k]);
        atomicMax(&b[3 + k], mx[k]);
    }
    if (cnt) atomicAdd(n_valid, cnt);
}

// Field layout of the packed key, least significant first:
// k1.z, k1.y, k1.x, k0.z, k0.y, k0.x, skipped-triangle flag.
struct Packing {
    long long mn[3];
    int width[3];
    int total;
};

__device__ __forceinline__ uint64_t packed_word(const float* __restrict__ V, uint64_t nV,
                                                const uint32_t* __restrict__ I, uint32_t r, const Packing& p,
                                                int word) {
    long long k0[3], k1[3];
    const bool ok = record_key(V, nV, I, r, k0, k1);
    const uint64_t f[7] = {ok ? (uint64_t)(k1[2] - p.mn[2]) : 0, ok ? (uint64_t)(k1[1] - p.mn[1]) : 0,
                           ok ? (uint64_t)(k1[0] - p.mn[0]) : 0, ok ? (uint64_t)(k0[2] - p.mn[2]) : 0,
                           ok ? (uint64_t)(k0[1] - p.mn[1]) : 0, ok ? (uint64_t)(k0[0] - p.mn[0]) : 0,
                           ok ? 0ull : 1ull};
    const int w[7] = {p.width[2], p.width[1], p.width[0], p.width[2], p.width[1], p.width[0], 1};
    const int lo = 64 * word, hi = lo + 64;
    uint64_t out = 0;
    int pos = 0;
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        const int a = pos, b = pos + w[i];  // the field holds bits [a, b)
        if (w[i] > 0 && b > lo && a < hi) {
            const int s0 = max(a, lo), s1 = min(b, hi);
            const int n = s1 - s0;
            const uint64_t mask = n >= 64 ? ~0ull : ((1ull << n) - 1ull);
            out |= ((f[i] >> (s0 - a)) & mask) << (s0 - lo);
        }
        pos = b;
    }
    return out;
}

__global__ void k_iota(uint32_t* __restrict__ p, uint64_t n) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i < n) p[i] = (uint32_t)i;
}

// keys[j] = the given word of the packed key of record perm[j].
__global__ void k_word(const float* __restrict__ V, uint64_t nV, const uint32_t* __restrict__ I,
                       const uint32_t* __restrict__ perm, uint64_t m, Packing p, int word,
                       uint64_t* __restrict__ keys) {
    const uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (j < m) keys[j] = packed_word(V, nV, I, perm[j], p, word);
}

// head[j] = 1 when sorted record j starts a run of equal keys.
__global__ void k_heads(const float* __restrict__ V, uint64_t nV, const uint32_t* __restrict__ I,
                        const uint32_t* __restrict__ perm, uint64_t mv, uint32_t* __restrict__ head) {
    const uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (j >= mv) return;
    if (j == 0) {
        head[0] = 1;
        return;
    }
    long long a0[3], a1[3], b0[3], b1[3];
    record_key(V, nV, I, perm[j], a0, a1);
    record_key(V, nV, I, perm[j - 1], b0, b1);
    bool same = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) same = same && a0[k] == b0[k] && a1[k] == b1[k];
    head[j] = same ? 0u : 1u;
}

// (run, object) keys of the sorted records; the run of record j is gid[j] + head[j] - 1
// (gid = exclusive scan of the heads).
__global__ void k_run_obj(const int32_t* __restrict__ T, const uint32_t* __restrict__ perm,
                          const uint32_t* __restrict__ head, const uint32_t* __restrict__ gid, uint64_t mv,
                          uint64_t* __restrict__ key2, uint32_t* __restrict__ val2) {
    const uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (j >= mv) return;
    const uint32_t run = gid[j] + head[j] - 1;
    key2[j] = ((uint64_t)run << 32) | (uint32_t)T[perm[j] / 3];
    val2[j] = (uint32_t)j;
}

// keep[j] = 1 for the first record (in record order) of each (run, object).
__global__ void k_keep(const uint64_t* __restrict__ key2, const uint32_t* __restrict__ val2, uint64_t mv,
                       uint32_t* __restrict__ keep) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= mv) return;
    keep[val2[i]] = (i == 0 || key2[i] != key2[i - 1]) ? 1u : 0u;
}

// The payload: each kept record writes its object at its rank among kept records and
// counts itself in its run; each run's first record (always kept) writes the endpoints in
// its own orientation and the run's offset.
__global__ void k_emit(const float* __restrict__ V, const uint32_t* __restrict__ I, const int32_t* __restrict__ T,
                       const uint32_t* __restrict__ perm, const uint32_t* __restrict__ head,
                       const uint32_t* __restrict__ gid, const uint32_t* __restrict__ keep,
                       const uint32_t* __restrict__ kpos, uint64_t mv, float* __restrict__ starts,
                       float* __restrict__ ends, int32_t* __restrict__ offsets, int32_t* __restrict__ counts,
                       int32_t* __restrict__ sources) {
    const uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (j >= mv) return;
    const uint32_t r = perm[j];
    const uint32_t run = gid[j] + head[j] - 1;
    if (keep[j]) {
        sources[kpos[j]] = T[r / 3];
        atomicAdd(&counts[run], 1);
    }
    if (!head[j]) return;
    const uint64_t t = r / 3;
    const int e = (int)(r % 3);
    const uint32_t a = I[3 * t + e], b = I[3 * t + (e == 2 ? 0 : e + 1)];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        starts[3 * (uint64_t)run + k] = V[3 * (uint64_t)a + k];
        ends[3 * (uint64_t)run + k] = V[3 * (uint64_t)b + k];
    }
    offsets[run] = (int32_t)kpos[j];
}



// --- by vertices ---------------------------------------------------------------------

constexpr uint32_t kBucketSmall = 32;   // records of a list that one thread sorts
constexpr uint32_t kBucketBig = 4096;   // records of a list that one block sorts
constexpr uint32_t kFirst = 1u << 31;   // in a long list's record: the first of its run with its object
constexpr int kStageItems = 3072;       // records of 256 lists staged in shared memory

// Per-axis range of the vertices' quantised coordinates.
__global__ void __launch_bounds__(kPT) k_vq_bounds(const float* __restrict__ V, uint64_t nV,
                                                   long long* __restrict__ b) {
    long long v[6] = {LLONG_MAX, LLONG_MAX, LLONG_MAX, LLONG_MIN, LLONG_MIN, LLONG_MIN};
    for (uint64_t i = blockIdx.x * (uint64_t)kPT + threadIdx.x; i < nV; i += (uint64_t)gridDim.x * kPT) {
        long long q[3];
        quantise(V, (uint32_t)i, q);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            v[k] = min(v[k], q[k]);
            v[3 + k] = max(v[3 + k], q[k]);
        }
    }
    __shared__ long long red[6][kPT / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const long long y = __shfl_xor_sync(0xffffffffu, v[k], o);
            v[k] = k < 3 ? min(v[k], y) : max(v[k], y);
        }
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int k = 0; k < 6; ++k) red[k][threadIdx.x >> 5] = v[k];
    __syncthreads();
    if (threadIdx.x < 6) {
        const int k = threadIdx.x;
        long long x = red[k][0];
        for (int w = 1; w < kPT / 32; ++w) x = k < 3 ? min(x, red[k][w]) : max(x, red[k][w]);
        if (k < 3) atomicMin(&b[k], x);
        else atomicMax(&b[k], x);
    }
}

// The given 64-bit word of a vertex's packed key: z, y, x fields, least significant first.
__device__ __forceinline__ uint64_t vertex_word(const float* __restrict__ V, uint32_t v, const Packing& p, int word) {
    long long q[3];
    quantise(V, v, q);
    const int lo = 64 * word, hi = lo + 64;
    uint64_t out = 0;
    int pos = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int k = 2 - i, a = pos, b = pos + p.width[k];  // the field holds bits [a, b)
        if (p.width[k] > 0 && b > lo && a < hi) {
            const uint64_t f = (uint64_t)(q[k] - p.mn[k]);
            const int s0 = max(a, lo), n = min(b, hi) - s0;
            out |= ((f >> (s0 - a)) & (n >= 64 ? ~0ull : ((1ull << n) - 1ull))) << (s0 - lo);
        }
        pos = b;
    }
    return out;
}

// keys[j] = the word of vertex perm[j]; word 0 starts from (and writes) perm[j] = j.
__global__ void __launch_bounds__(kPT) k_vertex_word(const float* __restrict__ V, uint64_t nV, Packing p, int word,
                                                     uint32_t* __restrict__ perm, uint64_t* __restrict__ keys) {
    const uint64_t j = blockIdx.x * (uint64_t)kPT + threadIdx.x;
    if (j >= nV) return;
    const uint32_t v = word == 0 ? (uint32_t)j : perm[j];
    if (word == 0) perm[j] = v;
    keys[j] = vertex_word(V, v, p, word);
}

// head[j] = 1 when sorted vertex j is at another quantised position than the one before.
__global__ void __launch_bounds__(kPT) k_vertex_heads(const float* __restrict__ V, uint64_t nV,
                                                      const uint32_t* __restrict__ perm,
                                                      uint32_t* __restrict__ head) {
    const uint64_t j = blockIdx.x * (uint64_t)kPT + threadIdx.x;
    if (j >= nV) return;
    long long a[3] = {0, 0, 0}, b[3] = {0, 0, 0};
    quantise(V, perm[j], a);
    if (j) quantise(V, perm[j - 1], b);
    head[j] = j == 0 || a[0] != b[0] || a[1] != b[1] || a[2] != b[2] ? 1u : 0u;
}

__global__ void __launch_bounds__(kPT) k_vertex_rank(uint64_t nV, const uint32_t* __restrict__ perm,
                                                     const uint32_t* __restrict__ head,
                                                     const uint32_t* __restrict__ before,
                                                     uint32_t* __restrict__ rank) {
    const uint64_t j = blockIdx.x * (uint64_t)kPT + threadIdx.x;
    if (j < nV) rank[perm[j]] = before[j] + head[j] - 1u;
}

// Counts (FILL false) or lists (FILL true) the records of every lower rank; the fill counts
// the lists' lengths down to zero.  Triangles with an index >= nV are skipped, as the
// reference skips them (EdgePreprocessor.cpp:64-66).  Eight lanes and more of one rank share
// one atomic: where a mesh has collapsed, all of them queue on a few words.
template <bool FILL>
__global__ void __launch_bounds__(kPT) k_rank_lists(const uint32_t* __restrict__ I, uint64_t nF, uint64_t nV,
                                                    const uint32_t* __restrict__ rank, uint32_t* __restrict__ count,
                                                    const uint32_t* __restrict__ start,
                                                    uint64_t* __restrict__ items) {
    constexpr unsigned int kAll = 0xffffffffu;
    const uint64_t t = blockIdx.x * (uint64_t)kPT + threadIdx.x;
    const int lane = threadIdx.x & 31;
    uint32_t r[3] = {0, 0, 0};
    bool valid = t < nF;
    if (valid) {
        const uint32_t v[3] = {I[3 * t], I[3 * t + 1], I[3 * t + 2]};
        valid = v[0] < nV && v[1] < nV && v[2] < nV;
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (valid) r[k] = __ldg(&rank[v[k]]);
    }
    const unsigned int counted = __ballot_sync(kAll, valid);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const uint32_t a = r[e], b = r[e == 2 ? 0 : e + 1], lo = min(a, b), hi = max(a, b);
        uint32_t slot = 0;
        unsigned int todo = counted;
        while (todo) {  // the same in every lane
            const int leader = __ffs(todo) - 1;
            const uint32_t one = __shfl_sync(kAll, lo, leader);
            const unsigned int group = __ballot_sync(kAll, lo == one) & todo;
            const uint32_t n = __popc(group);
            if (n < 8) break;
            uint32_t base = 0;
            if (lane == leader) base = FILL ? atomicSub(&count[one], n) : atomicAdd(&count[one], n);
            base = __shfl_sync(kAll, base, leader);
            if (group >> lane & 1u) slot = base - 1u - __popc(group & ((1u << lane) - 1u));
            todo &= ~group;
        }
        if (todo >> lane & 1u) {
            if (FILL) slot = atomicSub(&count[lo], 1u) - 1u;
            else atomicAdd(&count[lo], 1u);
        }
        if (FILL && valid) items[start[lo] + slot] = (uint64_t)hi << 32 | (uint32_t)(3 * t + e);
    }
}

// Whether record i of a sorted list is the first of its run with its object.
template <class P>
__device__ __forceinline__ bool first_of_object(const P& x, int i, const int32_t* __restrict__ T) {
    const uint32_t hi = (uint32_t)(x[i] >> 32);
    const int32_t o = T[(uint32_t)x[i] / 3];
    for (int j = i - 1; j >= 0 && (uint32_t)(x[j] >> 32) == hi; --j)
        if (T[(uint32_t)x[j] / 3] == o) return false;
    return true;
}

// Sorts one list by one thread and counts its edges and sources.
template <class P>
__device__ __forceinline__ void sort_list(P x, int n, const int32_t* __restrict__ T, uint32_t& ne, uint32_t& ns) {
    for (int i = 1; i < n; ++i) {
        const uint64_t v = x[i];
        int j = i;
        for (; j > 0 && x[j - 1] > v; --j) x[j] = x[j - 1];
        x[j] = v;
    }
    ne = ns = 0;
    for (int i = 0; i < n; ++i) {
        ne += i == 0 || (x[i] >> 32) != (x[i - 1] >> 32);
        ns += first_of_object(x, i, T);
    }
}

// One thread per list, the records of a block's 256 lists staged in shared memory when they
// fit.  Lists longer than kBucketSmall go to big[0..*n_big); one longer than kBucketBig sets
// *too_long.
__global__ void __launch_bounds__(kPT) k_list_sort(uint64_t* __restrict__ items, const uint32_t* __restrict__ start,
                                                   uint64_t n_lists, const int32_t* __restrict__ T,
                                                   uint32_t* __restrict__ ne, uint32_t* __restrict__ ns,
                                                   uint32_t* __restrict__ big, uint32_t* __restrict__ n_big,
                                                   uint32_t* __restrict__ too_long) {
    __shared__ uint64_t stage[kStageItems];
    const uint64_t b0 = blockIdx.x * (uint64_t)kPT, b = b0 + threadIdx.x;
    const uint32_t first = start[b0], end = start[min(b0 + kPT, n_lists)];
    const bool staged = end - first <= (uint32_t)kStageItems;
    if (staged)
        for (uint32_t i = threadIdx.x; i < end - first; i += kPT) stage[i] = items[first + i];
    __syncthreads();
    if (b < n_lists) {
        const uint32_t s = start[b], n = start[b + 1] - s;
        uint32_t e = 0, c = 0;
        if (n > kBucketSmall) {
            big[atomicAdd(n_big, 1u)] = (uint32_t)b;
            if (n > kBucketBig) atomicOr(too_long, 1u);
        } else if (staged) {
            sort_list(stage + (s - first), (int)n, T, e, c);
        } else {
            sort_list(items + s, (int)n, T, e, c);
        }
        if (n <= kBucketSmall) {
            ne[b] = e;
            ns[b] = c;
        }
    }
    __syncthreads();
    if (staged)
        for (uint32_t i = threadIdx.x; i < end - first; i += kPT) items[first + i] = stage[i];
}

// Ascending bitonic sort of x[0..m), m a power of two, by the block.
__device__ __forceinline__ void block_sort(uint64_t* x, uint32_t m) {
    for (uint32_t k = 2; k <= m; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < m; i += kPT) {
                const uint32_t p = i ^ j;
                if (p > i && (x[i] > x[p]) == ((i & k) == 0)) {
                    const uint64_t t = x[i];
                    x[i] = x[p];
                    x[p] = t;
                }
            }
            __syncthreads();
        }
}

// One block per long list: a bitonic sort in shared memory by (higher rank, record), then one
// by (run, object, place), which puts a run's records of one object side by side, its first
// record first: that record is marked kFirst.  Looking back through the run for each record
// took as many loads in a row as the square of the run's length (a run of 1,300 objects: 80 ms,
// now 0.54 with everything else).
__global__ void __launch_bounds__(kPT) k_list_sort_big(uint64_t* __restrict__ items, const uint32_t* __restrict__ start,
                                                       const int32_t* __restrict__ T, uint32_t* __restrict__ ne,
                                                       uint32_t* __restrict__ ns, const uint32_t* __restrict__ big,
                                                       const uint32_t* __restrict__ n_big) {
    constexpr int kPer = kBucketBig / kPT, kPlaceBits = 12;
    static_assert(kBucketBig == 1u << kPlaceBits, "a place's bits");
    __shared__ uint64_t x[kBucketBig];
    __shared__ uint32_t sum[2];
    for (uint32_t q = blockIdx.x; q < *n_big; q += gridDim.x) {
        const uint32_t b = big[q], s = start[b], n = start[b + 1] - s;
        if (n > kBucketBig) continue;  // the records path takes the whole input
        uint32_t m = 64;
        while (m < n) m <<= 1;
        for (uint32_t i = threadIdx.x; i < m; i += kPT) x[i] = i < n ? items[s + i] : ~0ull;
        if (threadIdx.x < 2) sum[threadIdx.x] = 0;
        __syncthreads();
        block_sort(x, m);
        uint32_t e = 0, c = 0;
        uint64_t key[kPer];  // place of the run's head, object, place
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const uint32_t i = threadIdx.x + k * kPT;
            if (i >= n) continue;
            const uint64_t v = x[i];
            items[s + i] = v;
            e += i == 0 || (v >> 32) != (x[i - 1] >> 32);
            uint32_t lo = 0, hi = i;  // the first place of this higher rank
            while (lo < hi) {
                const uint32_t mid = (lo + hi) / 2;
                if ((x[mid] >> 32) < (v >> 32)) lo = mid + 1;
                else hi = mid;
            }
            key[k] = (uint64_t)lo << (32 + kPlaceBits) | (uint64_t)(uint32_t)T[(uint32_t)v / 3] << kPlaceBits | i;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const uint32_t i = threadIdx.x + k * kPT;
            if (i < m) x[i] = i < n ? key[k] : ~0ull;
        }
        __syncthreads();
        block_sort(x, m);
        for (uint32_t i = threadIdx.x; i < n; i += kPT)
            if (i == 0 || (x[i] >> kPlaceBits) != (x[i - 1] >> kPlaceBits)) {
                items[s + (uint32_t)(x[i] & (kBucketBig - 1))] |= kFirst;
                ++c;
            }
        atomicAdd(&sum[0], e);
        atomicAdd(&sum[1], c);
        __syncthreads();
        if (threadIdx.x == 0) {
            ne[b] = sum[0];
            ns[b] = sum[1];
        }
        __syncthreads();
    }
}

// The endpoints of record r in its triangle's orientation, as edge `at` of the payload.
__device__ __forceinline__ void write_endpoints(const float* __restrict__ V, const uint32_t* __restrict__ I, uint32_t r,
                                                uint64_t at, float* __restrict__ starts, float* __restrict__ ends) {
    const uint64_t t = r / 3;
    const int e = (int)(r % 3);
    const uint32_t a = I[3 * t + e], b = I[3 * t + (e == 2 ? 0 : e + 1)];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        starts[3 * at + k] = V[3 * (uint64_t)a + k];
        ends[3 * at + k] = V[3 * (uint64_t)b + k];
    }
}

// The payload of the lists that one thread sorted: its edges from epos[b], its sources from
// spos[b].
__global__ void __launch_bounds__(kPT) k_list_emit(const float* __restrict__ V, const uint32_t* __restrict__ I,
                                                   const int32_t* __restrict__ T, const uint64_t* __restrict__ items,
                                                   const uint32_t* __restrict__ start, uint64_t n_lists,
                                                   const uint32_t* __restrict__ epos, const uint32_t* __restrict__ spos,
                                                   float* __restrict__ starts, float* __restrict__ ends,
                                                   int32_t* __restrict__ offsets, int32_t* __restrict__ counts,
                                                   int32_t* __restrict__ sources) {
    const uint64_t b = blockIdx.x * (uint64_t)kPT + threadIdx.x;
    if (b >= n_lists) return;
    const uint32_t s = start[b];
    const int n = (int)(start[b + 1] - s);
    if (n == 0 || (uint32_t)n > kBucketSmall) return;
    const uint64_t* x = items + s;
    int64_t edge = (int64_t)epos[b] - 1;
    uint32_t src = spos[b], from = src;
    for (int i = 0; i < n; ++i) {
        if (i == 0 || (x[i] >> 32) != (x[i - 1] >> 32)) {
            if (i) counts[edge] = (int32_t)(src - from);
            ++edge;
            from = src;
            offsets[edge] = (int32_t)src;
            write_endpoints(V, I, (uint32_t)x[i], (uint64_t)edge, starts, ends);
        }
        if (first_of_object(x, i, T)) sources[src++] = T[(uint32_t)x[i] / 3];
    }
    counts[edge] = (int32_t)(src - from);
}

// The payload of the long lists, one block each: every thread a contiguous part, its places
// from a scan of the parts' counts; an edge's count is the distance to the next edge's offset.
__global__ void __launch_bounds__(kPT) k_list_emit_big(const float* __restrict__ V, const uint32_t* __restrict__ I,
                                                       const int32_t* __restrict__ T, const uint64_t* __restrict__ items,
                                                       const uint32_t* __restrict__ start,
                                                       const uint32_t* __restrict__ epos,
                                                       const uint32_t* __restrict__ spos,
                                                       const uint32_t* __restrict__ big,
                                                       const uint32_t* __restrict__ n_big, float* __restrict__ starts,
                                                       float* __restrict__ ends, int32_t* __restrict__ offsets,
                                                       int32_t* __restrict__ counts, int32_t* __restrict__ sources) {
    __shared__ uint64_t x[kBucketBig];
    __shared__ uint32_t pe[kPT], ps[kPT];
    for (uint32_t q = blockIdx.x; q < *n_big; q += gridDim.x) {
        const uint32_t b = big[q], s = start[b];
        const int n = (int)(start[b + 1] - s);
        for (int i = threadIdx.x; i < n; i += kPT) x[i] = items[s + i];
        __syncthreads();
        const int per = (n + kPT - 1) / kPT, i0 = min(n, (int)threadIdx.x * per), i1 = min(n, i0 + per);
        uint32_t ne = 0, ns = 0;
        for (int i = i0; i < i1; ++i) {
            ne += i == 0 || (x[i] >> 32) != (x[i - 1] >> 32);
            ns += ((uint32_t)x[i] & kFirst) != 0;
        }
        pe[threadIdx.x] = ne;
        ps[threadIdx.x] = ns;
        __syncthreads();
        uint32_t e = epos[b], src = spos[b], e_end = e, src_end = src;
        for (int k = 0; k < kPT; ++k) {
            e += k < (int)threadIdx.x ? pe[k] : 0u;
            src += k < (int)threadIdx.x ? ps[k] : 0u;
            e_end += pe[k];
            src_end += ps[k];
        }
        for (int i = i0; i < i1; ++i) {
            const uint32_t r = (uint32_t)x[i] & ~kFirst;
            if (i == 0 || (x[i] >> 32) != (x[i - 1] >> 32)) {
                offsets[e] = (int32_t)src;
                write_endpoints(V, I, r, e++, starts, ends);
            }
            if ((uint32_t)x[i] & kFirst) sources[src++] = T[r / 3];
        }
        __syncthreads();
        for (uint32_t k = epos[b] + threadIdx.x; k < e_end; k += kPT)
            counts[k] = (k + 1 < e_end ? offsets[k + 1] : (int32_t)src_end) - offsets[k];
    }
}

// Record r's key by its endpoints' ranks, its skipped-triangle flag above them.
__global__ void __launch_bounds__(kPT) k_rank_word(const uint32_t* __restrict__ I, uint64_t m, uint64_t nV,
                                                   const uint32_t* __restrict__ rank, int bits,
                                                   uint64_t* __restrict__ keys) {
    const uint64_t r = blockIdx.x * (uint64_t)kPT + threadIdx.x;
    if (r >= m) return;
    const uint64_t t = r / 3;
    const int e = (int)(r - 3 * t);
    const uint32_t v[3] = {I[3 * t], I[3 * t + 1], I[3 * t + 2]};
    if (v[0] >= nV || v[1] >= nV || v[2] >= nV) {
        keys[r] = 1ull << (2 * bits);
        return;
    }
    const uint32_t a = rank[v[e]], b = rank[v[e == 2 ? 0 : e + 1]];
    keys[r] = (uint64_t)min(a, b) << bits | max(a, b);
}

__global__ void __launch_bounds__(kPT) k_key_heads(const uint64_t* __restrict__ keys, uint64_t mv,
                                                   uint32_t* __restrict__ head) {
    const uint64_t j = blockIdx.x * (uint64_t)kPT + threadIdx.x;
    if (j < mv) head[j] = j == 0 || keys[j] != keys[j - 1] ? 1u : 0u;
}

struct EdgeOut {
    float* starts;
    float* ends;
    int32_t* offsets;
    int32_t* counts;
    int32_t* sources;
    uint64_t capacity;
};

// Turns the end of a path's counting (totals htot, sort error word) into the call's answer
// so far: RS_OK when the payload may be written.
int payload_status(const uint32_t* htot, uint32_t sort_err, const EdgeOut& out, uint64_t* h_nE, uint64_t* h_nS,
                   cudaStream_t s) {
    if (sort_err) {
        sort_error_clear(s);
        return RS_ERR_ITER_LIMIT;
    }
    *h_nE = htot[0];
    *h_nS = htot[1];
    return htot[0] > out.capacity || htot[1] > out.capacity ? RS_ERR_OUTPUT_OVERFLOW : RS_OK;
}

unsigned blocks_of(uint64_t n) { return (unsigned)((n + kPT - 1) / kPT); }

// The vertices' ranks, when the records are to be sorted by them, and the number of records of
// valid triangles.
struct Ranks {
    uint32_t* rank = nullptr;
    uint64_t n_valid = 0;
};

// ranks->n_valid is left zero unless a list is too long for it (nothing is written then); the
// ranks are the caller's to free.
int extract_by_vertices(const float* V, uint64_t nV, const uint32_t* I, uint64_t nF, const int32_t* T,
                        const EdgeOut& out, uint64_t* h_nE, uint64_t* h_nS, Ranks* ranks, cudaStream_t s) {
    const uint64_t m = 3 * nF;
    Scratch sc{s};
    long long* qb = nullptr;  // bounds; then the words: edges, sources, long lists, too long
    uint32_t *perm = nullptr, *rank = ranks->rank, *head = nullptr, *before = nullptr;
    uint64_t* keys = nullptr;
    cudaError_t e = sc.get(&qb, 8 * sizeof(long long));
    if (e == cudaSuccess) e = sc.get(&perm, nV * 4);
    if (e == cudaSuccess) e = sc.get(&head, (nV + 1) * 4);
    if (e == cudaSuccess) e = sc.get(&before, (nV + 1) * 4);
    if (e == cudaSuccess) e = sc.get(&keys, std::max(nV, m) * 8);
    if (e != cudaSuccess) return to_status(e);
    const long long init[6] = {LLONG_MAX, LLONG_MAX, LLONG_MAX, LLONG_MIN, LLONG_MIN, LLONG_MIN};
    long long hb[6];
    e = cudaMemcpyAsync(qb, init, sizeof(init), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        launch(k_vq_bounds, (unsigned)std::min<uint64_t>(blocks_of(nV), 4ull * sm_count()), kPT, 0, s, V, nV, qb);
        e = cudaMemcpyAsync(hb, qb, sizeof(hb), cudaMemcpyDeviceToHost, s);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return to_status(e);
    Packing p;
    p.total = 0;
    for (int k = 0; k < 3; ++k) {
        p.mn[k] = hb[k];
        p.width[k] = bits_for((unsigned long long)hb[3 + k] - (unsigned long long)hb[k]);
        p.total += p.width[k];
    }
    for (int w = 0; w < std::max(1, (p.total + 63) / 64) && e == cudaSuccess; ++w) {
        launch(k_vertex_word, blocks_of(nV), kPT, 0, s, V, nV, p, w, perm, keys);
        e = radix_sort_u64(keys, perm, nV, std::min(64, p.total - 64 * w), s);
    }
    uint32_t* words = reinterpret_cast<uint32_t*>(qb);
    if (e == cudaSuccess) e = cudaMemsetAsync(words, 0, 4 * sizeof(uint32_t), s);
    if (e == cudaSuccess) {
        launch(k_vertex_heads, blocks_of(nV), kPT, 0, s, V, nV, (const uint32_t*)perm, head);
        e = exclusive_scan_u32(head, before, nV, nullptr, s);
    }
    if (e == cudaSuccess)
        launch(k_vertex_rank, blocks_of(nV), kPT, 0, s, nV, (const uint32_t*)perm, (const uint32_t*)head,
               (const uint32_t*)before, rank);
    // Ranks are below nV, so there are nV lists (the last ones empty).  The sort's arrays are
    // free: perm becomes the lists' lengths, head their starts, keys their records.
    uint32_t *count = perm, *start = head;
    uint64_t* items = keys;
    if (e == cudaSuccess) e = cudaMemsetAsync(count, 0, nV * 4, s);
    if (e == cudaSuccess) {
        launch(k_rank_lists<false>, blocks_of(nF), kPT, 0, s, I, nF, nV, (const uint32_t*)rank, count,
               (const uint32_t*)nullptr, (uint64_t*)nullptr);
        e = exclusive_scan_u32(count, start, nV, start + nV, s);
    }
    uint32_t *ne = nullptr, *ns = nullptr, *big = nullptr;
    if (e == cudaSuccess) e = sc.get(&ne, nV * 4);
    if (e == cudaSuccess) e = sc.get(&ns, nV * 4);
    if (e == cudaSuccess) e = sc.get(&big, (m / kBucketSmall + 1) * 4);
    uint32_t h[5] = {0, 0, 0, 0, 0};
    if (e == cudaSuccess) {
        launch(k_rank_lists<true>, blocks_of(nF), kPT, 0, s, I, nF, nV, (const uint32_t*)rank, count,
               (const uint32_t*)start, items);
        launch(k_list_sort, blocks_of(nV), kPT, 0, s, items, (const uint32_t*)start, nV, T, ne, ns, big, words + 2,
               words + 3);
        launch(k_list_sort_big, 4u * sm_count(), kPT, 0, s, items, (const uint32_t*)start, T, ne, ns,
               (const uint32_t*)big, (const uint32_t*)(words + 2));
        e = exclusive_scan_u32(ne, ne, nV, words, s);
        if (e == cudaSuccess) e = exclusive_scan_u32(ns, ns, nV, words + 1, s);
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, words, 16, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = sort_error_read(&h[4], s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return to_status(e);
    if (h[3] && !h[4]) {
        uint32_t valid = 0;
        e = cudaMemcpyAsync(&valid, start + nV, 4, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        ranks->n_valid = valid;
        return to_status(e);
    }
    const int st = payload_status(h, h[4], out, h_nE, h_nS, s);
    if (st != RS_OK || h[0] == 0) return st;
    launch(k_list_emit, blocks_of(nV), kPT, 0, s, V, I, T, (const uint64_t*)items, (const uint32_t*)start, nV,
           (const uint32_t*)ne, (const uint32_t*)ns, out.starts, out.ends, out.offsets, out.counts, out.sources);
    if (h[2])
        launch(k_list_emit_big, (unsigned)std::min<uint64_t>(h[2], 4u * sm_count()), kPT, 0, s, V, I, T,
               (const uint64_t*)items, (const uint32_t*)start, (const uint32_t*)ne, (const uint32_t*)ns,
               (const uint32_t*)big, (const uint32_t*)(words + 2), out.starts, out.ends, out.offsets, out.counts,
               out.sources);
    e = cudaGetLastError();
    const cudaError_t e2 = cudaStreamSynchronize(s);
    return to_status(e == cudaSuccess ? e2 : e);
}

// The records path: all records sorted, by their endpoints' ranks or (ranks null) by their
// packed quantised key.
int extract_by_records(const float* d_vertices, uint64_t nV, const uint32_t* d_indices, uint64_t nF,
                       const int32_t* d_tri2obj, const EdgeOut& out, uint64_t* h_nE, uint64_t* h_nS, const Ranks* ranks,
                       cudaStream_t s) {
    const uint64_t m = 3 * nF;
    cudaError_t e = cudaSuccess;
    long long hb[6];
    unsigned long long hv = 0;
    uint32_t htot[2] = {0, 0};
    {
        Scratch sc{s};
        long long* qb = nullptr;
        uint32_t *perm = nullptr, *head = nullptr, *gid = nullptr, *keep = nullptr, *kpos = nullptr,
                 *val2 = nullptr;
        uint64_t* keys = nullptr;
        e = sc.get(&qb, 8 * sizeof(long long));
        if (e == cudaSuccess) e = sc.get(&perm, m * 4);
        if (e == cudaSuccess) e = sc.get(&keys, m * 8);
        if (e != cudaSuccess) return to_status(e);
        const unsigned nb = blocks_of(m);
        if (ranks) {
            hv = ranks->n_valid;
            const int bits = bits_for(nV - 1);  // at most 31: nV <= m
            launch(k_iota, nb, kPT, 0, s, perm, m);
            launch(k_rank_word, nb, kPT, 0, s, d_indices, m, nV, (const uint32_t*)ranks->rank, bits, keys);
            e = radix_sort_u64(keys, perm, m, 2 * bits + 1, s);
        } else {
            unsigned long long* nvalid = reinterpret_cast<unsigned long long*>(qb + 6);
            const long long init[7] = {LLONG_MAX, LLONG_MAX, LLONG_MAX, LLONG_MIN, LLONG_MIN, LLONG_MIN, 0};
            e = cudaMemcpyAsync(qb, init, sizeof(init), cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) {
                launch(k_q_bounds, 4 * sm_count(), kPT, 0, s, d_vertices, nV, d_indices, m, qb, nvalid);
                e = cudaGetLastError();
            }
            if (e == cudaSuccess) e = cudaMemcpyAsync(hb, qb, sizeof(hb), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaMemcpyAsync(&hv, nvalid, 8, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess || hv == 0) return to_status(e);

            Packing p;
            p.total = 1;
            for (int k = 0; k < 3; ++k) {
                p.mn[k] = hb[k];
                p.width[k] = bits_for((unsigned long long)hb[3 + k] - (unsigned long long)hb[k]);
                p.total += 2 * p.width[k];
            }
            const int nwords = (p.total + 63) / 64;
            launch(k_iota, nb, kPT, 0, s, perm, m);
            for (int w = 0; w < nwords && e == cudaSuccess; ++w) {
                launch(k_word, nb, kPT, 0, s, d_vertices, nV, d_indices, (const uint32_t*)perm, m, p, w, keys);
                e = radix_sort_u64(keys, perm, m, std::min(64, p.total - 64 * w), s);
            }
        }
        // Valid records sort first (flag bit 0); runs and sources over those alone.
        const uint64_t mv = hv;
        const unsigned nbv = (unsigned)((mv + kPT - 1) / kPT);
        uint32_t* tot = reinterpret_cast<uint32_t*>(qb);
        if (e == cudaSuccess) e = sc.get(&head, mv * 4);
        if (e == cudaSuccess) e = sc.get(&gid, mv * 4);
        if (e == cudaSuccess) e = sc.get(&keep, mv * 4);
        if (e == cudaSuccess) e = sc.get(&kpos, mv * 4);
        if (e == cudaSuccess) e = sc.get(&val2, mv * 4);
        if (e == cudaSuccess) {
            if (ranks) launch(k_key_heads, nbv, kPT, 0, s, (const uint64_t*)keys, mv, head);
            else launch(k_heads, nbv, kPT, 0, s, d_vertices, nV, d_indices, (const uint32_t*)perm, mv, head);
            e = exclusive_scan_u32(head, gid, mv, tot, s);
        }
        if (e == cudaSuccess) {
            launch(k_run_obj, nbv, kPT, 0, s, d_tri2obj, (const uint32_t*)perm, (const uint32_t*)head,
                   (const uint32_t*)gid, mv, keys, val2);
            e = radix_sort_u64(keys, val2, mv, 32 + bits_for(mv), s);  // run < mv
        }
        if (e == cudaSuccess) {
            launch(k_keep, nbv, kPT, 0, s, (const uint64_t*)keys, (const uint32_t*)val2, mv, keep);
            e = exclusive_scan_u32(keep, kpos, mv, tot + 1, s);
        }
        uint32_t sort_err = 0;
        if (e == cudaSuccess) e = cudaMemcpyAsync(htot, tot, 8, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = sort_error_read(&sort_err, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return to_status(e);
        const int st = payload_status(htot, sort_err, out, h_nE, h_nS, s);
        if (st != RS_OK) return st;
        e = cudaMemsetAsync(out.counts, 0, (size_t)htot[0] * sizeof(int32_t), s);
        if (e == cudaSuccess) {
            launch(k_emit, nbv, kPT, 0, s, d_vertices, d_indices, d_tri2obj, (const uint32_t*)perm,
                   (const uint32_t*)head, (const uint32_t*)gid, (const uint32_t*)keep, (const uint32_t*)kpos, mv,
                   out.starts, out.ends, out.offsets, out.counts, out.sources);
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return to_status(e);
}

}  // namespace
}  // namespace rs

using namespace rs;

extern "C" int rs_extract_edges(const float* d_vertices, uint64_t nV, const uint32_t* d_indices, uint64_t nF,
                                const int32_t* d_tri2obj, float* d_starts, float* d_ends, int32_t* d_offsets,
                                int32_t* d_counts, int32_t* d_sources, uint64_t capacity, uint64_t* h_nE,
                                uint64_t* h_nS, void* stream) {
    if (!h_nE || !h_nS) return RS_ERR_INVALID;
    *h_nE = *h_nS = 0;
    if ((nF && (!d_indices || !d_tri2obj)) || (nV && !d_vertices)) return RS_ERR_INVALID;
    const uint64_t m = 3 * nF;
    if (m == 0 || nV == 0) return RS_OK;
    if (m > 0x7fffffffull) return RS_ERR_TOO_LARGE;  // int32 offsets, u32 record ids
    if (!d_starts || !d_ends || !d_offsets || !d_counts || !d_sources) return RS_ERR_INVALID;
    const EdgeOut out{d_starts, d_ends, d_offsets, d_counts, d_sources, capacity};
    cudaStream_t s = (cudaStream_t)stream;
    // More vertices than corners: most are in no triangle, and sorting them would cost more
    // than sorting the records.
    if (nV <= m) {
        Scratch sc{s};
        Ranks ranks;
        const cudaError_t e = sc.get(&ranks.rank, nV * 4);
        if (e != cudaSuccess) return to_status(e);
        const int st = extract_by_vertices(d_vertices, nV, d_indices, nF, d_tri2obj, out, h_nE, h_nS, &ranks, s);
        if (st != RS_OK || ranks.n_valid == 0) return st;
        return extract_by_records(d_vertices, nV, d_indices, nF, d_tri2obj, out, h_nE, h_nS, &ranks, s);
    }
    return extract_by_records(d_vertices, nV, d_indices, nF, d_tri2obj, out, h_nE, h_nS, nullptr, s);
}
