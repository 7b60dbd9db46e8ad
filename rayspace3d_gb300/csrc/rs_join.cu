// rs_join.cu -- edge-ray overlap and the containment fallback.
//
// Edge rays replace __raygen__mesh_overlap_edges / trace_edge_multi_hits_edges
// (query/src/cuda/mesh_overlap_edges.cu:106-216) and __raygen__mesh_overlap
// (mesh_intersection.cu:16-91,288-334): a warp traces up to 32 unique edges as a packet, each
// once (the reference re-traces per hit and, in the intersection variant, per source
// object), takes their crossings with the reference's hit rule and inserts (source, target)
// pairs straight into the pair table; edges of many crossings follow, a warp each.  The
// edges a broad phase keeps are binned by the Morton cell of their midpoint first, so that
// the rays of a warp start close together and descend the same subtrees.  Containment
// replaces __raygen__mesh_containment_anyhit + __anyhit__ah_containment
// (mesh_intersection_anyhit.cu:46-240): one +Z ray per source object by a warp (in packets
// first when there are very many), the object ids of its crossings in shared memory instead
// of a 256-slot global scratch per object; only the per-source diagnostics take a thread an
// object with the parities in registers.
#include <algorithm>
#include <climits>

#include <mutex>

#include "rs_engine.h"
#include "rs_prims.cuh"
#include "rs_query_core.cuh"

namespace rs {
namespace {

constexpr int kT = 128;
constexpr int kTargets = 32;
constexpr int kFastStack = 32;  // shared-memory stack entries per lane of the edge-ray kernels
constexpr int kCellBits = 5;    // 32^3 Morton cells order the live edges
constexpr int kCells = 1 << (3 * kCellBits);
// Jobs with more edges than this are traced in live-list order (no binning): the cell
// ranks and the ordered list would cost 8 more bytes per edge.
constexpr uint64_t kBinMaxEdges = 1ull << 27;
// Fewer live edges than this are traced in live-list order: the scan and the scatter would
// cost more than the coherence saves.
constexpr unsigned int kBinMinLive = 1u << 16;

// Edge rays over the edges order[0..*n_order) of a payload of n_direct edges (or over all of
// them when order is null), in packets that the warps of a resident grid take from *next; a
// packet has as many edges as give every warp one (32 at most), since the lists of a few
// thousand edges wait on their longest packet.  The edges it defers go to
// deferred[0..*n_def).  entry (nullable): the node each listed edge's traversal starts from.
constexpr int kPacketWarps = 4;
// Steps after which a packet leaves its unfinished edges to the long path, a warp for each:
// the order by cell puts a cluster's longest edges together, and a join otherwise ends
// waiting for a few packets of them (2.2 and 2.4 ms for the two directions of a clustered
// join, 14 and 6 of 24 warps an SM in flight on average; now 0.65 + 0.54 and 0.53 +
// 1.03 ms).  512 and 128 steps: 4 % and 1 % more of it; a join whose sizes are uneven,
// but not clustered, takes 7 us more than without a limit at 256 steps and 240 at 128.
constexpr uint32_t kPacketSteps = 256;

__global__ void __launch_bounds__(32 * kPacketWarps, 6) k_edge_rays(
    EdgePayload p, const uint32_t* __restrict__ order, const uint32_t* __restrict__ live,
    const unsigned int* __restrict__ n_order, uint64_t n_direct, const BNode* __restrict__ nodes, uint32_t max_steps,
    const float4* __restrict__ tris, int swap, PairTable table, uint32_t* __restrict__ deferred,
    unsigned int* __restrict__ n_def, const uint32_t* __restrict__ order_entry,
    const uint32_t* __restrict__ live_entry, unsigned int* __restrict__ next) {
    __shared__ RayPacket packets[kPacketWarps];
    RayPacket& sm = packets[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const uint64_t n = live ? (uint64_t)*n_order : n_direct;
    // The cell-ordered list when the job was binned and is long enough, else the live list.
    const uint32_t* entry = nullptr;
    if (live) {
        const bool binned = order && n >= kBinMinLive;
        entry = binned ? order_entry : live_entry;
        order = binned ? order : live;
    }
    const uint64_t warps = (uint64_t)gridDim.x * kPacketWarps;
    const uint32_t size = (uint32_t)min((n + warps - 1) / warps, (uint64_t)32);
    for (;;) {
        unsigned int k = 0;
        if (lane == 0) k = atomicAdd(next, 1u);
        k = __shfl_sync(0xffffffffu, k, 0);
        const uint64_t base = (uint64_t)k * size;
        if (base >= n) return;
        const uint64_t j = base + lane;
        bool valid = (uint32_t)lane < size && j < n;
        const uint32_t e = !valid ? 0u : order ? order[j] : (uint32_t)j;
        const int start = valid && entry ? (int)entry[j] : 0;
        valid = valid && e < n_direct;  // always, for a list of this payload's edges
        if (edge_packet(sm, p, valid, e, start, nodes, min(max_steps, kPacketSteps), tris, swap, table))
            deferred[atomicAdd(n_def, 1u)] = e;
        __syncwarp();
    }
}

// One edge by one warp, its crossings in ranges of t (range_collect).  Lane 0 walks a range with
// the table's hit rule, and the pairs of the hits taken are inserted by all lanes (one lane's
// inserts, a few hundred dependent atomics an edge, took a tenth of a clustered join's
// k_edge_long_warp).  An edge of a large object in a dense cluster overlaps thousands of boxes,
// and the one-thread loop kept a whole join waiting (17 ms of 57).  A full list that threw its
// traversal away and began again with half the range took 84 ms for the edges of 20,000 boxes that
// reach through 2,000 others, where a thread an edge had taken 75; now 39.
// Returns false when range_collect does; pairs of ranges walked before that are in the table,
// where the one-thread loop's start from the beginning finds them.
__device__ __forceinline__ bool edge_ray_warp(RangeWarp& w_sm, const EdgePayload& p, uint64_t i,
                                              const BNode* __restrict__ nodes, uint32_t max_steps,
                                              const float4* __restrict__ tris, int swap, const PairTable& table) {
    const int lane = threadIdx.x & 31;
    Ray r;
    if (!segment_ray_of(p.starts[3 * i], p.starts[3 * i + 1], p.starts[3 * i + 2], p.ends[3 * i], p.ends[3 * i + 1],
                        p.ends[3 * i + 2], r))
        return true;
    const float tmax = r.tmax;
    float above = -INFINITY;
    EdgeWalk w;
    int32_t last = INT_MIN;
    int nh = 0;
    unsigned int tests = 0;
    do {
        if (!range_collect<-1>(w_sm, nodes, max_steps, tris, r, above, nh, tests)) return false;
        range_sort(w_sm, nh);
        int found = 0;  // objects to insert, over those walked
        if (lane == 0)
            for (int a = 0; a < nh && !w.done; ++a) {
                if (!w.take(range_t(w_sm, a), table.max_hits, table.next_float)) continue;
                if (w_sm.obj[a] == last) continue;
                last = w_sm.obj[a];
                w_sm.obj[found++] = last;
            }
        found = __shfl_sync(0xffffffffu, found, 0);
        __syncwarp();
        for (int a = lane; a < found; a += 32)
            insert_sources(table, p.sources + p.offsets[i], p.counts[i], w_sm.obj[a], swap);
        __syncwarp();
    } while (!__shfl_sync(0xffffffffu, (int)w.done, 0) && next_range(r, tmax, above));
    add_tests(tests);
    if (lane == 0) count_edge(table, w.n);
    __syncwarp();
    return true;
}

// Long path over the deferred edges, one warp per edge; the one-thread loop (segment_long, in
// lane 0, 16 crossings a traversal) is left for hundreds of crossings at one distance.
constexpr int kLongWarps = kRangeWarps;

__global__ void __launch_bounds__(32 * kLongWarps, 4) k_edge_long_warp(EdgePayload p, const uint32_t* __restrict__ deferred,
                                                                    const unsigned int* __restrict__ n_def,
                                                                    const BNode* __restrict__ nodes, uint32_t max_steps,
                                                                    const float4* __restrict__ tris, int swap,
                                                                    PairTable table) {
    __shared__ RangeWarp sm[kLongWarps];
    const unsigned int n = *n_def;
    const int wi = threadIdx.x >> 5;
    const unsigned int nw = gridDim.x * kLongWarps;
    for (unsigned int j = blockIdx.x * kLongWarps + wi; j < n; j += nw) {  // warp-uniform
        const uint32_t e = deferred[j];
        if (!edge_ray_warp(sm[wi], p, e, nodes, max_steps, tris, swap, table) &&
            (threadIdx.x & 31) == 0)
            edge_ray_long(p, e, nodes, max_steps, tris, swap, table);
        __syncwarp();
    }
}

// Legacy per-triangle overlap (mesh_overlap.cu:126-179): record r = 3 t + e is edge e of
// source triangle t.  Triangles with an index >= nV set *bad and are skipped.  Records the
// fast path defers go to deferred (when given; else they run the long path here).
__global__ void __launch_bounds__(kT) k_tri_edge_join(const float* __restrict__ V, uint64_t nV,
                                                      const uint32_t* __restrict__ I,
                                                      const int32_t* __restrict__ T, uint64_t m,
                                                      const BNode* __restrict__ nodes, uint32_t max_steps,
                                                      const float4* __restrict__ tris, int swap, PairTable table,
                                                      unsigned int* __restrict__ bad, uint32_t* __restrict__ deferred,
                                                      unsigned int* __restrict__ n_def) {
    __shared__ EdgeSmem<kT, kFastStack> sm;
    const uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (r >= m) return;
    const uint64_t t = r / 3;
    if (I[3 * t] >= nV || I[3 * t + 1] >= nV || I[3 * t + 2] >= nV) {
        if (r % 3 == 0) atomicOr(bad, 1u);
        return;
    }
    Ray ray;
    if (!triangle_edge_of(V, I, r, ray)) return;
    if (deferred) {
        if (!segment_fast<kFastStack>(sm.column(threadIdx.x), ray, T + t, 1, nodes, max_steps, tris, swap, table))
            deferred[atomicAdd(n_def, 1u)] = (uint32_t)r;
    } else {
        segment_long(ray, T + t, 1, nodes, max_steps, tris, swap, table);
    }
}

__global__ void __launch_bounds__(kT) k_tri_edge_long(const float* __restrict__ V, const uint32_t* __restrict__ I,
                                                      const int32_t* __restrict__ T,
                                                      const uint32_t* __restrict__ deferred,
                                                      const unsigned int* __restrict__ n_def,
                                                      const BNode* __restrict__ nodes, uint32_t max_steps,
                                                      const float4* __restrict__ tris, int swap, PairTable table) {
    const unsigned int n = *n_def;
    for (unsigned int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const uint64_t r = deferred[j];
        Ray ray;
        if (triangle_edge_of(V, I, r, ray)) segment_long(ray, T + r / 3, 1, nodes, max_steps, tris, swap, table);
    }
}

// Broad-phase widening (the broad phase below says why it covers every hit).
constexpr float kCullAbs = 1e-4f;
constexpr float kCullRel = 4e-6f;

__device__ __forceinline__ float cull_margin(float l, float h) {
    return kCullRel * (fmaxf(fabsf(l), fabsf(h)) + (h - l));
}

__device__ __forceinline__ int f2ord(float f) {
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
// Of a range's maximum: one without a number is the empty box's (its minimum, 0x7fffffff, is).
__device__ __forceinline__ int f2ord_max(float f) { return isnan(f) ? (int)0x80000000 : f2ord(f); }
__device__ __forceinline__ float ord2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// The box of edge i's segment widened like a broad-phase query box: kCullAbs plus the
// relative margin of the box, per axis.
__device__ __forceinline__ void edge_query_box(const EdgePayload& p, uint64_t i, float* qlo, float* qhi) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float a = p.starts[3 * i + k], b = p.ends[3 * i + k];
        const float l = fminf(a, b), h = fmaxf(a, b);
        const float m = kCullAbs + cull_margin(l, h);
        qlo[k] = l - m;
        qhi[k] = h + m;
    }
}

// An object box (ordered ints, min xyz then max xyz) widened by its margin overlaps the
// (already widened) query box.
__device__ __forceinline__ bool box_overlaps(const int* __restrict__ ob, const float* qlo, const float* qhi) {
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float l = ord2f(__ldg(&ob[k])), h = ord2f(__ldg(&ob[3 + k]));
        const float m = cull_margin(l, h);
        ok = ok && (l - m <= qhi[k]) && (h + m >= qlo[k]);
    }
    return ok;
}

// The edges of one source set traced against the other set's BVH, with the source
// objects' broad-phase flags and the job's work lists.
struct EdgeJob {
    EdgePayload p;
    uint64_t nE;
    const uint8_t* cull;  // flag (or partner count) per source object below n_cull
    uint64_t n_cull;
    const int32_t* part;  // partner lists (nullable), as EdgeCull
    const float4* pbox;   // the target set's object boxes, widened
    uint64_t n_pbox;
    uint32_t* live;       // live edges, in arrival order
    uint32_t* rank;       // rank of each live edge within its cell; then the deferred edges
    uint32_t* order;      // live edges by cell (binned jobs)
    uint32_t* cells;      // kCells counts, then their exclusive prefix sums (binned jobs)
    // Entry nodes (nullable, as EdgeCull): per source object, then per edge of live and of
    // order -- the node an edge's traversal starts from.
    const uint32_t* entry;
    uint32_t* live_entry;
    uint32_t* order_entry;
    // Slab index (nullable, as EdgeCull): the payload's slab keys, the source objects' own
    // boxes, and one flag per slab (zeroed) for the slabs that may hold a live edge.
    const long long* xindex;
    const int* sbox;
    uint8_t* covered;
    uint64_t n_slab;
    unsigned int* n_live;
    unsigned int* n_def;
    const BNode* nodes;
    uint32_t max_steps;
    const float4* tris;
    int swap;
};

__device__ __forceinline__ uint32_t spread5(uint32_t v) {  // 5 bits -> every third bit
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

// Morton cell (32^3 over the target BVH's root box) of edge i's midpoint.  Written with
// rounded intrinsics so every kernel that calls it computes the same cell.
__device__ __forceinline__ uint32_t edge_cell(const EdgeJob& j, uint64_t i) {
    const float4 na = __ldg(&j.nodes[0].a), nb = __ldg(&j.nodes[0].b), nc = __ldg(&j.nodes[0].c);
    const float lo[3] = {fminf(na.x, nb.z), fminf(na.y, nb.w), fminf(na.z, nc.x)};
    const float hi[3] = {fmaxf(na.w, nc.y), fmaxf(nb.x, nc.z), fmaxf(nb.y, nc.w)};
    uint32_t code = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float m = __fmul_rn(__fadd_rn(j.p.starts[3 * i + k], j.p.ends[3 * i + k]), 0.5f);
        const float ext = __fsub_rn(hi[k], lo[k]);
        float q = ext > 0.0f ? __fmul_rn(__fdiv_rn(__fsub_rn(m, lo[k]), ext), (float)(1 << kCellBits)) : 0.0f;
        q = fminf(fmaxf(q, 0.0f), (float)((1 << kCellBits) - 1));
        code |= spread5((uint32_t)q) << k;
    }
    return code;
}

// Eight 32-bit values from a 32-byte boundary.
__device__ __forceinline__ void load_ints8(const int32_t* __restrict__ p, int32_t (&v)[8]) {
    asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "l"(p));
}

// Both sets' object boxes widened by their margins, as box_overlaps widens them.
__global__ void __launch_bounds__(256) k_wide_boxes(const int* __restrict__ boxA, uint64_t nA,
                                                    const int* __restrict__ boxB, uint64_t nB,
                                                    float4* __restrict__ out) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= nA + nB) return;
    const int* ob = i < nA ? boxA + 6 * i : boxB + 6 * (i - nA);
    float lo[3], hi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float l = ord2f(ob[k]), h = ord2f(ob[3 + k]);
        const float m = cull_margin(l, h);
        lo[k] = l - m;
        hi[k] = h + m;
    }
    out[2 * i] = make_float4(lo[0], lo[1], lo[2], 0.0f);
    out[2 * i + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
}

// Whether edge i of job j is live, given its source count ns, its source list sp, and its
// first source so0 with that object's flag c0 (loaded by the caller).
__device__ __forceinline__ bool edge_is_live(const EdgeJob& j, uint64_t i, int ns, const int32_t* sp, int32_t so0,
                                             uint8_t c0) {
    float qlo[3], qhi[3];
    bool have_box = false;
    for (int q = 0; q < ns; ++q) {
        const int32_t so = q == 0 ? so0 : sp[q];
        if (so < 0 || (uint64_t)so >= j.n_cull) return true;
        const uint8_t c = q == 0 ? c0 : j.cull[so];
        if (c == 0) continue;
        if (!j.part || c == kCandAll) return true;
        // The edge is live when its own widened box reaches a partner's widened box.
        if (!have_box) {
            edge_query_box(j.p, i, qlo, qhi);
            have_box = true;
        }
        // The list and each partner's box by one 32-byte load.
        int32_t pl[kPartners];
        load_ints8(j.part + (uint64_t)so * kPartners, pl);
#pragma unroll
        for (int k = 0; k < kPartners; ++k) {
            if (k >= (int)c) break;
            if (pl[k] < 0 || (uint64_t)pl[k] >= j.n_pbox) return true;
            int32_t w[8];
            load_ints8(reinterpret_cast<const int32_t*>(j.pbox + 2 * (uint64_t)pl[k]), w);
            if (__int_as_float(w[0]) <= qhi[0] && __int_as_float(w[4]) >= qlo[0] && __int_as_float(w[1]) <= qhi[1] &&
                __int_as_float(w[5]) >= qlo[1] && __int_as_float(w[2]) <= qhi[2] && __int_as_float(w[6]) >= qlo[2])
                return true;
        }
    }
    return false;
}

// Broad phase: the edges with at least one candidate source object (k_cull_flag /
// k_cull_query) are appended to their job's `live` list; in binned jobs each also takes a
// rank within its cell (one warp-aggregated atomic per cell and warp).  Each thread takes
// kLiveEdges edges (a block's edges are contiguous, kLiveEdges rounds of blockDim) and
// issues the dependent loads of all of them together -- count and offset, first source,
// its flag -- so that a wave of threads keeps several chains in flight.  Bound by those
// chains' latency: two edges a thread at 32 registers (180 us for 9.6 M edges of a dense join)
// beat four at 64 and at 40 (245, 215) and one (295).  Blocks below blocks0 run job j0, the
// others j1.
constexpr int kLiveEdges = 2;

// Appends the block's edges first + u * kLiveThreads of each thread to their job's live list
// where any[u] (every thread of the block calls it): one atomic per block -- one per warp and
// round, all on one word, took most of the kernel's time -- the entry nodes beside them, and
// in binned jobs each edge's rank within its cell.
constexpr int kLiveThreads = 256;

template <int U>
__device__ __forceinline__ void live_append(const EdgeJob& j, uint64_t first, const bool (&any)[U],
                                            const uint32_t (&en)[U]) {
    constexpr int kWarps = kLiveThreads / 32;
    static_assert(U * kWarps <= 32, "one lane per warp and round");
    __shared__ uint32_t s_cnt[32];
    __shared__ uint32_t s_pos;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned int below = (1u << lane) - 1u;
    unsigned int m[U], some = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        m[u] = __ballot_sync(0xffffffffu, any[u]);
        some |= m[u];
        if (lane == 0) s_cnt[u * kWarps + warp] = __popc(m[u]);
    }
    if (!__syncthreads_or((int)(some != 0))) return;  // most blocks of a sparse join
    if (warp == 0) {
        const uint32_t c = lane < U * kWarps ? s_cnt[lane] : 0u;
        uint32_t x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        s_cnt[lane] = x - c;
        if (lane == 31) s_pos = x ? atomicAdd(j.n_live, x) : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (!m[u]) continue;  // warp-uniform
        const uint64_t i = first + (uint64_t)u * kLiveThreads;
        const unsigned int pos = s_pos + s_cnt[u * kWarps + warp] + __popc(m[u] & below);
        if (any[u]) j.live[pos] = (uint32_t)i;
        if (any[u] && j.live_entry) j.live_entry[pos] = en[u];
        if (j.order) {
            // Every lane takes part in the match (lanes without a live edge with a cell of
            // their own, kCells + lane), so that the mask is the full warp.
            const uint32_t cell = any[u] ? edge_cell(j, i) : (uint32_t)kCells + lane;
            const unsigned int peers = __match_any_sync(0xffffffffu, cell);
            const int leader = __ffs(peers) - 1;
            unsigned int r0 = 0;
            if (any[u] && lane == leader) r0 = atomicAdd(&j.cells[cell], (unsigned int)__popc(peers));
            r0 = __shfl_sync(0xffffffffu, r0, leader);
            if (any[u]) j.rank[pos] = r0 + __popc(peers & below);
        }
    }
}

__global__ void __launch_bounds__(kLiveThreads, 8) k_edge_live(EdgeJob j0, EdgeJob j1, unsigned int blocks0) {
    const bool second = blockIdx.x >= blocks0;
    const EdgeJob& j = second ? j1 : j0;
    const uint64_t base = (uint64_t)(blockIdx.x - (second ? blocks0 : 0u)) * blockDim.x * kLiveEdges + threadIdx.x;
    int ns[kLiveEdges], off[kLiveEdges];
    int32_t so0[kLiveEdges];
    uint8_t c0[kLiveEdges];
    uint32_t en[kLiveEdges];
#pragma unroll
    for (int u = 0; u < kLiveEdges; ++u) {
        const uint64_t i = base + (uint64_t)u * blockDim.x;
        const bool valid = i < j.nE;
        ns[u] = valid ? j.p.counts[i] : 0;
        off[u] = valid ? j.p.offsets[i] : 0;
    }
#pragma unroll
    for (int u = 0; u < kLiveEdges; ++u) so0[u] = ns[u] > 0 ? j.p.sources[off[u]] : -1;
#pragma unroll
    for (int u = 0; u < kLiveEdges; ++u) {
        const bool in = ns[u] > 0 && so0[u] >= 0 && (uint64_t)so0[u] < j.n_cull;
        c0[u] = in ? j.cull[so0[u]] : (uint8_t)0;
        // One source: its entry node (its partner query ran when its flag is set); more
        // sources: the root.
        en[u] = (j.entry && in && ns[u] == 1) ? j.entry[so0[u]] : 0u;
    }
    bool any[kLiveEdges];
#pragma unroll
    for (int u = 0; u < kLiveEdges; ++u)
        any[u] = ns[u] > 0 && edge_is_live(j, base + (uint64_t)u * blockDim.x, ns[u], j.p.sources + off[u], so0[u], c0[u]);
    live_append<kLiveEdges>(j, base, any, en);
}

// Slab index of an edge payload (rs_edge_index).  The reference's payload is in std::map
// order of its edges' quantised endpoint pairs, lower endpoint first
// (EdgePreprocessor.cpp:41-119: llround(x * 1e5) per coordinate), so it is sorted by the
// quantised x of each edge's lower endpoint -- the smaller of its two quantised x.  Slab b
// holds edges [b * kSlab, (b + 1) * kSlab); index[3 + b] is the key of its first edge.
// index[0] = 1 when the keys never decrease and no source id is negative (else 0),
// index[1] = the largest source id, index[2] = the edge count it was built for.  The
// live-edge check then visits only the slabs whose key range meets the quantised x range
// of an object with a partner: every edge of an object lies between its box's quantised x
// bounds (llround is monotone), and every live edge has such a source.
constexpr uint64_t kSlab = 256;

__device__ __forceinline__ long long edge_key_x(const EdgePayload& p, uint64_t e) {
    return min(llround((double)p.starts[3 * e] * 1e5), llround((double)p.ends[3 * e] * 1e5));
}

// word[0]: 1 once a key decreases or a source id is negative; word[1]: the largest source id.
__global__ void __launch_bounds__(256) k_edge_index(EdgePayload p, uint64_t nE, uint64_t nS,
                                                    long long* __restrict__ index, int* __restrict__ word) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    bool bad = false;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < nE; e += stride) {
        const long long x = edge_key_x(p, e);
        if (e % kSlab == 0) index[3 + e / kSlab] = x;
        if (e + 1 < nE && edge_key_x(p, e + 1) < x) bad = true;
    }
    int mx = -1;
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < nS; k += stride) {
        const int src = p.sources[k];
        bad |= src < 0;
        mx = max(mx, src);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&word[0], 1);
    if ((threadIdx.x & 31) == 0) atomicMax(&word[1], mx);
}

__global__ void k_edge_index_head(long long* __restrict__ index, const int* __restrict__ word, uint64_t nE) {
    index[0] = word[0] ? 0 : 1;
    index[1] = word[1];
    index[2] = (long long)nE;
}

// Slabs of each job that may hold a live edge, one warp per source object: an object with
// a partner (flag set) covers the slabs whose keys can fall in its box's quantised x range.
// A payload whose index says it is not in key order, was built for another edge count, or
// whose source ids reach past the flags, covers every slab (each edge is then checked, as
// without an index).  Blocks below blocks0 run job j0, the others j1.
constexpr int kMarkWarps = 8;

__global__ void __launch_bounds__(32 * kMarkWarps) k_slab_mark(EdgeJob j0, EdgeJob j1, unsigned int blocks0) {
    const bool second = blockIdx.x >= blocks0;
    const EdgeJob& j = second ? j1 : j0;
    const int lane = threadIdx.x & 31;
    const uint64_t o = (uint64_t)(blockIdx.x - (second ? blocks0 : 0u)) * kMarkWarps + (threadIdx.x >> 5);
    const long long* xq = j.xindex + 3;
    const bool ordered =
        j.xindex[0] == 1 && j.xindex[1] < (long long)j.n_cull && j.xindex[2] == (long long)j.nE;
    if (!ordered) {
        if (o == 0)
            for (uint64_t b = lane; b < j.n_slab; b += 32) j.covered[b] = 1;
        return;
    }
    if (o >= j.n_cull || j.cull[o] == 0) return;
    const float lo = ord2f(j.sbox[6 * o]), hi = ord2f(j.sbox[6 * o + 3]);
    if (!(lo <= hi)) return;  // no triangles, hence no edges
    const long long qlo = llround((double)lo * 1e5), qhi = llround((double)hi * 1e5);
    // first slab whose first key is >= qlo (the one before it may hold keys >= qlo too), and
    // the last slab whose first key is <= qhi.
    uint64_t a = 0, b = j.n_slab;
    while (a < b) {
        const uint64_t m = (a + b) / 2;
        if (xq[m] < qlo) a = m + 1;
        else b = m;
    }
    const uint64_t first = a > 0 ? a - 1 : 0;
    a = 0;
    b = j.n_slab;
    while (a < b) {
        const uint64_t m = (a + b) / 2;
        if (xq[m] <= qhi) a = m + 1;
        else b = m;
    }
    if (a == 0) return;  // every key is above qhi
    for (uint64_t s = first + lane; s < a; s += 32) j.covered[s] = 1;
}

// The live-edge check of k_edge_live over the covered slabs only, one block (kSlab threads)
// per slab.  Blocks below blocks0 run job j0, the others j1.
__global__ void __launch_bounds__(kSlab) k_edge_live_slab(EdgeJob j0, EdgeJob j1, unsigned int blocks0) {
    const bool second = blockIdx.x >= blocks0;
    const EdgeJob& j = second ? j1 : j0;
    const uint64_t sl = blockIdx.x - (second ? blocks0 : 0u);
    if (sl >= j.n_slab || !j.covered[sl]) return;  // block-uniform
    const uint64_t i = sl * kSlab + threadIdx.x;
    const bool valid = i < j.nE;
    const int ns = valid ? j.p.counts[i] : 0;
    const int off = valid ? j.p.offsets[i] : 0;
    const int32_t so0 = ns > 0 ? j.p.sources[off] : -1;
    const bool in = ns > 0 && so0 >= 0 && (uint64_t)so0 < j.n_cull;
    const uint8_t c0 = in ? j.cull[so0] : (uint8_t)0;
    const uint32_t en[1] = {(j.entry && in && ns == 1) ? j.entry[so0] : 0u};
    const bool any[1] = {ns > 0 && edge_is_live(j, i, ns, j.p.sources + off, so0, c0)};
    static_assert(kSlab == kLiveThreads, "one slab per block");
    live_append<1>(j, i, any, en);
}

// Exclusive prefix sums of the kCells cell counts of each binned job, in place (one block
// of 1024 threads per job, 32 cells per thread).
__global__ void __launch_bounds__(1024) k_cell_scan(uint32_t* c0, uint32_t* c1, const unsigned int* __restrict__ n0,
                                                   const unsigned int* __restrict__ n1) {
    __shared__ uint32_t warp_sum[32];
    uint32_t* c = blockIdx.x ? c1 : c0;
    if (!c || *(blockIdx.x ? n1 : n0) < kBinMinLive) return;
    constexpr int kPer = kCells / 1024;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    uint32_t v[kPer];
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        v[k] = c[t * kPer + k];
        sum += v[k];
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warp_sum[w] = inc;
    __syncthreads();
    if (w == 0) {
        uint32_t x = warp_sum[lane], xi = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, xi, o);
            if (lane >= o) xi += y;
        }
        warp_sum[lane] = xi - x;
    }
    __syncthreads();
    uint32_t run = warp_sum[w] + inc - sum;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        c[t * kPer + k] = run;
        run += v[k];
    }
}

// Live edges of the binned jobs into cell order.  Blocks below blocks0 run j0, the others
// j1, each job's blocks striding over its live list.
__global__ void __launch_bounds__(256) k_edge_order(EdgeJob j0, EdgeJob j1, unsigned int blocks0,
                                                    unsigned int blocks1) {
    const bool second = blockIdx.x >= blocks0;
    const EdgeJob& j = second ? j1 : j0;
    if (!j.order) return;
    const unsigned int nb = second ? blocks1 : blocks0;
    const unsigned int n = *j.n_live;
    if (n < kBinMinLive) return;
    for (unsigned int k = (blockIdx.x - (second ? blocks0 : 0u)) * blockDim.x + threadIdx.x; k < n;
         k += nb * blockDim.x) {
        const uint32_t e = j.live[k];
        const uint32_t pos = j.cells[edge_cell(j, e)] + j.rank[k];
        if (pos < n) {  // always: the cell is recomputed with the same arithmetic
            j.order[pos] = e;
            if (j.order_entry) j.order_entry[pos] = j.live_entry[k];
        }
    }
}

// A stream per device for the second direction's rays, forked from and joined back into
// the join's stream, with its two events, created once.  The caller holds *lock (the
// device's mutex) from recording the fork event until the join's stream waits on the
// joined event, so that host threads never record over each other's events.  False when
// they cannot be had: both directions then run on the join's stream.
bool ray_side_stream(cudaStream_t* st_out, cudaEvent_t* fork, cudaEvent_t* joined, std::unique_lock<std::mutex>* lock) {
    struct Side {
        cudaStream_t st = nullptr;
        cudaEvent_t fork = nullptr, joined = nullptr;
        bool ok = false;
        std::mutex mu;
    };
    static Side side[64];
    static std::mutex create_mu;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return false;
    Side& x = side[dev];
    std::lock_guard<std::mutex> g(create_mu);
    if (!x.ok) {
        x.ok = cudaStreamCreateWithFlags(&x.st, cudaStreamNonBlocking) == cudaSuccess &&
               cudaEventCreateWithFlags(&x.fork, cudaEventDisableTiming) == cudaSuccess &&
               cudaEventCreateWithFlags(&x.joined, cudaEventDisableTiming) == cudaSuccess;
        if (!x.ok) {
            cudaGetLastError();
            return false;
        }
    }
    *st_out = x.st;
    *fork = x.fork;
    *joined = x.joined;
    *lock = std::unique_lock<std::mutex>(x.mu);
    return true;
}

__global__ void k_first_tri_init(int32_t* __restrict__ first, uint64_t nObj, unsigned int* __restrict__ n_left) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i == 0) *n_left = 0;
    if (i < nObj) first[i] = INT_MAX;
}

// The lowest triangle of every object.  Only the first triangle of a run of one object can be
// it: with a triangle's atomic each, the 5,500 triangles an object of a 16.5 M-triangle set
// queued on one word and took 4.5 ms; its 3,000 runs take the pass over t2o.
constexpr int kFirstPer = 4;  // triangles a thread

__global__ void __launch_bounds__(256) k_first_tri(const int32_t* __restrict__ t2o, uint64_t nF,
                                                   int32_t* __restrict__ first, uint64_t nObj) {
    const uint64_t base = blockIdx.x * (uint64_t)(256 * kFirstPer) + threadIdx.x;
    int32_t o[kFirstPer], before[kFirstPer];
#pragma unroll
    for (int k = 0; k < kFirstPer; ++k) {
        const uint64_t t = base + 256 * (uint64_t)k;
        o[k] = t < nF ? __ldg(&t2o[t]) : -1;
        before[k] = t < nF && t > 0 ? __ldg(&t2o[t - 1]) : -1;
    }
#pragma unroll
    for (int k = 0; k < kFirstPer; ++k)
        if (o[k] >= 0 && o[k] != before[k] && (uint64_t)o[k] < nObj)
            atomicMin(&first[o[k]], (int32_t)(base + 256 * (uint64_t)k));
}

__global__ void k_max_obj(const int32_t* __restrict__ t2o, uint64_t nF, int* __restrict__ mx) {
    int m = -1;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < nF; t += (uint64_t)gridDim.x * blockDim.x)
        m = max(m, t2o[t]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(mx, m);
}

// --- broad phase of the overlap join ---------------------------------------------------
//
// If the slab test of an edge ray passes for a triangle box, each coordinate range of
// the ray's segment [1e-6, len + 1e-6] comes within 1.1e-6 + 7u*L of that box (u =
// 2^-24, L = edge length; the slab, direction and length arithmetic rounds at most
// seven times relative to L).  The segment lies in the box of every source object of
// the edge up to the edge payload's 1e-5 endpoint quantisation (a shared edge carries
// its first object's endpoints).  Boxes are therefore compared widened: the triangle
// box by kCullRel * (largest |coordinate| + extent) per axis, the object box by that
// and kCullAbs; the sum covers 1.2e-5 + 7u*L more than five times over (L <= the
// object box's extent).  An object whose widened box overlaps no widened triangle box
// of the other set cannot be the source of a pair, so its edges are not traced.  Each
// set's flags come from its own objects' queries against the other set's BVH.


__global__ void k_obj_box_init(int* __restrict__ box, uint64_t n_obj) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i < 6 * n_obj) box[i] = (i % 6) < 3 ? 0x7fffffff : (int)0x80000000;
}

// Object boxes from the leaf-ordered triangles (consecutive leaves mostly share an
// object, so lanes with equal objects reduce first and one lane updates the box).
__global__ void k_obj_boxes(const float4* __restrict__ tris, uint64_t n, int* __restrict__ box, uint64_t n_obj) {
    const uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float4 p = __ldg(&tris[3 * k]), q = __ldg(&tris[3 * k + 1]), r = __ldg(&tris[3 * k + 2]);
    const int32_t obj = __float_as_int(q.w);
    int v[6] = {f2ord(fminf(fminf(p.x, q.x), r.x)), f2ord(fminf(fminf(p.y, q.y), r.y)),
                f2ord(fminf(fminf(p.z, q.z), r.z)), f2ord_max(fmaxf(fmaxf(p.x, q.x), r.x)),
                f2ord_max(fmaxf(fmaxf(p.y, q.y), r.y)), f2ord_max(fmaxf(fmaxf(p.z, q.z), r.z))};
    const unsigned int peers = __match_any_sync(__activemask(), obj);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        v[c] = __reduce_min_sync(peers, v[c]);
        v[3 + c] = __reduce_max_sync(peers, v[3 + c]);
    }
    if ((int)(threadIdx.x & 31) != __ffs(peers) - 1) return;
    if (obj < 0 || (uint64_t)obj >= n_obj) return;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        atomicMin(&box[6 * (uint64_t)obj + c], v[c]);
        atomicMax(&box[6 * (uint64_t)obj + 3 + c], v[3 + c]);
    }
}

// [l, h] widened by its margin overlaps the (already widened) query box.
__device__ __forceinline__ bool cull_overlap(float l0, float l1, float l2, float h0, float h1, float h2,
                                             const float* qlo, const float* qhi) {
    const float m0 = cull_margin(l0, h0), m1 = cull_margin(l1, h1), m2 = cull_margin(l2, h2);
    return l0 - m0 <= qhi[0] && h0 + m0 >= qlo[0] && l1 - m1 <= qhi[1] && h1 + m1 >= qlo[1] &&
           l2 - m2 <= qhi[2] && h2 + m2 >= qlo[2];
}

// The objects of one set (their boxes) queried against the other set's BVH.
struct CullJob {
    const int* box;  // ordered-int min xyz, max xyz per object
    uint64_t n_obj;
    const BNode* nodes;
    uint32_t max_steps;
    const float4* tris;
    uint8_t* cand;
    int32_t* part;    // nullable: partner lists (kPartners per object)
    uint32_t* entry;  // nullable (partner mode): entry node per object queried
    // Nullable (partner mode): the other set's object boxes, and the number of them that
    // overlap each object's box (k_box_pairs).
    const int* obox;
    uint64_t n_other;
    uint32_t* most;
};

// Flag pass, one thread per object of one set: does its widened box overlap any widened
// triangle box of the other set's BVH?  cand[o] = 1 on the first overlap, or when the query
// runs out of its node budget or stack; 0 otherwise.  Node boxes contain their triangles'
// boxes and the widening grows with the box, so node culling is conservative.  Most
// objects of a sparse join overlap nothing, and a lone thread answers that in one descent.
// Blocks below blocks0 run job j0, the others j1 (both directions of a join in one launch).
constexpr uint32_t kFlagBudget = 256;  // node visits of a flag query

__global__ void __launch_bounds__(kT) k_cull_flag(CullJob j0, CullJob j1, unsigned int blocks0) {
    const bool second = blockIdx.x >= blocks0;
    const CullJob j = second ? j1 : j0;
    const uint64_t a = (uint64_t)(blockIdx.x - (second ? blocks0 : 0u)) * blockDim.x + threadIdx.x;
    if (a >= j.n_obj) return;
    const BNode* __restrict__ nodes = j.nodes;
    const float4* __restrict__ tris = j.tris;
    float qlo[3], qhi[3];
    bool empty = false;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float l = ord2f(j.box[6 * a + c]), h = ord2f(j.box[6 * a + 3 + c]);
        empty |= !(l <= h);
        const float m = kCullAbs + cull_margin(l, h);
        qlo[c] = l - m;
        qhi[c] = h + m;
    }
    if (empty) {  // no triangle of this object, hence no edges
        j.cand[a] = 0;
        return;
    }
    int stack[kStack];
    int sp = 0, node = 0;
    uint8_t result = 0;
    const uint32_t budget = min(j.max_steps, kFlagBudget);
    for (uint32_t step = 0;; ++step) {
        if (step > budget) {
            result = 1;
            break;
        }
        const BNode bn = load_node(nodes, node);
        const float4 na = bn.a, nb = bn.b, nc = bn.c;
        const int4 nd = bn.d;
        bool h0 = cull_overlap(na.x, na.y, na.z, na.w, nb.x, nb.y, qlo, qhi);
        bool h1 = cull_overlap(nb.z, nb.w, nc.x, nc.y, nc.z, nc.w, qlo, qhi);
#pragma unroll 1
        for (int side = 0; side < 2 && !result; ++side) {
            const bool h = side == 0 ? h0 : h1;
            const int first = side == 0 ? nd.x : nd.z, cnt = side == 0 ? nd.y : nd.w;
            if (!h || cnt == 0) continue;
            for (int k = first; k < first + cnt; ++k) {
                const float4 p = __ldg(&tris[3 * (size_t)k]), q = __ldg(&tris[3 * (size_t)k + 1]),
                             r = __ldg(&tris[3 * (size_t)k + 2]);
                if (cull_overlap(fminf(fminf(p.x, q.x), r.x), fminf(fminf(p.y, q.y), r.y),
                                 fminf(fminf(p.z, q.z), r.z), fmaxf(fmaxf(p.x, q.x), r.x),
                                 fmaxf(fmaxf(p.y, q.y), r.y), fmaxf(fmaxf(p.z, q.z), r.z), qlo, qhi)) {
                    result = 1;
                    break;
                }
            }
        }
        if (result) break;
        if (nd.y > 0) h0 = false;
        if (nd.w > 0) h1 = false;
        if (h0 && h1) {
            if (sp == kStack) {
                result = 1;
                break;
            }
            stack[sp++] = nd.z;
            node = nd.x;
        } else if (h0) {
            node = nd.x;
        } else if (h1) {
            node = nd.z;
        } else {
            if (sp == 0) break;
            node = stack[--sp];
        }
    }
    j.cand[a] = result;
}

// Partner queries: the distinct objects of the other set's triangles whose widened boxes
// overlap an object's widened box go to part[o * kPartners ...] and cand[o] = their number,
// or kCandAll when there are more than kPartners or the queries ran out of budget or stack.
//
// Also recorded is the object's entry node: the deepest node of the walk's opening chain,
// where each step hits no leaf and one inner child.  Every triangle whose widened box
// overlaps the object's widened box lies under it, so the rays of the object's edges (whose
// boxes lie inside that box) may start there instead of at the root and still meet every
// triangle they can hit.
//
// A warp takes as many objects as give every resident warp a packet.  Each lane walks its
// object's opening chain alone (most objects of a sparse join end there), then the warp's
// (node, object) pairs lie on one shared-memory stack and its (leaf, object) pairs in a ring,
// as in the ray packets: each step pops up to 32 nodes, and 32 leaves at a time are tested.
// A partner takes the first free place of its object's list by compare-and-swap; an object
// whose list is full drops out, and so does one that has found as many partners as there are
// boxes overlapping its own (most, nullable): a large object otherwise walks thousands of
// nodes of a partner that it found at the first.  A thread per object for the flags and a warp
// per object for the partners took 1,070 us on 3,001 + 3,001 uneven objects and 260 on 10k +
// 10k dense ones, a warp's lanes a quarter full; this takes 640 (with k_box_pairs) and 176.
constexpr int kCullWarps = 4;
constexpr int kCullResident = 8;           // blocks an SM holds
constexpr int kCullStack = 384;            // (node, object) pairs
constexpr int kCullRing = 128;             // (leaf, object) pairs
constexpr uint32_t kPartnerBudget = 8192;  // node visits per object of a packet

struct CullPacket {
    float4 lo[32], hi[32];  // widened boxes of the packet's objects
    int node[kCullStack];
    uint2 leaf[kCullRing];  // first triangle; count << 5 | object
    int32_t part[kPartners][32];
    int state[32];          // 0 searching, 1 every object is a candidate, 2 all partners found
    int most[32];           // partners there can be
    unsigned char own[kCullStack];
};

// For every object of one set, the number of the other set's objects whose widened boxes
// overlap its own, and the first kPartners of them as its partner list: every partner is among
// them, since a triangle's box lies in its object's -- in a set without triangles of an id below
// zero, which are a partner of no box: such a set has no lists.  One warp per object.
__global__ void __launch_bounds__(256) k_box_pairs(CullJob j0, CullJob j1, unsigned int blocks0) {
    const bool second = blockIdx.x >= blocks0;
    const CullJob j = second ? j1 : j0;
    const uint64_t a = (uint64_t)(blockIdx.x - (second ? blocks0 : 0u)) * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (a >= j.n_obj) return;
    float qlo[3], qhi[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float l = ord2f(j.box[6 * a + c]), h = ord2f(j.box[6 * a + 3 + c]);
        const float m = kCullAbs + cull_margin(l, h);
        qlo[c] = l - m;
        qhi[c] = h + m;
    }
    uint32_t n = 0;
    for (uint64_t b0 = 0; b0 < j.n_other; b0 += 32) {
        const uint64_t b = b0 + lane;
        const bool in = b < j.n_other && box_overlaps(j.obox + 6 * b, qlo, qhi);
        const unsigned int m = __ballot_sync(0xffffffffu, in);
        const uint32_t at = n + __popc(m & ((1u << lane) - 1u));
        if (in && at < kPartners) j.part[a * kPartners + at] = (int32_t)b;
        n += __popc(m);
    }
    if (lane == 0) j.most[a] = n;
}

__global__ void __launch_bounds__(32 * kCullWarps, kCullResident) k_cull_query(CullJob j0, CullJob j1, unsigned int packets0,
                                                                unsigned int packets, uint32_t size) {
    constexpr unsigned int kAll = 0xffffffffu;
    __shared__ CullPacket s_packet[kCullWarps];
    CullPacket& sm = s_packet[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned int below = (1u << lane) - 1u;
    for (unsigned int pk = blockIdx.x * kCullWarps + (threadIdx.x >> 5); pk < packets; pk += gridDim.x * kCullWarps) {
        const bool second = pk >= packets0;
        const BNode* __restrict__ nodes = second ? j1.nodes : j0.nodes;
        const float4* __restrict__ tris = second ? j1.tris : j0.tris;
        const uint64_t n_obj = second ? j1.n_obj : j0.n_obj;
        const uint32_t max_steps = second ? j1.max_steps : j0.max_steps;
        const uint64_t a = (uint64_t)(pk - (second ? packets0 : 0u)) * size + lane;
        const bool mine = (uint32_t)lane < size && a < n_obj;
        float qlo[3] = {0.0f, 0.0f, 0.0f}, qhi[3] = {0.0f, 0.0f, 0.0f};
        int most = 0x7fffffff;
        bool query = mine;
        if (mine) {
            const uint32_t* m = second ? j1.most : j0.most;
            if (m) most = (int)min(m[a], 0x7fffffffu);
            query = most > 0;
            const int* box = (second ? j1.box : j0.box) + 6 * a;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float l = ord2f(box[c]), h = ord2f(box[3 + c]);
                query = query && l <= h;  // else no triangle of this object, hence no edges
                const float m = kCullAbs + cull_margin(l, h);
                qlo[c] = l - m;
                qhi[c] = h + m;
            }
        }
        // The opening chain, alone.
        int entry = 0;
        for (uint32_t step = 0; query && step < max_steps; ++step) {
            const BNode bn = load_node(nodes, entry);
            const bool h0 = cull_overlap(bn.a.x, bn.a.y, bn.a.z, bn.a.w, bn.b.x, bn.b.y, qlo, qhi);
            const bool h1 = cull_overlap(bn.b.z, bn.b.w, bn.c.x, bn.c.y, bn.c.z, bn.c.w, qlo, qhi);
            if (!h0 && !h1) query = false;
            if (h0 == h1 || (h0 ? bn.d.y : bn.d.w) > 0) break;
            entry = h0 ? bn.d.x : bn.d.z;
        }
        sm.lo[lane] = make_float4(qlo[0], qlo[1], qlo[2], 0.0f);
        sm.hi[lane] = make_float4(qhi[0], qhi[1], qhi[2], 0.0f);
#pragma unroll
        for (int k = 0; k < kPartners; ++k) sm.part[k][lane] = -1;
        sm.state[lane] = 0;
        sm.most[lane] = most;
        const unsigned int queried = __ballot_sync(kAll, query);
        if (query) {
            const int at = __popc(queried & below);
            sm.node[at] = entry;
            sm.own[at] = (unsigned char)lane;
        }
        __syncwarp();
        int sp = __popc(queried);
        uint32_t head = 0, queued = 0, visits = 0;
        const uint32_t budget = kPartnerBudget * (uint32_t)sp;
        bool ok = true;
        while (sp > 0 || queued > 0) {
            if (queued >= 32u || sp == 0) {
                const uint32_t m = min(queued, 32u);
                const uint2 leaf = (uint32_t)lane < m ? sm.leaf[(head + lane) & (kCullRing - 1)] : make_uint2(0u, 0u);
                head += m;
                queued -= m;
                const int cnt = (int)(leaf.y >> 5), o = (int)(leaf.y & 31u);
                for (int k = 0; k < cnt && !sm.state[o]; ++k) {
                    const size_t t = 3 * ((size_t)leaf.x + k);
                    const float4 q = __ldg(&tris[t + 1]);
                    const int32_t pobj = __float_as_int(q.w);
                    bool known = false;
#pragma unroll
                    for (int u = 0; u < kPartners; ++u) known |= sm.part[u][o] == pobj;
                    if (known && pobj >= 0) continue;
                    const float4 p = __ldg(&tris[t]), r = __ldg(&tris[t + 2]);
                    const float4 l = sm.lo[o], h = sm.hi[o];
                    const float blo[3] = {l.x, l.y, l.z}, bhi[3] = {h.x, h.y, h.z};
                    if (!cull_overlap(fminf(fminf(p.x, q.x), r.x), fminf(fminf(p.y, q.y), r.y),
                                      fminf(fminf(p.z, q.z), r.z), fmaxf(fmaxf(p.x, q.x), r.x),
                                      fmaxf(fmaxf(p.y, q.y), r.y), fmaxf(fmaxf(p.z, q.z), r.z), blo, bhi))
                        continue;
                    int u = pobj < 0 ? kPartners : 0;  // -1 marks a free place
                    for (; u < kPartners; ++u) {
                        const int32_t old = atomicCAS(&sm.part[u][o], -1, pobj);
                        if (old == -1 || old == pobj) break;
                    }
                    if (u == kPartners) sm.state[o] = 1;
                    else if (u + 1 == sm.most[o]) sm.state[o] = 2;
                }
                __syncwarp();
                continue;
            }
            const int take = min(min(sp, 32), max(kCullStack - kStackRoom - sp, 1));
            sp -= take;
            visits += (uint32_t)take;
            if (visits > budget) {
                ok = false;
                sp += take;
                break;
            }
            bool h0 = false, h1 = false;
            int o = 0;
            int4 nd = make_int4(0, 0, 0, 0);
            if (lane < take) {
                o = sm.own[sp + lane];
                if (!sm.state[o]) {
                    const BNode bn = load_node(nodes, sm.node[sp + lane]);
                    const float4 l = sm.lo[o], h = sm.hi[o];
                    const float blo[3] = {l.x, l.y, l.z}, bhi[3] = {h.x, h.y, h.z};
                    h0 = cull_overlap(bn.a.x, bn.a.y, bn.a.z, bn.a.w, bn.b.x, bn.b.y, blo, bhi);
                    h1 = cull_overlap(bn.b.z, bn.b.w, bn.c.x, bn.c.y, bn.c.z, bn.c.w, blo, bhi);
                    nd = bn.d;
                }
            }
            __syncwarp();  // popped entries are read before they are overwritten
            const bool l0 = h0 && nd.y > 0, l1 = h1 && nd.w > 0;
            const unsigned int ml0 = __ballot_sync(kAll, l0), ml1 = __ballot_sync(kAll, l1);
            const uint32_t at = head + queued;
            if (l0)
                sm.leaf[(at + __popc(ml0 & below)) & (kCullRing - 1)] =
                    make_uint2((uint32_t)nd.x, (uint32_t)nd.y << 5 | (uint32_t)o);
            if (l1)
                sm.leaf[(at + __popc(ml0) + __popc(ml1 & below)) & (kCullRing - 1)] =
                    make_uint2((uint32_t)nd.z, (uint32_t)nd.w << 5 | (uint32_t)o);
            queued += __popc(ml0) + __popc(ml1);
            const bool p0 = h0 && nd.y <= 0, p1 = h1 && nd.w <= 0;
            const unsigned int mp0 = __ballot_sync(kAll, p0), mp1 = __ballot_sync(kAll, p1);
            const int pushed = __popc(mp0) + __popc(mp1);
            if (sp + pushed > kCullStack) {  // the popped objects lose a node
                if (lane < take && sm.state[o] == 0) sm.state[o] = 1;
                __syncwarp();
                continue;
            }
            if (p0) {
                const int i = sp + __popc(mp0 & below);
                sm.node[i] = nd.x;
                sm.own[i] = (unsigned char)o;
            }
            if (p1) {
                const int i = sp + __popc(mp0) + __popc(mp1 & below);
                sm.node[i] = nd.z;
                sm.own[i] = (unsigned char)o;
            }
            sp += pushed;
            __syncwarp();
        }
        if (!ok) {  // objects with something left
            for (int i = lane; i < sp; i += 32)
                if (sm.state[sm.own[i]] == 0) sm.state[sm.own[i]] = 1;
            for (uint32_t i = lane; i < queued; i += 32) {
                const uint32_t o = sm.leaf[(head + i) & (kCullRing - 1)].y & 31u;
                if (sm.state[o] == 0) sm.state[o] = 1;
            }
        }
        __syncwarp();
        if (mine) {
            // A walk cut short keeps the list of overlapping boxes, when that is whole.
            most = sm.most[lane];
            const bool cut = sm.state[lane] == 1, boxes = cut && most <= kPartners;
            int32_t* part = (second ? j1.part : j0.part) + a * kPartners;
            uint32_t* en = second ? j1.entry : j0.entry;
            int np = 0;
#pragma unroll
            for (int u = 0; u < kPartners; ++u) {
                const int32_t b = sm.part[u][lane];
                np += b >= 0;
                if (!boxes) part[u] = b;
            }
            (second ? j1.cand : j0.cand)[a] = boxes ? (uint8_t)most : cut ? kCandAll : (uint8_t)np;
            if (en) en[a] = (uint32_t)entry;
        }
        __syncwarp();
    }
}

// Optional per-source outputs of the containment pass (the reference's pair-hit and
// containment-tracking buffers, query/src/utilities/PairHitTracking.h,
// ContainmentTracking.h): distinct targets crossed, and the odd-parity targets with
// their crossing counts (traversal order within each pass).
struct Tracking {
    int max_targets;
    int32_t* target_ids;      // [nObj * max_targets], -1 where unused
    uint32_t* target_hits;    // [nObj * max_targets]
    uint32_t* candidates;     // [nObj]
};

// The ray of source object o; false when it has none.
__device__ __forceinline__ bool containment_ray(const float* __restrict__ V, uint64_t nV,
                                                const uint32_t* __restrict__ I, const int32_t* __restrict__ first,
                                                uint64_t o, Ray& r) {
    const int32_t ft = first[o];
    if (ft == INT_MAX) return false;
    const uint32_t vi = I[3 * (uint64_t)ft];
    if (vi >= nV) return false;
    r = make_ray(V[3 * (uint64_t)vi], V[3 * (uint64_t)vi + 1], V[3 * (uint64_t)vi + 2], 0.0f, 0.0f, 1.0f, 1e-4f, 1e10f);
    return true;
}

__device__ __forceinline__ unsigned long long containment_key(uint64_t o, uint32_t target, int swap) {
    return swap ? (((unsigned long long)target << 32) | (uint32_t)o)
                : (((unsigned long long)(uint32_t)o << 32) | target);
}

// One object's ray by one thread, any number of targets.
template <bool TRACK>
__device__ __forceinline__ void containment_thread(const Ray& r, uint64_t o, const BNode* __restrict__ nodes,
                                                   uint32_t max_steps, const float4* __restrict__ tris, int swap,
                                                   const PairTable& table, const Tracking& trk) {
    // Parity per target object in passes of at most kTargets objects: pass p tracks the
    // kTargets smallest object ids (as uint32) above the largest id of pass p-1.  A list
    // member is inserted at its first crossing and never evicted (evictions only drop the
    // largest member for a smaller newcomer, and the largest only decreases), so every
    // tracked parity is complete; a pass that had to turn an id away runs another pass.
    uint32_t tgt[kTargets];
    uint32_t hits[TRACK ? kTargets : 1];
    uint32_t lo = 0;
    bool bounded = false;
    unsigned int crossings = 0, candidates = 0, tests = 0;
    int out = 0;
    for (;;) {
        uint32_t par = 0;  // parity bit per list entry
        int nt = 0;
        bool more = false;
        const bool ok = traverse<2>(nodes, max_steps, r, [&](int f, int cnt) {
            for (int k = f; k < f + cnt; ++k) {
                float a[3], b[3], c[3];
                uint32_t tid;
                int32_t obj;
                load_tri(tris, k, a, b, c, tid, obj);
                const uint32_t id = (uint32_t)obj;
                if (bounded && id <= lo) continue;
                if (more && nt == kTargets && (bounded || !table.stats)) {  // above every member of a full list
                    uint32_t mx = 0;
                    for (int j = 0; j < nt; ++j) mx = max(mx, tgt[j]);
                    if (id > mx) continue;
                }
                float t;
                ++tests;
                if (!hit_triangle<2>(r, a, b, c, t)) continue;
                if (!bounded) ++crossings;
                int j = 0;
                for (; j < nt; ++j)
                    if (tgt[j] == id) break;
                if (j < nt) {
                    par ^= 1u << j;
                    if (TRACK) ++hits[j];
                } else if (nt < kTargets) {
                    tgt[nt] = id;
                    if (TRACK) hits[nt] = 1;
                    par |= 1u << nt;
                    ++nt;
                } else {
                    more = true;
                    int jm = 0;
                    for (int q = 1; q < nt; ++q)
                        if (tgt[q] > tgt[jm]) jm = q;
                    if (id < tgt[jm]) {
                        tgt[jm] = id;
                        if (TRACK) hits[jm] = 1;
                        par |= 1u << jm;
                    }
                }
            }
        });
        if (!ok) {
            atomicOr(table.status, ST_STACK_OVERFLOW);
            return;
        }
        candidates += (unsigned int)nt;
        uint32_t mx = 0;
        for (int j = 0; j < nt; ++j) {
            mx = max(mx, tgt[j]);
            if (!((par >> j) & 1u)) continue;
            table_insert(table, containment_key(o, tgt[j], swap));
            if (TRACK && out < trk.max_targets) {
                trk.target_ids[o * trk.max_targets + out] = (int32_t)tgt[j];
                trk.target_hits[o * trk.max_targets + out] = hits[j];
                ++out;
            }
        }
        if (!more) break;
        lo = mx;
        bounded = true;
    }
    add_tests(tests);
    if (table.stats) {
        atomicAdd(&table.stats[4], 1ull);
        if (crossings) atomicAdd(&table.stats[5], (unsigned long long)crossings);
        if (candidates) atomicAdd(&table.stats[6], (unsigned long long)candidates);
    }
    if (TRACK) trk.candidates[o] = candidates;
}

// One thread per object, with the per-source diagnostics.
__global__ void __launch_bounds__(kT) k_containment_tracked(const float* __restrict__ V, uint64_t nV,
                                                            const uint32_t* __restrict__ I,
                                                            const int32_t* __restrict__ first, uint64_t nObj,
                                                            const BNode* __restrict__ nodes, uint32_t max_steps,
                                                            const float4* __restrict__ tris, int swap, PairTable table,
                                                            Tracking trk) {
    const uint64_t o = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (o >= nObj) return;
    trk.candidates[o] = 0;
    for (int q = 0; q < trk.max_targets; ++q) {
        trk.target_ids[o * trk.max_targets + q] = -1;
        trk.target_hits[o * trk.max_targets + q] = 0;
    }
    Ray r;
    if (containment_ray(V, nV, I, first, o, r))
        containment_thread<true>(r, o, nodes, max_steps, tris, swap, table, trk);
}

// One warp per object: up to 32 nodes a step from a shared-memory stack, as the edge rays of
// short lists, and the object ids of all crossings in a list; a target is inserted when it
// occurs an odd number of times.  One thread per object made the join wait on its longest
// chain of dependent node loads, with one warp for 32 objects.
//
// A list that fills up keeps each object's parity, and when that leaves it half full or more,
// the lower half of its ids: the traversal goes on for them alone, and the next pass takes the
// ids above.  Left to the one-thread passes, with 31 lanes idle, 20,000 objects under 300 boxes
// (600 crossings) took 39.7 ms where a thread for each object had taken 4.2; now 1.15.  A step
// pops no more nodes than leave kStackRoom entries: a wide traversal turns into a depth-first
// one, and only a tree deeper than that runs out of stack and goes to the one-thread passes.
constexpr int kContWarps = 4;    // objects per block
constexpr int kContStack = 320;  // entries of a warp's stack
constexpr int kContHits = 512;   // crossings a warp keeps
// Objects from which rays are traced in packets first.  80,000 objects with a target of 3 large
// spheres, 20,000 and 100,000 dense ones: 298, 632 and 4,500 us with packets, 500, 735 and 3,970
// without (a thread an object: 410, 980, 54,000); 200,000 objects: 395, 1,190 and 9,590 against 895,
// 1,445 and 8,590.  At 40,000 packets save 100 us at most and cost 950 where every ray is long.
constexpr uint64_t kContPackets = 65536;

// Sorts the warp's list of nh ids and leaves one of an object that occurs an odd number of
// times, and none (even: two) of the others; then, from half of kContHits on, the ids up to the
// middle one, which becomes *up.  Returns the number left.
__device__ __noinline__ int fold_ids(uint32_t* ids, int nh, bool even, uint32_t* up) {
    constexpr unsigned int kAll = 0xffffffffu;
    constexpr int kPer = kContHits / 32;
    const int lane = threadIdx.x & 31;
    for (int i = nh + lane; i < kContHits; i += 32) ids[i] = 0xffffffffu;
    __syncwarp();
    for (int k = 2; k <= kContHits; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = lane; i < kContHits; i += 32) {
                const int q = i ^ j;
                if (q > i && (ids[i] > ids[q]) == ((i & k) == 0)) {
                    const uint32_t t = ids[i];
                    ids[i] = ids[q];
                    ids[q] = t;
                }
            }
            __syncwarp();
        }
    uint32_t v[kPer];
    unsigned int keep = 0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const int i = 32 * q + lane;
        v[q] = ids[i];
        if (i >= nh) continue;
        int lo = 0, hi = i;  // the first place of this id
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (ids[mid] < v[q]) lo = mid + 1;
            else hi = mid;
        }
        const bool last = i + 1 == nh || ids[i + 1] != v[q];
        const bool before_last = !last && (i + 2 == nh || ids[i + 2] != v[q]);
        const int count = i + (last ? 1 : 2) - lo;
        if ((last && (count & 1 || even)) || (before_last && !(count & 1) && even)) keep |= 1u << q;
    }
    __syncwarp();
    int n = 0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const unsigned int m = __ballot_sync(kAll, keep >> q & 1u);
        if (keep >> q & 1u) ids[n + __popc(m & ((1u << lane) - 1u))] = v[q];
        n += __popc(m);
    }
    __syncwarp();
    if (n < kContHits / 2) return n;
    *up = ids[n / 2 - 1];
    n = n / 2 < n && ids[n / 2] == *up ? n / 2 + 1 : n / 2;
    __syncwarp();
    return n;
}

// The object's crossings in passes of ids by the whole warp, for rays of more of them than one
// list holds, or of more nodes than its stack does.
__device__ __forceinline__ void containment_many(const Ray& r, uint64_t o, int* stack, uint32_t* ids,
                                                 const BNode* __restrict__ nodes, uint32_t max_steps,
                                                 const float4* __restrict__ tris, int swap, const PairTable& table) {
    constexpr unsigned int kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned int below = (1u << lane) - 1u;
    unsigned int tests = 0, crossings = 0, targets = 0;
    bool ok = true, bounded = false;
    uint32_t above = 0, up = 0xffffffffu;  // this pass: ids > above (bounded), <= up
    for (;;) {
        if (lane == 0) stack[0] = 0;
        __syncwarp();
        int sp = 1, nh = 0;
        uint32_t visits = 0;
        while (sp > 0) {
            const int take = min(min(sp, 32), max(kContStack - kStackRoom - sp, 1));
            const int node = lane < take ? stack[sp - take + lane] : -1;
            __syncwarp();
            sp -= take;
            visits += (uint32_t)take;
            bool h[2] = {false, false};
            int leaf[2] = {0, 0}, cnt[2] = {0, 0};
            if (node >= 0) {
                const BNode bn = load_node(nodes, node);
                const float4 na = bn.a, nb = bn.b, nc = bn.c;
                const int4 nd = bn.d;
                const float lo0[3] = {na.x, na.y, na.z}, hi0[3] = {na.w, nb.x, nb.y};
                const float lo1[3] = {nb.z, nb.w, nc.x}, hi1[3] = {nc.y, nc.z, nc.w};
                float en, ex;
                h[0] = slab<2>(r, lo0, hi0, r.tmin, r.tmax, en, ex);
                h[1] = slab<2>(r, lo1, hi1, r.tmin, r.tmax, en, ex);
                leaf[0] = nd.x;
                cnt[0] = nd.y;
                leaf[1] = nd.z;
                cnt[1] = nd.w;
            }
            const bool p0 = h[0] && cnt[0] == 0, p1 = h[1] && cnt[1] == 0;
            const unsigned b0 = __ballot_sync(kAll, p0), b1 = __ballot_sync(kAll, p1);
            const int pushed = __popc(b0) + __popc(b1);
            if (visits > max_steps || sp + pushed > kContStack) {
                ok = false;
                break;
            }
            int pos = sp + __popc(b0 & below) + __popc(b1 & below);
            if (p0) stack[pos++] = leaf[0];
            if (p1) stack[pos] = leaf[1];
            sp += pushed;
            // Triangles of the leaves hit: the first child's, then the second's.
            const int n0 = h[0] ? cnt[0] : 0, n1 = h[1] ? cnt[1] : 0;
            tests += (unsigned int)(n0 + n1);
            const int rounds = __reduce_max_sync(kAll, n0 + n1);
            for (int k = 0; k < rounds; ++k) {
                bool hit = false;
                uint32_t tid;
                int32_t obj = 0;
                if (k < n0 + n1) {
                    float a[3], b[3], c[3], t;
                    load_tri(tris, k < n0 ? leaf[0] + k : leaf[1] + (k - n0), a, b, c, tid, obj);
                    hit = hit_triangle<2>(r, a, b, c, t);
                }
                unsigned m = __ballot_sync(kAll, hit);
                if (!bounded) crossings += __popc(m);
                if (bounded || up != 0xffffffffu) {  // this pass leaves ids out
                    hit = hit && (uint32_t)obj <= up && !(bounded && (uint32_t)obj <= above);
                    m = __ballot_sync(kAll, hit);
                }
                if (nh + __popc(m) > kContHits) {  // the same in every lane
                    nh = fold_ids(ids, nh, table.stats != nullptr, &up);
                    hit = hit && (uint32_t)obj <= up;
                    m = __ballot_sync(kAll, hit);
                }
                if (hit) ids[nh + __popc(m & below)] = (uint32_t)obj;
                nh += __popc(m);
            }
            __syncwarp();
        }
        __syncwarp();
        if (!ok) break;
        unsigned int distinct = 0;
        for (int a = lane; a < nh; a += 32) {
            const uint32_t id = ids[a];
            int before = 0, all = 0;
            for (int b = 0; b < nh; ++b) {
                const bool same = ids[b] == id;
                all += same;
                before += same && b < a;
            }
            if (before) continue;  // its first occurrence decides
            ++distinct;
            if (all & 1) table_insert(table, containment_key(o, id, swap));
        }
        targets += distinct;
        __syncwarp();
        if (up == 0xffffffffu) break;
        above = up;
        up = 0xffffffffu;
        bounded = true;
    }
    if (!ok) {  // finds the pairs of the passes before again
        if (lane == 0) containment_thread<false>(r, o, nodes, max_steps, tris, swap, table, Tracking{});
        return;
    }
    add_tests(tests);
    if (table.stats) {
        targets = __reduce_add_sync(kAll, targets);
        if (lane == 0) {
            atomicAdd(&table.stats[4], 1ull);
            if (crossings) atomicAdd(&table.stats[5], (unsigned long long)crossings);
            if (targets) atomicAdd(&table.stats[6], (unsigned long long)targets);
        }
    }
}

// Objects 0..nObj-1, or list[0..*n_list).  Those left over follow when the warp is through with
// the others: called from the loop they cost the others up to 12 % (1,000 objects under 200 boxes
// 190 -> 218 us), in a launch of their own 2 % of a join of 150 objects.  deferred (nObj words):
// every warp has the places of the objects that it takes.  64 registers, some spilled, and 8
// blocks an SM beat 72 and 7: 200,000 objects in 100,000 spheres 9.6 ms against 11.0.
__global__ void __launch_bounds__(32 * kContWarps, 8) k_containment(
    const float* __restrict__ V, uint64_t nV, const uint32_t* __restrict__ I, const int32_t* __restrict__ first,
    uint64_t nObj, const BNode* __restrict__ nodes, uint32_t max_steps, const float4* __restrict__ tris, int swap,
    PairTable table, const uint32_t* __restrict__ list, const unsigned int* __restrict__ n_list, uint32_t* deferred) {
    constexpr unsigned int kAll = 0xffffffffu;
    __shared__ int s_stack[kContWarps][kContStack];
    __shared__ uint32_t s_id[kContWarps][kContHits];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const unsigned int below = (1u << lane) - 1u;
    int* stack = s_stack[wi];
    uint32_t* ids = s_id[wi];
    const uint64_t k0 = blockIdx.x * (uint64_t)kContWarps + wi, warps = (uint64_t)gridDim.x * kContWarps;
    const uint64_t n = list ? (uint64_t)*n_list : nObj;
    uint64_t left = k0;
    for (uint64_t k = k0; k < n; k += warps) {
        const uint64_t o = list ? list[k] : k;
        Ray r;
        if (!containment_ray(V, nV, I, first, o, r)) continue;  // the same in every lane
        if (lane == 0) stack[0] = 0;
        __syncwarp();
        int sp = 1, nh = 0;
        uint32_t visits = 0;
        bool ok = true;
        unsigned int tests = 0;
        while (sp > 0) {
            const int take = min(min(sp, 32), max(kContStack - kStackRoom - sp, 1));
            const int node = lane < take ? stack[sp - take + lane] : -1;
            __syncwarp();
            sp -= take;
            visits += (uint32_t)take;
            bool h[2] = {false, false};
            int leaf[2] = {0, 0}, cnt[2] = {0, 0};
            if (node >= 0) {
                const BNode bn = load_node(nodes, node);
                const float4 na = bn.a, nb = bn.b, nc = bn.c;
                const int4 nd = bn.d;
                const float lo0[3] = {na.x, na.y, na.z}, hi0[3] = {na.w, nb.x, nb.y};
                const float lo1[3] = {nb.z, nb.w, nc.x}, hi1[3] = {nc.y, nc.z, nc.w};
                float en, ex;
                h[0] = slab<2>(r, lo0, hi0, r.tmin, r.tmax, en, ex);
                h[1] = slab<2>(r, lo1, hi1, r.tmin, r.tmax, en, ex);
                leaf[0] = nd.x;
                cnt[0] = nd.y;
                leaf[1] = nd.z;
                cnt[1] = nd.w;
            }
            const bool p0 = h[0] && cnt[0] == 0, p1 = h[1] && cnt[1] == 0;
            const unsigned b0 = __ballot_sync(kAll, p0), b1 = __ballot_sync(kAll, p1);
            const int pushed = __popc(b0) + __popc(b1);
            if (visits > max_steps || sp + pushed > kContStack) {
                ok = false;
                break;
            }
            int pos = sp + __popc(b0 & below) + __popc(b1 & below);
            if (p0) stack[pos++] = leaf[0];
            if (p1) stack[pos] = leaf[1];
            sp += pushed;
            // Triangles of the leaves hit: the first child's, then the second's.
            const int n0 = h[0] ? cnt[0] : 0, n1 = h[1] ? cnt[1] : 0;
            tests += (unsigned int)(n0 + n1);
            const int rounds = __reduce_max_sync(kAll, n0 + n1);
            for (int k = 0; k < rounds; ++k) {
                bool hit = false;
                uint32_t tid;
                int32_t obj = 0;
                if (k < n0 + n1) {
                    float a[3], b[3], c[3], t;
                    load_tri(tris, k < n0 ? leaf[0] + k : leaf[1] + (k - n0), a, b, c, tid, obj);
                    hit = hit_triangle<2>(r, a, b, c, t);
                }
                const unsigned m = __ballot_sync(kAll, hit);
                const int at = nh + __popc(m & below);
                if (hit && at < kContHits) ids[at] = (uint32_t)obj;
                nh += __popc(m);
            }
            __syncwarp();
            if (nh > kContHits) break;
        }
        __syncwarp();
        if (!ok || nh > kContHits) {
            if (lane == 0) deferred[left] = (uint32_t)o;
            left += warps;
            __syncwarp();
            continue;
        }
        add_tests(tests);
        unsigned int distinct = 0;
        for (int a = lane; a < nh; a += 32) {
            const uint32_t id = ids[a];
            int before = 0, all = 0;
            for (int b = 0; b < nh; ++b) {
                const bool same = ids[b] == id;
                all += same;
                before += same && b < a;
            }
            if (before) continue;  // its first occurrence decides
            ++distinct;
            if (all & 1) table_insert(table, containment_key(o, id, swap));
        }
        if (table.stats) {
            distinct = __reduce_add_sync(kAll, distinct);
            if (lane == 0) {
                atomicAdd(&table.stats[4], 1ull);
                if (nh) atomicAdd(&table.stats[5], (unsigned long long)nh);
                if (distinct) atomicAdd(&table.stats[6], (unsigned long long)distinct);
            }
        }
        __syncwarp();
    }
    for (uint64_t k = k0; k < left; k += warps) {
        const uint64_t o = deferred[k];
        Ray r;
        if (containment_ray(V, nV, I, first, o, r)) containment_many(r, o, stack, ids, nodes, max_steps, tris, swap, table);
        __syncwarp();
    }
}

// Many objects, `size` a packet (RayPacket); those of more than kPacketHits crossings, or of an
// unfinished packet, go to deferred[0..*n_def), for k_containment.  With objects enough to fill
// the GPU it is the lanes that count: most rays of a sparse set visit a few dozen nodes and cross
// little, and a warp for each has one lane in ten busy.
__global__ void __launch_bounds__(32 * kContWarps, 6) k_containment_packets(
    const float* __restrict__ V, uint64_t nV, const uint32_t* __restrict__ I, const int32_t* __restrict__ first,
    uint64_t nObj, uint32_t size, const BNode* __restrict__ nodes, uint32_t max_steps, const float4* __restrict__ tris,
    int swap, PairTable table, uint32_t* __restrict__ deferred, unsigned int* __restrict__ n_def) {
    __shared__ RayPacket packets[kContWarps];
    RayPacket& sm = packets[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    for (uint64_t k = blockIdx.x * (uint64_t)kContWarps + (threadIdx.x >> 5); k * size < nObj;
         k += (uint64_t)gridDim.x * kContWarps) {
        const uint64_t o = k * size + lane;
        Ray r;
        const bool valid = (uint32_t)lane < size && o < nObj && containment_ray(V, nV, I, first, o, r);
        const unsigned int unfinished =
            packet_trace<2>(sm, r, valid, 0, nodes, min(max_steps, kPacketSteps), tris, 1e-4f);
        const int n = valid ? sm.n[lane] : 0;
        if (valid && (unfinished >> lane & 1u || n > kPacketHits)) {
            deferred[atomicAdd(n_def, 1u)] = (uint32_t)o;
        } else if (valid) {
            unsigned int targets = 0;
            for (int a = 0; a < n; ++a) {
                const uint32_t id = __float_as_uint(__ldg(&tris[3 * (size_t)sm.tri[a][lane] + 1].w));
                int before = 0, all = 0;
                for (int b = 0; b < n; ++b) {
                    const bool same = __float_as_uint(__ldg(&tris[3 * (size_t)sm.tri[b][lane] + 1].w)) == id;
                    all += same;
                    before += same && b < a;
                }
                if (before) continue;  // its first occurrence decides
                ++targets;
                if (all & 1) table_insert(table, containment_key(o, id, swap));
            }
            if (table.stats) {
                atomicAdd(&table.stats[4], 1ull);
                if (n) atomicAdd(&table.stats[5], (unsigned long long)n);
                if (targets) atomicAdd(&table.stats[6], (unsigned long long)targets);
            }
        }
        __syncwarp();
    }
}

}  // namespace

int recheck_join(int op, unsigned long long* out) { return recheck_op(op, out); }

void table_given(rs_pairset* ps) {
    ps->known_count = -1;
    ps->pristine = false;
    if (ps->over) ps->over_dirty = true;
}

PairTable table_view(rs_pairset* ps) {
    table_given(ps);
    PairTable t;
    t.slots = ps->slots;
    t.capacity = ps->capacity;
    t.pow2 = ps->pow2;
    t.max_probes = ps->max_probes;
    t.status = reinterpret_cast<unsigned int*>(ps->meta);
    t.count = ps->meta + 1;
    t.stats = ps->track ? ps->meta + 2 : nullptr;
    t.max_hits = ps->edge_max_hits;
    t.next_float = ps->edge_next_float;
    t.over = ps->over;
    t.over_mask = kOverSlots - 1;
    t.over_count = ps->meta + kOverWord;
    t.spill_at = std::max<unsigned long long>(1, ps->capacity / 4 * 3 + (ps->capacity % 4) * 3 / 4);
    return t;
}

}  // namespace rs

using namespace rs;

namespace rs {
// Launches one edge-ray direction without waiting for it (status lands in the table's meta word).
cudaError_t edge_jobs_async(EdgeJob* job, int n_jobs, rs_pairset* ps, cudaStream_t s);

// Blocks of k_edge_rays for at most n edges: one resident wave.
static unsigned packet_grid(uint64_t n) {
    static const int per_sm = [] {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_edge_rays, 32 * kPacketWarps, 0);
        return std::max(b, 1);
    }();
    return (unsigned)std::min<uint64_t>((n + kPacketWarps - 1) / kPacketWarps, (uint64_t)per_sm * sm_count());
}

// Every edge of a payload, in payload order (no broad phase), in chunks of 2^31 edges so
// that edge ids fit the 32-bit deferred list (a chunk's payload pointers are offset; the
// offsets still index the whole sources array).
static cudaError_t edge_all_async(const rs_bvh* target, EdgePayload p, uint64_t nE, int swap, rs_pairset* ps,
                                  cudaStream_t s) {
    constexpr uint64_t kChunk = 1ull << 31;
    const uint64_t cap = std::min(nE, kChunk);
    uint32_t* deferred = nullptr;
    unsigned int* n_def = nullptr;
    cudaError_t e = dmalloc((void**)&deferred, std::max<uint64_t>(cap, 1) * sizeof(uint32_t), s);
    if (e == cudaSuccess) e = dmalloc((void**)&n_def, 2 * sizeof(unsigned int), s);  // deferred, next packet
    const PairTable table = table_view(ps);
    const int ptok = prof_begin(P_EDGE_JOIN, s);
    for (uint64_t base = 0; base < nE && e == cudaSuccess; base += kChunk) {
        const uint64_t n = std::min(kChunk, nE - base);
        const EdgePayload q{p.starts + 3 * base, p.ends + 3 * base, p.offsets + base, p.counts + base, p.sources};
        e = cudaMemsetAsync(n_def, 0, 2 * sizeof(unsigned int), s);
        if (e != cudaSuccess) break;
        launch(k_edge_rays, packet_grid(n), 32 * kPacketWarps, 0, s, q, (const uint32_t*)nullptr, (const uint32_t*)nullptr,
               (const unsigned int*)nullptr, n,
               (const BNode*)target->nodes, max_steps(target), (const float4*)target->tris, swap, table, deferred,
               n_def, (const uint32_t*)nullptr, (const uint32_t*)nullptr, n_def + 1);
        launch(k_edge_long_warp, (unsigned)std::min<uint64_t>((n + kLongWarps - 1) / kLongWarps, 4ull * sm_count()),
               32 * kLongWarps, 0, s, q, (const uint32_t*)deferred, (const unsigned int*)n_def,
               (const BNode*)target->nodes, max_steps(target), (const float4*)target->tris, swap, table);
        e = cudaGetLastError();
    }
    prof_end(P_EDGE_JOIN, s, ptok);
    if (deferred) cudaFreeAsync(deferred, s);
    if (n_def) cudaFreeAsync(n_def, s);
    return e;
}

cudaError_t edge_join_async(const rs_bvh* target, const float* d_starts, const float* d_ends,
                            const int32_t* d_offsets, const int32_t* d_counts, const int32_t* d_sources, uint64_t nE,
                            int swap, rs_pairset* ps, cudaStream_t s, const EdgeCull& cull) {
    if (nE == 0 || target->n_tris == 0) return cudaSuccess;
    const EdgePayload p{d_starts, d_ends, d_offsets, d_counts, d_sources};
    if (!cull.cand || nE > 0xffffffffull) return edge_all_async(target, p, nE, swap, ps, s);
    EdgeJob job{};
    job.p = p;
    job.nE = nE;
    job.cull = cull.cand;
    job.n_cull = cull.n_obj;
    job.part = cull.part;
    job.pbox = cull.pbox;
    job.n_pbox = cull.n_pbox;
    job.entry = cull.part ? cull.entry : nullptr;
    job.xindex = cull.part ? cull.xindex : nullptr;
    job.sbox = cull.sbox;
    job.nodes = (const BNode*)target->nodes;
    job.max_steps = max_steps(target);
    job.tris = (const float4*)target->tris;
    job.swap = swap;
    return edge_jobs_async(&job, 1, ps, s);
}

// Live edges first, then rays for them only: the live checks of all jobs in one launch,
// the binning of their live edges by cell in two more, then each job's rays (the second
// job's on a side stream) and its deferred edges.  Each job's nE < 2^32 and its cull flags
// set.
cudaError_t edge_jobs_async(EdgeJob* job, int n_jobs, rs_pairset* ps, cudaStream_t s) {
    // One zeroed block: n_live[2], n_def[2], next packet[2], the cell counts of the binned jobs, then (slab
    // mode) each job's slab flags.
    uint32_t* zeroed = nullptr;
    EdgeJob jobs[2] = {};
    uint64_t blocks[2] = {0, 0}, total_e = 0;
    int n_bin = 0;
    // Slab mode when every job has a slab index (and partner lists): the live-edge check
    // visits only the slabs of objects with partners.
    bool slab = n_jobs > 0;
    for (int d = 0; d < n_jobs; ++d) {
        jobs[d] = job[d];
        if (jobs[d].nE <= kBinMaxEdges) ++n_bin;
        slab = slab && jobs[d].xindex && jobs[d].sbox && jobs[d].part;
    }
    auto a256 = [](size_t b) { return (b + 255) & ~size_t(255); };
    const size_t cbytes = a256((6 + (size_t)n_bin * kCells) * sizeof(uint32_t));
    size_t zbytes = cbytes;
    for (int d = 0; d < n_jobs && slab; ++d) {
        jobs[d].n_slab = (jobs[d].nE + kSlab - 1) / kSlab;
        zbytes += a256(std::max<uint64_t>(jobs[d].n_slab, 1));
    }
    // One allocation: the zeroed block, then each job's live, rank and (binned jobs) order
    // lists, each 256-byte aligned; one memset clears the zeroed block.
    size_t total = a256(zbytes);
    for (int d = 0; d < n_jobs; ++d) {
        const size_t bytes = a256(std::max<uint64_t>(jobs[d].nE, 1) * sizeof(uint32_t));
        const bool bin = jobs[d].nE <= kBinMaxEdges;
        total += ((bin ? 3 : 2) + (jobs[d].entry ? (bin ? 2 : 1) : 0)) * bytes;
    }
    cudaError_t e = dmalloc((void**)&zeroed, total, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(zeroed, 0, zbytes, s);
    uint32_t* next_cells = zeroed + 6;
    char* next_flags = reinterpret_cast<char*>(zeroed) + cbytes;
    char* next = reinterpret_cast<char*>(zeroed) + a256(zbytes);
    for (int d = 0; d < n_jobs && e == cudaSuccess; ++d) {
        EdgeJob& j = jobs[d];
        const size_t bytes = a256(std::max<uint64_t>(j.nE, 1) * sizeof(uint32_t));
        j.n_live = zeroed + d;
        j.n_def = zeroed + 2 + d;
        j.live = reinterpret_cast<uint32_t*>(next);
        j.rank = reinterpret_cast<uint32_t*>(next + bytes);
        next += 2 * bytes;
        if (j.nE <= kBinMaxEdges) {
            j.order = reinterpret_cast<uint32_t*>(next);
            next += bytes;
            j.cells = next_cells;
            next_cells += kCells;
        }
        if (j.entry) {
            j.live_entry = reinterpret_cast<uint32_t*>(next);
            next += bytes;
            if (j.order) {
                j.order_entry = reinterpret_cast<uint32_t*>(next);
                next += bytes;
            }
        }
        if (slab) {
            j.covered = reinterpret_cast<uint8_t*>(next_flags);
            next_flags += a256(std::max<uint64_t>(j.n_slab, 1));
        }
        blocks[d] = (j.nE + 256 * kLiveEdges - 1) / (256 * kLiveEdges);
        total_e += j.nE;
    }
    if (e == cudaSuccess && total_e) {
        const int ptok = prof_begin(P_EDGE_JOIN, s);
        if (slab) {
            uint64_t mb[2] = {0, 0};
            for (int d = 0; d < n_jobs; ++d) mb[d] = std::max<uint64_t>((jobs[d].n_cull + kMarkWarps - 1) / kMarkWarps, 1);
            launch(k_slab_mark, (unsigned)(mb[0] + mb[1]), 32 * kMarkWarps, 0, s, jobs[0], jobs[1], (unsigned)mb[0]);
            launch(k_edge_live_slab, (unsigned)(jobs[0].n_slab + jobs[1].n_slab), (unsigned)kSlab, 0, s, jobs[0],
                   jobs[1], (unsigned)jobs[0].n_slab);
        } else {
            launch(k_edge_live, (unsigned)(blocks[0] + blocks[1]), 256, 0, s, jobs[0], jobs[1], (unsigned)blocks[0]);
        }
        if (n_bin) {
            launch(k_cell_scan, 2, 1024, 0, s, jobs[0].cells, n_jobs > 1 ? jobs[1].cells : (uint32_t*)nullptr,
                   (const unsigned int*)jobs[0].n_live,
                   (const unsigned int*)(n_jobs > 1 ? jobs[1].n_live : jobs[0].n_live));
            const unsigned ob0 = (unsigned)std::min<uint64_t>(std::max<uint64_t>(blocks[0], 1), 4ull * sm_count());
            const unsigned ob1 = (unsigned)std::min<uint64_t>(blocks[1], 4ull * sm_count());
            launch(k_edge_order, ob0 + ob1, 256, 0, s, jobs[0], jobs[1], ob0, ob1);
        }
        // The rays of the second job on a side stream, concurrent with the first's: each
        // list's rays are latency-bound chains when the lists are short, and a full list
        // keeps the GPU busy either way.
        const PairTable table = table_view(ps);
        cudaStream_t side = nullptr;
        cudaEvent_t fork = nullptr, joined = nullptr;
        std::unique_lock<std::mutex> side_lock;
        if (n_jobs == 2 && ray_side_stream(&side, &fork, &joined, &side_lock) &&
            (cudaEventRecord(fork, s) != cudaSuccess || cudaStreamWaitEvent(side, fork, 0) != cudaSuccess)) {
            cudaGetLastError();
            side = nullptr;  // both on s
        }
        for (int d = 0; d < n_jobs; ++d) {
            const EdgeJob& j = jobs[d];
            cudaStream_t st = d == 1 && side ? side : s;
            launch(k_edge_rays, packet_grid(j.nE), 32 * kPacketWarps, 0, st, j.p, (const uint32_t*)j.order,
                   (const uint32_t*)j.live, (const unsigned int*)j.n_live, j.nE, j.nodes, j.max_steps, j.tris, j.swap,
                   table, j.rank, j.n_def, (const uint32_t*)j.order_entry, (const uint32_t*)j.live_entry,
                   zeroed + 4 + d);
            launch(k_edge_long_warp,
                   (unsigned)std::min<uint64_t>((j.nE + kLongWarps - 1) / kLongWarps, 4ull * sm_count()),
                   32 * kLongWarps, 0, st, j.p, (const uint32_t*)j.rank, (const unsigned int*)j.n_def, j.nodes,
                   j.max_steps, j.tris, j.swap, table);
        }
        if (side) {
            e = cudaEventRecord(joined, side);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(s, joined, 0);
            if (e != cudaSuccess) cudaStreamSynchronize(side);  // the lists are freed on s below
        }
        prof_end(P_EDGE_JOIN, s, ptok);
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    if (zeroed) cudaFreeAsync(zeroed, s);
    return e;
}

// Both edge directions of a join with both broad-phase flag sets: A's edges against B's
// BVH (swap 0) and B's edges against A's BVH (swap 1), rays of both in flight together.
cudaError_t edge_join_pair_async(const rs_bvh* A, const float* startsA, const float* endsA, const int32_t* offsetsA,
                                 const int32_t* countsA, const int32_t* sourcesA, uint64_t nEA, const EdgeCull& cullA,
                                 const rs_bvh* B, const float* startsB, const float* endsB, const int32_t* offsetsB,
                                 const int32_t* countsB, const int32_t* sourcesB, uint64_t nEB, const EdgeCull& cullB,
                                 rs_pairset* ps, cudaStream_t s) {
    EdgeJob job[2] = {};
    int n = 0;
    auto add = [&](const rs_bvh* target, EdgePayload p, uint64_t nE, const EdgeCull& c, int swap) {
        EdgeJob& j = job[n++];
        j.p = p;
        j.nE = nE;
        j.cull = c.cand;
        j.n_cull = c.n_obj;
        j.part = c.part;
        j.pbox = c.pbox;
        j.n_pbox = c.n_pbox;
        j.entry = c.part ? c.entry : nullptr;
        j.xindex = c.part ? c.xindex : nullptr;
        j.sbox = c.sbox;
        j.nodes = (const BNode*)target->nodes;
        j.max_steps = max_steps(target);
        j.tris = (const float4*)target->tris;
        j.swap = swap;
    };
    if (nEA && B->n_tris) add(B, EdgePayload{startsA, endsA, offsetsA, countsA, sourcesA}, nEA, cullA, 0);
    if (nEB && A->n_tris) add(A, EdgePayload{startsB, endsB, offsetsB, countsB, sourcesB}, nEB, cullB, 1);
    return n ? edge_jobs_async(job, n, ps, s) : cudaSuccess;
}

// Broad phase of both directions in one launch: set d's objects (A for d = 0, B for d = 1)
// are queried against the other set's BVH when cand[d] is given (either null: that
// direction is skipped), in partner mode when part[d] is given too.  Object boxes come from
// the build (k_morton) when they cover the set, else from its leaf triangles into
// temporaries.  With boxes_out, both sets' boxes are made and returned (the partner filter
// of the edge rays reads them) and the temporaries go to tmps_out, for the caller to free
// after those rays; otherwise they are freed here.
cudaError_t cull_impl(const rs_bvh* A, const rs_bvh* B, uint8_t* candA, uint8_t* candB, int32_t* partA,
                      int32_t* partB, uint32_t* entryA, uint32_t* entryB, const int** boxes_out, int** tmps_out,
                      cudaStream_t s) {
    const rs_bvh* src[2] = {A, B};
    const rs_bvh* other[2] = {B, A};
    uint8_t* cand[2] = {candA, candB};
    int32_t* part[2] = {partA, partB};
    uint32_t* entry[2] = {entryA, entryB};
    int* tmp[2] = {nullptr, nullptr};
    const int* boxes[2] = {nullptr, nullptr};
    CullJob job[2] = {};
    unsigned int blocks[2] = {0, 0};
    cudaError_t e = cudaSuccess;
    for (int d = 0; d < 2 && e == cudaSuccess; ++d) {
        const rs_bvh* h = src[d];
        if ((!cand[d] && !boxes_out) || h->n_obj == 0) continue;
        const int* box = h->obox;
        if (!box || h->n_obj > h->obox_cap) {
            e = dmalloc((void**)&tmp[d], 6 * h->n_obj * sizeof(int), s);
            if (e != cudaSuccess) break;
            launch(k_obj_box_init, (unsigned)((6 * h->n_obj + 255) / 256), 256, 0, s, tmp[d], h->n_obj);
            launch(k_obj_boxes, (unsigned)((h->n_tris + 255) / 256), 256, 0, s, (const float4*)h->tris, h->n_tris,
                   tmp[d], h->n_obj);
            box = tmp[d];
        }
        boxes[d] = box;
    }
    // Directions with partner lists are queried in packets, the others flagged object by object.
    uint64_t n_query = 0;
    for (int d = 0; d < 2 && e == cudaSuccess; ++d) {
        const rs_bvh* h = src[d];
        if (!cand[d] || h->n_obj == 0) continue;
        job[d] = CullJob{boxes[d], h->n_obj, (const BNode*)other[d]->nodes, max_steps(other[d]),
                         (const float4*)other[d]->tris, cand[d], part[d], part[d] ? entry[d] : nullptr, nullptr, 0,
                         nullptr};
        if (part[d]) n_query += h->n_obj;
        else blocks[d] = (unsigned int)((h->n_obj + kT - 1) / kT);
    }
    if (e == cudaSuccess && blocks[0] + blocks[1] > 0)
        launch(k_cull_flag, blocks[0] + blocks[1], kT, 0, s, job[0], job[1], blocks[0]);
    uint32_t* most = nullptr;
    if (e == cudaSuccess && n_query > 0) {
        // The boxes' lists pay where walks are long -- objects of many triangles -- and while
        // all pairs of boxes take little (44 us for 2 x 9 M tests, 330 at the limit of 2 x 67 M).
        // 3,001 + 3,001 objects of 5,500 triangles on average: 1,910 us of walks without them, 590
        // with them.  Objects of a few hundred triangles are walked in less time than the tests
        // take (10k + 10k of 320: 176 us).
        const bool long_walks = boxes[0] && boxes[1] && A->n_obj * B->n_obj <= (1ull << 26) &&
                                A->n_tris + B->n_tris >= 1024 * (A->n_obj + B->n_obj);
        const bool listed[2] = {long_walks && job[0].part && !B->unboxed, long_walks && job[1].part && !A->unboxed};
        if (listed[0] || listed[1]) e = dmalloc((void**)&most, n_query * sizeof(uint32_t), s);
        if (most && e == cudaSuccess) {
            uint32_t* next = most;
            unsigned bb[2] = {0, 0};
            for (int d = 0; d < 2; ++d) {
                if (!listed[d]) continue;
                job[d].obox = boxes[1 - d];
                job[d].n_other = other[d]->n_obj;
                job[d].most = next;
                next += job[d].n_obj;
                bb[d] = (unsigned)((job[d].n_obj + 7) / 8);
            }
            launch(k_box_pairs, bb[0] + bb[1], 256, 0, s, job[0], job[1], bb[0]);
        }
    }
    if (e == cudaSuccess && n_query > 0) {
        const uint64_t warps = (uint64_t)kCullResident * kCullWarps * sm_count();
        // A long walk wants all lanes for itself.
        const uint32_t size = most ? 1u : (uint32_t)std::min<uint64_t>((n_query + warps - 1) / warps, 32);
        auto packets_of = [&](int d) { return job[d].part ? (unsigned)((job[d].n_obj + size - 1) / size) : 0u; };
        const unsigned p0 = packets_of(0), all = p0 + packets_of(1);
        launch(k_cull_query, std::min((all + kCullWarps - 1) / kCullWarps, (unsigned)(kCullResident * sm_count())),
               32 * kCullWarps, 0, s, job[0], job[1], p0, all, size);
    }
    if (most) cudaFreeAsync(most, s);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (boxes_out && e == cudaSuccess) {
        boxes_out[0] = boxes[0];
        boxes_out[1] = boxes[1];
        tmps_out[0] = tmp[0];
        tmps_out[1] = tmp[1];
    } else {
        for (int* p : tmp)
            if (p) cudaFreeAsync(p, s);
    }
    return e;
}

// Queues the widening of both sets' object boxes (cull_impl's boxes_out) into out: two
// float4 per object, A's then B's.
cudaError_t wide_boxes_async(const int* boxA, uint64_t nA, const int* boxB, uint64_t nB, float4* out, cudaStream_t s) {
    launch(k_wide_boxes, (unsigned)((nA + nB + 255) / 256), 256, 0, s, boxA, nA, boxB, nB, out);
    return cudaGetLastError();
}

// Broad-phase flags of A's objects against B's BVH into candA and of B's objects against
// A's BVH into candB (either null: that direction is skipped), both in one launch.
cudaError_t cull_pair_async(const rs_bvh* A, const rs_bvh* B, uint8_t* candA, uint8_t* candB, cudaStream_t s) {
    return cull_impl(A, B, candA, candB, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, s);
}

// Broad-phase flags of `src`'s objects against `other`'s BVH.
cudaError_t cull_async(const rs_bvh* src, const rs_bvh* other, uint8_t* cand, cudaStream_t s) {
    return cull_pair_async(src, other, cand, nullptr, s);
}

// The distinct-key count read with the status is kept for rs_pairset_finalize/info.
int table_status(rs_pairset* ps, cudaStream_t s, cudaError_t e) {
    constexpr uint32_t kHard = ST_TABLE_FULL | ST_STACK_OVERFLOW | ST_ITER_LIMIT | ST_TARGET_OVERFLOW;
    for (int round = 0;; ++round) {
        unsigned long long m[kOverWord + 1] = {};
        if (e == cudaSuccess) e = cudaMemcpyAsync(m, ps->meta, sizeof(m), cudaMemcpyDeviceToHost, s);
        cudaError_t e2 = cudaStreamSynchronize(s);
        prof_collect();
        if (e == cudaSuccess) e = e2;
        if (e != cudaSuccess) return to_status(e);
        const uint32_t bits = (uint32_t)m[0];
        if ((bits & ST_SPILLED) && !(bits & kHard) && round < 4) {
            e = table_regrow(ps, m[1], m[kOverWord], s);
            continue;
        }
        // No spill: nothing went to the overflow table (a key goes there only after
        // ST_SPILLED is raised).  Otherwise the result is an error: empty it.
        if (!(bits & ST_SPILLED)) ps->over_dirty = false;
        else if ((e = over_clear(ps, s)) == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return to_status(e);
        const int st = status_from_bits(bits);
        ps->known_count = st == RS_OK ? (long long)m[1] : -1;
        return st;
    }
}
}  // namespace rs

extern "C" int rs_edge_index(const float* d_starts, const float* d_ends, const int32_t* d_sources, uint64_t nE,
                             uint64_t nS, int64_t* d_index, int* h_ordered, void* stream) {
    if (!d_index || (nE && (!d_starts || !d_ends)) || (nS && !d_sources)) return RS_ERR_INVALID;
    const void* q[4] = {d_starts, d_ends, d_sources, d_index};
    for (const void*& x : q)
        if (rs_kernel_pointer(x, &x) != RS_OK) return RS_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    int* word = nullptr;
    cudaError_t e = dmalloc((void**)&word, 2 * sizeof(int), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(word, 0, sizeof(int), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(word + 1, 0xff, sizeof(int), s);  // -1
    long long* index = reinterpret_cast<long long*>(const_cast<void*>(q[3]));
    if (e == cudaSuccess) {
        const EdgePayload p{static_cast<const float*>(q[0]), static_cast<const float*>(q[1]), nullptr, nullptr,
                            static_cast<const int32_t*>(q[2])};
        const uint64_t n = std::max<uint64_t>(std::max(nE, nS), 1);
        launch(k_edge_index, (unsigned)std::min<uint64_t>((n + 255) / 256, 4ull * sm_count()), 256, 0, s, p, nE, nS,
               index, word);
        launch(k_edge_index_head, 1, 1, 0, s, index, (const int*)word, nE);
        e = cudaGetLastError();
    }
    long long head = 0;
    if (e == cudaSuccess && h_ordered) {
        e = cudaMemcpyAsync(&head, index, sizeof(head), cudaMemcpyDefault, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e == cudaSuccess) *h_ordered = head == 1 ? 1 : 0;
    }
    if (word) cudaFreeAsync(word, s);
    return to_status(e);
}

extern "C" int rs_edge_join(const rs_bvh* target, const float* d_starts, const float* d_ends,
                            const int32_t* d_offsets, const int32_t* d_counts, const int32_t* d_sources,
                            uint64_t nE, int swap, rs_pairset* ps, void* stream) {
    if (!target || !ps || (nE && (!d_starts || !d_ends || !d_offsets || !d_counts || !d_sources)))
        return RS_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    int st = bvh_use(target, s);
    if (st == RS_OK) st = to_status(ps_use(ps, s));
    if (st != RS_OK) return st;
    cudaError_t e = edge_join_async(target, d_starts, d_ends, d_offsets, d_counts, d_sources, nE, swap, ps, s,
                                    EdgeCull{});
    return table_status(ps, s, e);
}

extern "C" int rs_triangle_join(const rs_bvh* target, const float* d_vertices, uint64_t nV, const uint32_t* d_indices,
                                uint64_t nF, const int32_t* d_tri2obj, int swap, rs_pairset* ps, void* stream) {
    if (!target || !ps || (nF && (!d_vertices || !d_indices || !d_tri2obj))) return RS_ERR_INVALID;
    const uint64_t m = 3 * nF;
    if (m == 0 || target->n_tris == 0) return RS_OK;
    cudaStream_t s = (cudaStream_t)stream;
    int st = bvh_use(target, s);
    if (st == RS_OK) st = to_status(ps_use(ps, s));
    if (st != RS_OK) return st;
    // bad flag and deferred count in one zeroed pair; records as 32-bit ids when they fit
    // (else every record runs the long path in the first kernel).
    unsigned int* flags = nullptr;
    uint32_t* deferred = nullptr;
    unsigned int hbad = 0;
    cudaError_t e = dmalloc((void**)&flags, 2 * sizeof(unsigned int), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(flags, 0, 2 * sizeof(unsigned int), s);
    if (e == cudaSuccess && m <= 0xffffffffull) e = dmalloc((void**)&deferred, m * sizeof(uint32_t), s);
    if (e == cudaSuccess) {
        const PairTable table = table_view(ps);
        const int ptok = prof_begin(P_EDGE_JOIN, s);
        launch(k_tri_edge_join, (unsigned)((m + kT - 1) / kT), kT, 0, s, d_vertices, nV, d_indices, d_tri2obj, m,
               (const BNode*)target->nodes, max_steps(target), (const float4*)target->tris, swap, table, flags,
               deferred, flags + 1);
        if (deferred)
            launch(k_tri_edge_long, (unsigned)std::min<uint64_t>((m + kT - 1) / kT, 2ull * sm_count()), kT, 0, s,
                   d_vertices, d_indices, d_tri2obj, (const uint32_t*)deferred, (const unsigned int*)(flags + 1),
                   (const BNode*)target->nodes, max_steps(target), (const float4*)target->tris, swap, table);
        prof_end(P_EDGE_JOIN, s, ptok);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&hbad, flags, sizeof(unsigned int), cudaMemcpyDeviceToHost, s);
    if (flags) cudaFreeAsync(flags, s);
    if (deferred) cudaFreeAsync(deferred, s);
    const int r = table_status(ps, s, e);
    if (r == RS_OK && hbad) return RS_ERR_INVALID;
    return r;
}

namespace rs {
// Queues the containment rays of source objects 0..nObj-1 (trk nullable).
static cudaError_t containment_async(const rs_bvh* target, const float* V, uint64_t nV, const uint32_t* I, uint64_t nF,
                              const int32_t* t2o, uint64_t nObj, int swap, rs_pairset* ps, const Tracking* trk,
                              cudaStream_t s) {
    if (nObj == 0 || nF == 0 || target->n_tris == 0) return cudaSuccess;
    int32_t* first = nullptr;  // first triangles, deferred objects, those the packets left, their number
    cudaError_t e = dmalloc((void**)&first, (3 * nObj + 1) * sizeof(int32_t), s);
    if (e != cudaSuccess) return e;
    uint32_t *deferred = reinterpret_cast<uint32_t*>(first + nObj), *left = deferred + nObj;
    unsigned int* n_left = left + nObj;
    launch(k_first_tri_init, (unsigned)((nObj + 255) / 256), 256, 0, s, first, nObj, n_left);
    launch(k_first_tri, (unsigned)((nF + 256 * kFirstPer - 1) / (256 * kFirstPer)), 256, 0, s, t2o, nF, first, nObj);
    const int ptok = prof_begin(P_CONTAINMENT, s);
    if (trk) {
        launch(k_containment_tracked, (unsigned)((nObj + kT - 1) / kT), kT, 0, s, V, nV, I, (const int32_t*)first, nObj,
               (const BNode*)target->nodes, max_steps(target), (const float4*)target->tris, swap, table_view(ps), *trk);
    } else {
        const PairTable table = table_view(ps);
        const unsigned grid = (unsigned)std::min<uint64_t>((nObj + kContWarps - 1) / kContWarps, 16ull * sm_count());
        const BNode* nodes = target->nodes;
        const float4* tris = target->tris;
        const uint32_t* list = nullptr;  // all objects
        if (nObj > kContPackets) {
            const uint64_t warps = 6ull * kContWarps * sm_count();  // a resident wave
            const uint32_t size = (uint32_t)std::min<uint64_t>((nObj + warps - 1) / warps, 32);
            launch(k_containment_packets, 6u * sm_count(), 32 * kContWarps, 0, s, V, nV, I, (const int32_t*)first, nObj,
                   size, nodes, max_steps(target), tris, swap, table, left, n_left);
            list = left;
        }
        launch(k_containment, grid, 32 * kContWarps, 0, s, V, nV, I, (const int32_t*)first, nObj, nodes,
               max_steps(target), tris, swap, table, list, (const unsigned int*)n_left, deferred);
    }
    prof_end(P_CONTAINMENT, s, ptok);
    e = cudaGetLastError();
    cudaFreeAsync(first, s);
    return e;
}

// Of every object of a built set.
cudaError_t containment_async(const rs_bvh* target, const rs_bvh* src, int swap, rs_pairset* ps, cudaStream_t s) {
    return containment_async(target, src->V, src->nV, src->I, src->nF, src->t2o, src->n_obj, swap, ps, nullptr, s);
}
}  // namespace rs

static int containment_impl(const rs_bvh* target, const float* d_src_vertices, uint64_t src_nV,
                            const uint32_t* d_src_indices, uint64_t src_nF, const int32_t* d_src_tri2obj, int swap,
                            rs_pairset* ps, const Tracking* trk, uint64_t trk_capacity, cudaStream_t s) {
    if (!target || !ps || (src_nF && (!d_src_vertices || !d_src_indices || !d_src_tri2obj))) return RS_ERR_INVALID;
    if (src_nF == 0 || target->n_tris == 0) return RS_OK;
    int st = bvh_use(target, s);
    if (st == RS_OK) st = to_status(ps_use(ps, s));
    if (st != RS_OK) return st;
    int* dmx = nullptr;
    int hmx = -1;
    cudaError_t e = dmalloc((void**)&dmx, sizeof(int), s);
    if (e == cudaSuccess) {
        cudaMemsetAsync(dmx, 0xff, sizeof(int), s);
        launch(k_max_obj, (unsigned)std::min<uint64_t>((src_nF + 1023) / 1024, 8ull * sm_count()), 256, 0, s,
               d_src_tri2obj, src_nF, dmx);
        e = cudaMemcpyAsync(&hmx, dmx, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    if (dmx) cudaFreeAsync(dmx, s);
    // Objects 0..max id (the reference sizes its launch by the number of distinct ids,
    // which is the same for the contiguous ids preprocess_dataset writes).
    const uint64_t nObj = hmx >= 0 ? (uint64_t)hmx + 1 : 0;
    if (trk && nObj > trk_capacity) return RS_ERR_OUTPUT_OVERFLOW;
    if (e == cudaSuccess)
        e = containment_async(target, d_src_vertices, src_nV, d_src_indices, src_nF, d_src_tri2obj, nObj, swap, ps, trk,
                              s);
    return table_status(ps, s, e);
}

extern "C" int rs_containment(const rs_bvh* target, const float* d_src_vertices, uint64_t src_nV,
                              const uint32_t* d_src_indices, uint64_t src_nF, const int32_t* d_src_tri2obj,
                              int swap, rs_pairset* ps, void* stream) {
    return containment_impl(target, d_src_vertices, src_nV, d_src_indices, src_nF, d_src_tri2obj, swap, ps, nullptr,
                            0, (cudaStream_t)stream);
}

extern "C" int rs_containment_tracked(const rs_bvh* target, const float* d_src_vertices, uint64_t src_nV,
                                      const uint32_t* d_src_indices, uint64_t src_nF, const int32_t* d_src_tri2obj,
                                      int swap, rs_pairset* ps, int max_targets, int32_t* d_target_ids,
                                      uint32_t* d_target_hits, uint32_t* d_candidate_counts, uint64_t capacity,
                                      void* stream) {
    if (max_targets <= 0 || !d_target_ids || !d_target_hits || !d_candidate_counts) return RS_ERR_INVALID;
    const Tracking trk{max_targets, d_target_ids, d_target_hits, d_candidate_counts};
    return containment_impl(target, d_src_vertices, src_nV, d_src_indices, src_nF, d_src_tri2obj, swap, ps, &trk,
                            capacity, (cudaStream_t)stream);
}
