// rs_query_core.cuh -- per-ray bodies shared by the single-query kernels (rs_pim.cu,
// rs_join.cu) and the batched persistent kernel (rs_batch.cu).
#pragma once
#include <climits>

#include "rs_device.cuh"
#include "rs_engine.h"

namespace rs {
namespace {

constexpr int kHits = 8;
constexpr float kEps = 1e-6f;
constexpr float kTmax = 1e16f;
constexpr int kFallbackIters = 1 << 16;

__device__ __forceinline__ bool hit_less(float t0, uint32_t i0, float t1, uint32_t i1) {
    return t0 < t1 || (t0 == t1 && i0 < i1);
}

// Iteration cap of the parity loop (raytracing.cu:26).
constexpr uint32_t kPimMaxIters = 10000;

// Advance rule of raytracing.cu:23-60 on hits sorted by (t, id): a hit counts when
// t >= threshold; the next threshold is t + 1e-6.  When t + 1e-6 rounds back to t
// (t >= 32) the reference's next trace starts at t and finds that hit again on every
// remaining iteration, so the count ends at the 10000-iteration cap; the count is
// capped there in any case.
struct Chain {
    float thr = kEps;
    uint32_t count = 0;
    int32_t first_obj = -1;
    __device__ __forceinline__ void step(float t, int32_t obj) {
        if (count < kPimMaxIters && t >= thr && t < kTmax) {
            if (count == 0) first_obj = obj;
            ++count;
            const float nt = __fadd_rn(t, kEps);
            if (!(nt > t)) count = kPimMaxIters;
            thr = nt;
        }
    }
};

// Hit sequence of the edge loops (mesh_overlap_edges.cu:106-178, mesh_intersection.cu:16-91,
// mesh_overlap.cu:13-70): repeated closest-hit traces over [t_min, len + 1e-6] with t_min
// starting at 1e-6 and moving to t + 1e-6 after each hit (t + 2e-4 when that does not
// advance), at most max_hits traces.  On hits sorted by (t, id) that is a greedy walk:
// a hit is taken when t >= t_min.  When neither step advances, every later trace finds the
// same hit again, which adds no pair, so the walk stops.  next_float selects the strict
// containment join's edge loop (mesh_containment.cu:99-170): t_min moves to the next float
// after t, so every distinct distance is taken once.
struct EdgeWalk {
    float thr = kEps;
    int n = 0;
    bool done = false;
    __device__ __forceinline__ bool take(float t, int max_hits, int next_float) {
        if (done || !(t >= thr)) return false;
        if (++n >= max_hits) done = true;
        float nt;
        if (next_float) {
            nt = nextafterf(t, INFINITY);
        } else {
            nt = __fadd_rn(t, kEps);
            if (!(nt > t)) nt = __fadd_rn(t, 2e-4f);
            if (!(nt > t)) done = true;
        }
        thr = nt;
        return true;
    }
};

// Up to kHits crossings in registers: predicated append, sorting network at the end.
struct HitList {
    float t[kHits];
    uint32_t id[kHits];
    int32_t obj[kHits];
    int n = 0;
    bool ovf = false;
    __device__ __forceinline__ void add(float tt, uint32_t ii, int32_t oo) {
        if (n >= kHits) {
            ovf = true;
            return;
        }
#pragma unroll
        for (int j = 0; j < kHits; ++j)
            if (j == n) {
                t[j] = tt;
                id[j] = ii;
                obj[j] = oo;
            }
        ++n;
    }
    // Odd-even transposition sort of all kHits slots (empty slots sort last).
    __device__ __forceinline__ void sort() {
#pragma unroll
        for (int j = 0; j < kHits; ++j)
            if (j >= n) {
                t[j] = INFINITY;
                id[j] = 0xffffffffu;
                obj[j] = -1;
            }
#pragma unroll
        for (int r = 0; r < kHits; ++r) {
#pragma unroll
            for (int j = r & 1; j + 1 < kHits; j += 2) {
                if (hit_less(t[j + 1], id[j + 1], t[j], id[j])) {
                    const float tt = t[j]; t[j] = t[j + 1]; t[j + 1] = tt;
                    const uint32_t ii = id[j]; id[j] = id[j + 1]; id[j + 1] = ii;
                    const int32_t oo = obj[j]; obj[j] = obj[j + 1]; obj[j + 1] = oo;
                }
            }
        }
    }
    // finish() of a list of at most two.
    __device__ __forceinline__ Chain finish2() const {
        Chain c;
        const bool swap = n == 2 && hit_less(t[1], id[1], t[0], id[0]);
        if (n >= 1) c.step(swap ? t[1] : t[0], swap ? obj[1] : obj[0]);
        if (n == 2) c.step(swap ? t[0] : t[1], swap ? obj[0] : obj[1]);
        return c;
    }
    __device__ __forceinline__ Chain finish() {
        sort();
        Chain c;
#pragma unroll
        for (int j = 0; j < kHits; ++j)
            if (j < n) c.step(t[j], obj[j]);
        return c;
    }
};


__device__ __forceinline__ void write_result(const Chain& ch, uint64_t i, int32_t* out_obj, uint8_t* out_in) {
    const bool inside = (ch.count & 1) != 0;
    if (out_obj) out_obj[i] = inside ? ch.first_obj : -1;
    if (out_in) out_in[i] = inside ? 1 : 0;
}

// Column grid of +e_AXIS rays: cells over the two other axes (u, v), each listing the
// triangles whose projected box touches it.  A list entry is 8 bytes: x = the leaf-ordered
// triangle, y = its box in the cell's own units, rounded outwards -- bits 0-5 and 6-11 the
// u range in 64ths of the cell, 12-17 and 18-23 the v range, 24-31 its highest point along
// the ray axis in 256ths of the mesh's extent.  The same monotone formulas give a query
// point's cell and units, so an entry whose ranges miss the point's units, or whose highest
// point lies below them, is a triangle that the ray cannot cross.
struct GridView {
    float u0, v0, su, sv, u1, v1;
    float w0, sw, w1;
    int gu, gv;
    const uint32_t* start;
    const uint2* list;
};

inline GridView grid_view(const rs_column_grid& c) {
    return GridView{c.u0, c.v0, c.su, c.sv, c.u1, c.v1, c.w0, c.sw, c.w1, c.gu, c.gv, c.start, c.list};
}

__device__ __forceinline__ float cell_units(float x, float x0, float s) { return __fmul_rn(__fsub_rn(x, x0), s); }

// Monotone cell index: identical for triangle boxes and query points.
__device__ __forceinline__ int cell_of(float x, float x0, float s, int g) {
    float f = floorf(cell_units(x, x0, s));
    f = fminf(fmaxf(f, 0.0f), (float)(g - 1));
    return (int)f;
}

// 64ths within cell c of a coordinate whose cell_units are f: monotone in f, clamped to the
// cell.  f - c is exact for f inside the cell.
__device__ __forceinline__ uint32_t unit_in_cell(float f, int c) {
    return (uint32_t)fminf(fmaxf(__fmul_rn(__fsub_rn(f, (float)c), 64.0f), 0.0f), 63.0f);
}

__device__ __forceinline__ uint32_t height_units(const GridView& g, float w) {
    return (uint32_t)fminf(fmaxf(cell_units(w, g.w0, g.sw), 0.0f), 255.0f);
}

__device__ __forceinline__ bool entry_may_hit(uint32_t e, uint32_t pu, uint32_t pv, uint32_t pw) {
    return (e & 63u) <= pu && ((e >> 6) & 63u) >= pu && ((e >> 12) & 63u) <= pv && ((e >> 18) & 63u) >= pv &&
           (e >> 24) >= pw;
}

// A point's cell list and its units (u | v << 8 | w << 16).
template <int AXIS>
__device__ __forceinline__ void grid_cell(const GridView& g, const float* p, uint32_t& begin, uint32_t& count,
                                          uint32_t& units) {
    constexpr int U = (AXIS + 1) % 3, V = (AXIS + 2) % 3;
    begin = 0;
    count = 0;
    units = 0;
    // A crossed triangle's box contains the point in u and v, and no triangle lies above w1.
    if (p[U] >= g.u0 && p[U] <= g.u1 && p[V] >= g.v0 && p[V] <= g.v1 && !(p[AXIS] > g.w1)) {
        const int cu = cell_of(p[U], g.u0, g.su, g.gu), cv = cell_of(p[V], g.v0, g.sv, g.gv);
        const int c = cv * g.gu + cu;
        begin = __ldg(&g.start[c]);
        count = __ldg(&g.start[c + 1]) - begin;
        units = unit_in_cell(cell_units(p[U], g.u0, g.su), cu) | unit_in_cell(cell_units(p[V], g.v0, g.sv), cv) << 8 |
                height_units(g, p[AXIS]) << 16;
    }
}

// One warp's shared memory for pim_grid_warp: crossing slots (kHits a point, or 32 * kHits of
// one point), the points, the work lists' owners and a ring of candidates to test.
struct GridWarpSlots {
    float t[kHits][32];
    uint32_t id[kHits][32];
    int32_t obj[kHits][32];
    int n[32];
    float p[3][32];
    uint4 rec[32];      // of the k-th point with candidates: list offset, units, lane
    uint2 ring[64];     // triangle, lane of its point
    // Points with candidates that wait for a full round (grid_points): coordinates, list
    // begin and length, units, number.
    float qp[3][64];
    uint32_t qb[64], qc[64], qu[64], qi[64];
};
constexpr int kDenseHits = 32 * kHits;
// Candidates a point from which a warp takes its points one at a time: the lists then fill
// whole rounds by themselves, and rays through that many boxes often cross more than kHits
// triangles.
constexpr uint32_t kDenseCandidates = 48;

// The advance rule on nh crossings that a warp holds, by repeated minima: the next counted
// crossing is the nearest at or beyond the threshold.  Distances are positive, so their bits
// order like them.  The same Chain in every lane.
__device__ __forceinline__ Chain dense_chain(const float* ht, const uint32_t* hid, const int32_t* hobj, int nh,
                                             int lane) {
    Chain ch;
    if (nh <= 32) {
        // Crossings that all lie a step or more apart are all counted, in whatever order they
        // were found, up to the first that a step does not move: almost every ray, and a third
        // of the instructions of the minima below.
        const bool mine = lane < nh;
        const float t = mine ? ht[lane] : INFINITY, nt = __fadd_rn(t, kEps);
        bool close = mine && !(t >= kEps && t < kTmax);
        for (int j = 0; j < nh; ++j) {
            const float o = __shfl_sync(0xffffffffu, t, j);
            close |= mine && j != lane && o >= t && o < nt;
        }
        if (!__any_sync(0xffffffffu, close)) {
            const uint32_t near = __reduce_min_sync(0xffffffffu, __float_as_uint(t));
            const unsigned int first = __ballot_sync(0xffffffffu, mine && __float_as_uint(t) == near);
            ch.count = __any_sync(0xffffffffu, mine && !(nt > t)) ? kPimMaxIters : (uint32_t)nh;
            if (first) ch.first_obj = hobj[__ffs(first) - 1];
            return ch;
        }
    }
    for (;;) {
        uint32_t best = 0xffffffffu;
        for (int h = lane; h < nh; h += 32) {
            const float t = ht[h];
            if (t >= ch.thr && t < kTmax) best = min(best, __float_as_uint(t));
        }
        best = __reduce_min_sync(0xffffffffu, best);
        if (best == 0xffffffffu) return ch;
        const float t = __uint_as_float(best);
        int32_t obj = -1;
        if (ch.count == 0) {  // the object of the smallest id at that distance
            uint32_t low = 0xffffffffu;
            for (int h = lane; h < nh; h += 32)
                if (ht[h] == t && hid[h] <= low) {
                    low = hid[h];
                    obj = hobj[h];
                }
            const uint32_t lowest = __reduce_min_sync(0xffffffffu, low);
            obj = __shfl_sync(0xffffffffu, obj, __ffs(__ballot_sync(0xffffffffu, low == lowest)) - 1);
        }
        ch.step(t, obj);
        if (ch.count == kPimMaxIters) return ch;
    }
}

// Warp-cooperative column-grid query of the warp's 32 points (all lanes call it; lanes
// without a point pass valid = false, lanes whose point was filtered out keep = false).
// Bound by instruction issue, so the work is cut rather than the bytes: of the 5 candidates
// that a point of the level-4 sphere finds in its cell, 1.5 pass the 8-byte entry's ranges,
// and only those are loaded and tested exactly.
//  * The cells' lists are flattened into one work list, 32 entries a round; the owner of an
//    entry follows from one OR-reduction of the round's list heads.  Entries that pass are
//    queued in a ring and tested 32 at a time, every lane with a triangle.  Crossings go to
//    the points' slots, and each lane walks its own in (t, id) order.
//  * A point with more than kHits crossings, and every point of a warp whose lists are long,
//    is taken by the whole warp: up to kDenseHits crossings, walked by repeated minima.
//    Beyond that overflow() takes the point.
// (b, cnt, units: the point's list and units, grid_cell; cnt 0 for a lane with nothing to test.)
template <int AXIS, class Ovf>
__device__ __forceinline__ void pim_grid_warp(const GridView& g, const float4* __restrict__ tris, const float* p,
                                              bool valid, uint32_t b, uint32_t cnt, uint32_t units, uint64_t i,
                                              int32_t* __restrict__ out_obj, uint8_t* __restrict__ out_in,
                                              GridWarpSlots& sl, Ovf&& overflow) {
    constexpr unsigned int kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned int below = (1u << lane) - 1u;
    const float dx = AXIS == 0 ? 1.0f : 0.0f, dy = AXIS == 1 ? 1.0f : 0.0f, dz = AXIS == 2 ? 1.0f : 0.0f;
    const unsigned int listed = __ballot_sync(kAll, cnt != 0);
    if (listed == 0) {
        if (valid) write_result(Chain{}, i, out_obj, out_in);
        return;
    }
    uint32_t inc = cnt;  // warp prefix sum of the candidate counts
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kAll, inc, o);
        if (lane >= o) inc += y;
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) sl.p[q][lane] = p[q];
    sl.n[lane] = 0;
    float* ht = &sl.t[0][0];
    uint32_t* hid = &sl.id[0][0];
    int32_t* hobj = &sl.obj[0][0];
    uint32_t tests = 0;
    // First all points at once (owner -1), unless their lists are long, then the points that
    // the whole warp takes, one by one.
    uint32_t total = __shfl_sync(kAll, inc, 31);
    uint32_t start = cnt ? inc - cnt : ~0u;  // where this lane's list starts in the work list
    unsigned int dense = 0;
    int owner = -1;
    if (cnt) sl.rec[__popc(listed & below)] = make_uint4(b - start, units, (uint32_t)lane, 0u);
    if (total >= 32u * kDenseCandidates) {
        dense = listed;
        if (valid && cnt == 0) write_result(Chain{}, i, out_obj, out_in);
        total = 0;
    }
    __syncwarp();
    for (;;) {
        uint32_t head = 0, queued = 0, owners = 0;
        for (uint32_t base = 0; base < total || queued; base += 32) {
            if (base < total) {
                const uint32_t j = base + lane;
                // Bit q of heads: a list starts at entry base + q.
                const unsigned int heads = __reduce_or_sync(kAll, start - base < 32u ? 1u << (start - base) : 0u);
                const uint4 rec = sl.rec[owners + __popc(heads & (below | 1u << lane)) - 1u];
                owners += __popc(heads);
                uint2 e = make_uint2(0u, 0u);
                bool pass = false;
                if (j < total) {
                    e = __ldg(&g.list[rec.x + j]);
                    pass = entry_may_hit(e.y, rec.y & 255u, (rec.y >> 8) & 255u, rec.y >> 16);
                }
                const unsigned int m = __ballot_sync(kAll, pass);
                if (pass) sl.ring[(head + queued + __popc(m & below)) & 63u] = make_uint2(e.x, rec.z);
                queued += __popc(m);
                __syncwarp();
                if (queued < 32u && base + 32u < total) continue;
            }
            // Exact test of up to 32 queued candidates.
            const uint32_t m = min(queued, 32u);
            if ((uint32_t)lane < m) {
                const uint2 e = sl.ring[(head + lane) & 63u];
                float a[3], bb[3], cc[3];
                uint32_t tid;
                int32_t obj;
                load_tri(tris, (int)e.x, a, bb, cc, tid, obj);
                const Ray r = make_ray(sl.p[0][e.y], sl.p[1][e.y], sl.p[2][e.y], dx, dy, dz, kEps, kTmax);
                float t;
                if (hit_triangle<AXIS>(r, a, bb, cc, t)) {
                    const int k = atomicAdd(&sl.n[e.y], 1);
                    if (k < (owner < 0 ? kHits : kDenseHits)) {
                        const int at = owner < 0 ? k * 32 + (int)e.y : k;
                        ht[at] = t;
                        hid[at] = tid;
                        hobj[at] = obj;
                    }
                }
            }
            tests += m;
            head += m;
            queued -= m;
            __syncwarp();
        }
        if (owner < 0) {
            const int nh = sl.n[lane];
            const int most = __reduce_max_sync(kAll, nh);
            if (total) {
                dense = __ballot_sync(kAll, nh > kHits);
                if (valid && nh <= kHits) {
                    HitList hl;
#pragma unroll
                    for (int q = 0; q < kHits; ++q)
                        if (q < nh) {
                            hl.t[q] = sl.t[q][lane];
                            hl.id[q] = sl.id[q][lane];
                            hl.obj[q] = sl.obj[q][lane];
                        }
                    hl.n = nh;
                    write_result(most <= 2 ? hl.finish2() : hl.finish(), i, out_obj, out_in);
                }
            }
        } else {
            const int nh = sl.n[owner];
            if (nh > kDenseHits) {
                if (lane == owner) overflow();
            } else {
                const Chain ch = dense_chain(ht, hid, hobj, nh, lane);
                if (lane == owner) write_result(ch, i, out_obj, out_in);
            }
        }
        if (dense == 0) break;
        owner = __ffs(dense) - 1;
        dense &= dense - 1;
        total = __shfl_sync(kAll, cnt, owner);
        start = lane == 0 ? 0u : ~0u;
        __syncwarp();  // the slots are read: free for the next point
        if (lane == owner) {
            sl.rec[0] = make_uint4(b, units, (uint32_t)lane, 0u);
            sl.n[lane] = 0;
        }
        __syncwarp();
    }
    add_tests(lane == 0 ? tests : 0u);
}

// Points first, first + stride, ... below end, one per lane and round (first: this lane's
// point; every lane of a warp runs the same rounds): load(i, p) reads a point, keep(p)
// filters it.  Points without candidates are answered at once; the others wait in shared
// memory until they fill a round of pim_grid_warp, which otherwise runs two thirds empty for
// points spread over a box around the mesh.
template <int AXIS, class Load, class Keep, class Ovf>
__device__ __forceinline__ void grid_points(const GridView& g, const float4* __restrict__ tris, uint64_t first,
                                            uint64_t end, uint64_t stride, int32_t* __restrict__ out_obj,
                                            uint8_t* __restrict__ out_in, GridWarpSlots& sl, Load&& load, Keep&& keep,
                                            Ovf&& overflow) {
    const int lane = threadIdx.x & 31;
    uint32_t head = 0, waiting = 0;
    float p[3] = {0.0f, 0.0f, 0.0f};
    uint64_t i = first;
    if (i < end) load(i, p);
    bool more = i - lane < end;  // warp-uniform: lane 0 has the least number of the round
    while (more || waiting) {
        if (more) {
            uint32_t b = 0, cnt = 0, units = 0;
            const bool valid = i < end;
            if (valid && keep(p)) grid_cell<AXIS>(g, p, b, cnt, units);
            if (valid && cnt == 0) write_result(Chain{}, i, out_obj, out_in);
            const unsigned int m = __ballot_sync(0xffffffffu, cnt != 0);
            if (cnt) {
                const uint32_t at = (head + waiting + __popc(m & ((1u << lane) - 1u))) & 63u;
#pragma unroll
                for (int q = 0; q < 3; ++q) sl.qp[q][at] = p[q];
                sl.qb[at] = b;
                sl.qc[at] = cnt;
                sl.qu[at] = units;
                sl.qi[at] = (uint32_t)i;
            }
            waiting += __popc(m);
            i += stride;
            more = i - lane < end;
            if (i < end) load(i, p);  // on its way while this round is tested
            __syncwarp();
            if (waiting < 32u && more) continue;
        }
        const uint32_t take = min(waiting, 32u), at = (head + lane) & 63u;
        const bool mine = (uint32_t)lane < take;
        float t[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) t[q] = mine ? sl.qp[q][at] : 0.0f;
        const uint32_t k = mine ? sl.qi[at] : 0u;
        pim_grid_warp<AXIS>(g, tris, t, mine, mine ? sl.qb[at] : 0u, mine ? sl.qc[at] : 0u, mine ? sl.qu[at] : 0u, k,
                            out_obj, out_in, sl, [&]() { overflow(k); });
        head += take;
        waiting -= take;
        __syncwarp();
    }
}

// One ray by one thread, for what pim_range_ray leaves over: up to kLongHits crossings from one
// traversal; beyond them each round re-traverses the BVH and takes the smallest (t, id) above
// the previous one, so the crossings are walked in the same order as the sorted list.
constexpr int kLongHits = 64;

// Entries that a warp's traversal keeps free of its stack when it pops many nodes at a time: one
// for each level of the tree that it then descends by one node at a time.  Popping what just fits
// fills the stack to its last entry, and the next node with two inner children breaks off.
constexpr int kStackRoom = 64;

template <int AXIS>
__device__ __forceinline__ void pim_fallback_ray(const BNode* __restrict__ nodes, uint32_t max_steps,
                                                 const float4* __restrict__ tris, const Ray& r,
                                                 unsigned int* __restrict__ status, int32_t* __restrict__ out_obj,
                                                 uint8_t* __restrict__ out_in, uint64_t i) {
    // One traversal into a local list of up to kLongHits crossings, insertion-sorted by
    // (t, id); only rays with more crossings walk them by re-traversal below.
    {
        float lt[kLongHits];
        uint32_t lid[kLongHits];
        int32_t lobj[kLongHits];
        int n = 0;
        bool more = false;
        const bool ok = traverse<AXIS, kStack>(nodes, max_steps, r, [&](int first, int c) {
            for (int k = first; k < first + c; ++k) {
                float a[3], b[3], cc[3];
                uint32_t tid;
                int32_t obj;
                load_tri(tris, k, a, b, cc, tid, obj);
                float t;
                if (!hit_triangle<AXIS>(r, a, b, cc, t)) continue;
                if (n == kLongHits) {
                    more = true;
                    continue;
                }
                int j = n++;
                while (j > 0 && hit_less(t, tid, lt[j - 1], lid[j - 1])) {
                    lt[j] = lt[j - 1];
                    lid[j] = lid[j - 1];
                    lobj[j] = lobj[j - 1];
                    --j;
                }
                lt[j] = t;
                lid[j] = tid;
                lobj[j] = obj;
            }
        });
        if (!ok) {
            atomicOr(status, ST_STACK_OVERFLOW);
            write_result(Chain{}, i, out_obj, out_in);
            return;
        }
        if (!more) {
            Chain ch;
            for (int j = 0; j < n; ++j) ch.step(lt[j], lobj[j]);
            write_result(ch, i, out_obj, out_in);
            return;
        }
    }
    Chain ch;
    float pt = -INFINITY;
    uint32_t pid = 0;
    bool have_prev = false;
    int it = 0;
    for (; it < kFallbackIters && ch.count < kPimMaxIters; ++it) {
        float bt = INFINITY;
        uint32_t bid = 0xffffffffu;
        int32_t bobj = -1;
        bool found = false;
        const bool ok = traverse<AXIS, kStack>(nodes, max_steps, r, [&](int first, int c) {
            for (int k = first; k < first + c; ++k) {
                float a[3], b[3], cc[3];
                uint32_t tid;
                int32_t obj;
                load_tri(tris, k, a, b, cc, tid, obj);
                float t;
                if (!hit_triangle<AXIS>(r, a, b, cc, t)) continue;
                if (have_prev && !hit_less(pt, pid, t, tid)) continue;
                if (!found || hit_less(t, tid, bt, bid)) {
                    found = true;
                    bt = t;
                    bid = tid;
                    bobj = obj;
                }
            }
        });
        if (!ok) {
            atomicOr(status, ST_STACK_OVERFLOW);
            break;
        }
        if (!found) break;
        ch.step(bt, bobj);
        pt = bt;
        pid = bid;
        have_prev = true;
    }
    if (it == kFallbackIters) atomicOr(status, ST_ITER_LIMIT);
    write_result(ch, i, out_obj, out_in);
}

// Rays of many crossings, one warp each: up to 32 nodes a step from a shared-memory stack, and all
// crossings in a list, in ranges of t: a full list keeps those up to its middle one, which becomes
// the range's end, and the traversal goes on with what is left of its stack; the next range
// begins above it.  Sorted by (t, id), a range's crossings are walked by the caller's rule.  Visits
// the nodes that one thread's traversal of the range would, so it finds the same crossings.
//
// Points: what a query leaves over.  A thread a ray found the crossings beyond its 64th by a
// traversal each: 20,000 points in 300 shells, up to 600 crossings, took 10.3 s (4.8 while such
// rays shared their warps with others), now 1.8 ms; 2 M oblique rays of up to 40 crossings 23.5 ms,
// now 12.5.  Oblique rays of 9 to 12 crossings are the ones that threads had suited better: 5 M of
// them 7.9 ms, now 8.9.
constexpr int kRangeHits = 512;
constexpr int kRangeStack = 320;
constexpr int kRangeWarps = 4;  // a block

struct RangeWarp {
    uint64_t key[kRangeHits];  // t, id: positive distances order like their bits
    int32_t obj[kRangeHits];
    int stack[kRangeStack];
};

// Ascending bitonic sort of the warp's first n crossings.
__device__ __forceinline__ void range_sort(RangeWarp& w, int n) {
    const int lane = threadIdx.x & 31;
    int m = 32;
    while (m < n) m <<= 1;
    for (int i = n + lane; i < m; i += 32) w.key[i] = ~0ull;
    __syncwarp();
    for (int k = 2; k <= m; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = lane; i < m; i += 32) {
                const int q = i ^ j;
                const uint64_t a = w.key[i], b = w.key[q];
                if (q > i && (a > b) == ((i & k) == 0)) {
                    const int32_t o = w.obj[i];
                    w.key[i] = b;
                    w.key[q] = a;
                    w.obj[i] = w.obj[q];
                    w.obj[q] = o;
                }
            }
            __syncwarp();
        }
}

__device__ __forceinline__ float range_t(const RangeWarp& w, int i) {
    return __uint_as_float((uint32_t)(w.key[i] >> 32));
}

// Every crossing of ray r with t in (above, r.tmax] into the warp's list, unsorted, nh of them; when
// they are more than it holds, those of a range that begins there, whose end becomes r.tmax.
// False when the stack, the steps or, at one distance, the list run out.
template <int AXIS>
__device__ __forceinline__ bool range_collect(RangeWarp& w, const BNode* __restrict__ nodes, uint32_t max_steps,
                                              const float4* __restrict__ tris, Ray& r, float above, int& nh,
                                              unsigned int& tests) {
    constexpr unsigned int kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned int below = (1u << lane) - 1u;
    if (lane == 0) w.stack[0] = 0;
    __syncwarp();
    int sp = 1;
    uint32_t visits = 0;
    nh = 0;
    while (sp > 0) {
        const int take = min(min(sp, 32), max(kRangeStack - kStackRoom - sp, 1));
        const int node = lane < take ? w.stack[sp - take + lane] : -1;
        __syncwarp();
        sp -= take;
        visits += (uint32_t)take;
        bool h[2] = {false, false};
        int leaf[2] = {0, 0}, cnt[2] = {0, 0};
        if (node >= 0) {
            const BNode bn = load_node(nodes, node);
            const float lo0[3] = {bn.a.x, bn.a.y, bn.a.z}, hi0[3] = {bn.a.w, bn.b.x, bn.b.y};
            const float lo1[3] = {bn.b.z, bn.b.w, bn.c.x}, hi1[3] = {bn.c.y, bn.c.z, bn.c.w};
            float en, ex;
            h[0] = slab<AXIS>(r, lo0, hi0, r.tmin, r.tmax, en, ex);
            h[1] = slab<AXIS>(r, lo1, hi1, r.tmin, r.tmax, en, ex);
            leaf[0] = bn.d.x;
            cnt[0] = bn.d.y;
            leaf[1] = bn.d.z;
            cnt[1] = bn.d.w;
        }
        const bool p0 = h[0] && cnt[0] == 0, p1 = h[1] && cnt[1] == 0;
        const unsigned int b0 = __ballot_sync(kAll, p0), b1 = __ballot_sync(kAll, p1);
        const int pushed = __popc(b0) + __popc(b1);
        if (visits > max_steps || sp + pushed > kRangeStack) return false;
        int pos = sp + __popc(b0 & below) + __popc(b1 & below);
        if (p0) w.stack[pos++] = leaf[0];
        if (p1) w.stack[pos] = leaf[1];
        sp += pushed;
        // Triangles of the leaves hit: the first child's, then the second's.
        const int n0 = h[0] ? cnt[0] : 0, n1 = h[1] ? cnt[1] : 0;
        tests += (unsigned int)(n0 + n1);
        const int rounds = __reduce_max_sync(kAll, n0 + n1);
        for (int k = 0; k < rounds; ++k) {
            bool hit = false;
            float t = 0.0f;
            uint32_t tid = 0;
            int32_t obj = 0;
            if (k < n0 + n1) {
                float a[3], b[3], c[3];
                load_tri(tris, k < n0 ? leaf[0] + k : leaf[1] + (k - n0), a, b, c, tid, obj);
                hit = hit_triangle<AXIS>(r, a, b, c, t) && t > above;
            }
            unsigned int m = __ballot_sync(kAll, hit);
            if (nh + __popc(m) > kRangeHits) {
                range_sort(w, nh);
                const float mid = range_t(w, nh / 2);
                int n = nh / 2 + 1;
                while (n < nh && range_t(w, n) == mid) ++n;
                __syncwarp();
                r.tmax = mid;
                nh = n;
                hit = hit && t <= mid;
                m = __ballot_sync(kAll, hit);
                if (nh + __popc(m) > kRangeHits) return false;  // hundreds at one distance
            }
            if (hit) {
                const int at = nh + __popc(m & below);
                w.key[at] = (uint64_t)__float_as_uint(t) << 32 | tid;
                w.obj[at] = obj;
            }
            nh += __popc(m);
        }
        __syncwarp();
    }
    return true;
}

// The range after the one that ends at r.tmax; false when that was the last.
__device__ __forceinline__ bool next_range(Ray& r, float tmax, float& above) {
    if (r.tmax == tmax) return false;
    above = r.tmax;
    r.tmin = fmaxf(r.tmin, above);
    r.tmax = tmax;
    return true;
}

template <int AXIS>
__device__ __forceinline__ void pim_range_ray(RangeWarp& w, const BNode* __restrict__ nodes, uint32_t max_steps,
                                              const float4* __restrict__ tris, Ray r, unsigned int* __restrict__ status,
                                              int32_t* __restrict__ out_obj, uint8_t* __restrict__ out_in, uint64_t i) {
    const int lane = threadIdx.x & 31;
    const Ray whole = r;
    float above = -INFINITY;
    Chain ch;
    int walked = 0, nh = 0;
    unsigned int tests = 0;
    bool ok;
    while ((ok = range_collect<AXIS>(w, nodes, max_steps, tris, r, above, nh, tests))) {
        range_sort(w, nh);
        for (int k = 0; k < nh && ch.count < kPimMaxIters; ++k) ch.step(range_t(w, k), w.obj[k]);
        walked += nh;
        __syncwarp();
        if (ch.count >= kPimMaxIters || !next_range(r, whole.tmax, above)) break;
        if (walked >= kFallbackIters) {
            if (lane == 0) atomicOr(status, ST_ITER_LIMIT);
            break;
        }
    }
    __syncwarp();
    if (lane != 0) return;
    if (ok) write_result(ch, i, out_obj, out_in);
    else pim_fallback_ray<AXIS>(nodes, max_steps, tris, whole, status, out_obj, out_in, i);
}

// ---------------------------------------------------------------------------
// Edge rays by one thread.  The per-triangle join's fast path traces an edge once with its
// stack and its crossings (up to kEdgeHits) in a column of shared memory; an edge with more
// crossings, or a traversal deeper than the fast stack, is deferred untouched to the long
// path.  Payload edges go in packets and ranges (edge_packet below, edge_ray_warp) and come
// to the long path for hundreds of crossings at one distance only.
// ---------------------------------------------------------------------------
constexpr int kEdgeHits = 4;

// One thread's shared-memory column: element k of an array at base[k * stride].
struct EdgeColumn {
    int* stack;
    float* t;
    uint32_t* id;
    int32_t* obj;
    int stride;
};

// Shared-memory block of the fast path for T threads and a STACK-entry stack.
template <int T, int STACK>
struct EdgeSmem {
    int stack[STACK][T];
    float t[kEdgeHits][T];
    uint32_t id[kEdgeHits][T];
    int32_t obj[kEdgeHits][T];
    __device__ __forceinline__ EdgeColumn column(int tid) {
        return EdgeColumn{&stack[0][tid], &t[0][tid], &id[0][tid], &obj[0][tid], T};
    }
};

// The segment's ray as distance3f / normalize3f of mesh_overlap_edges.cu:47-60 compute it,
// one rounded operation at a time; false for edges shorter than 1e-6 (never traced).
__device__ __forceinline__ bool segment_ray_of(float sx, float sy, float sz, float ex, float ey, float ez, Ray& r) {
    const float dx = __fsub_rn(ex, sx), dy = __fsub_rn(ey, sy), dz = __fsub_rn(ez, sz);
    const float len = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
    if (len < 1e-6f) return false;
    r = make_ray(sx, sy, sz, __fdiv_rn(dx, len), __fdiv_rn(dy, len), __fdiv_rn(dz, len), 1e-6f, __fadd_rn(len, 1e-6f));
    return true;
}

// (source, target) -- (target, source) when swap -- for every source object of the edge.
__device__ __forceinline__ void insert_sources(const PairTable& table, const int32_t* __restrict__ src, int nsrc,
                                               int32_t obj, int swap) {
    for (int q = 0; q < nsrc; ++q) {
        const uint32_t sobj = (uint32_t)src[q];
        const unsigned long long key = swap ? (((unsigned long long)(uint32_t)obj << 32) | sobj)
                                            : (((unsigned long long)sobj << 32) | (uint32_t)obj);
        table_insert(table, key);
    }
}

__device__ __forceinline__ void count_edge(const PairTable& table, int taken) {
    if (table.stats) {
        atomicAdd(&table.stats[2], 1ull);
        if (taken) atomicAdd(&table.stats[3], (unsigned long long)taken);
    }
}

// Edge ray of mesh_overlap_edges.cu:106-216, fast path: one traversal over
// t in [1e-6, len + 1e-6] with the stack and crossings in the thread's shared-memory
// column; the crossings, sorted by (t, triangle id), are walked with the table's hit rule
// (EdgeWalk) and every target object of a hit taken is paired with every source object.
// Returns false, having inserted nothing, when the edge has more than kEdgeHits crossings
// or the traversal ran out of stack or steps: the caller then defers it to segment_long.
template <int STACK>
__device__ __forceinline__ bool segment_fast(const EdgeColumn& col, const Ray& r, const int32_t* __restrict__ src,
                                             int nsrc, const BNode* __restrict__ nodes, uint32_t max_steps,
                                             const float4* __restrict__ tris, int swap, const PairTable& table) {
    const int S = col.stride;
    int n = 0;
    unsigned int tests = 0;
    const bool ok = traverse_with<-1, STACK>(col.stack, S, nodes, max_steps, r, [&](int first, int cnt) {
        tests += (unsigned int)cnt;
        for (int k = first; k < first + cnt; ++k) {
            float a[3], b[3], c[3];
            uint32_t tid;
            int32_t obj;
            load_tri(tris, k, a, b, c, tid, obj);
            float t;
            if (!hit_triangle<-1>(r, a, b, c, t)) continue;
            if (n < kEdgeHits) {
                // Insertion into the sorted column.
                int j = n;
                while (j > 0 && hit_less(t, tid, col.t[(j - 1) * S], col.id[(j - 1) * S])) {
                    col.t[j * S] = col.t[(j - 1) * S];
                    col.id[j * S] = col.id[(j - 1) * S];
                    col.obj[j * S] = col.obj[(j - 1) * S];
                    --j;
                }
                col.t[j * S] = t;
                col.id[j * S] = tid;
                col.obj[j * S] = obj;
            }
            ++n;
        }
    });
    add_tests(tests);
    if (!ok || n > kEdgeHits) return false;
    EdgeWalk w;
    int32_t last = INT_MIN;
    for (int j = 0; j < n; ++j) {
        if (!w.take(col.t[j * S], table.max_hits, table.next_float)) continue;
        const int32_t obj = col.obj[j * S];
        if (obj == last) continue;
        last = obj;
        insert_sources(table, src, nsrc, obj, swap);
    }
    count_edge(table, w.n);
    return true;
}

// Long path, in the reference loop's order: the crossings in [t_min, len + 1e-6] are
// walked in (t, triangle id) order with the table's hit rule, kLongChunk at a time.  Each
// pass traverses once, nearer child first, and keeps the kLongChunk smallest crossings
// beyond the last one walked (the ray's tmax shrinks to the largest kept one once the
// chunk is full, so the pass visits little beyond it); the walk then takes them, and a full
// chunk starts the next pass after its last crossing.  A crossing's t does not depend on tmin or tmax (the
// node and triangle slab tests only accept or reject), so the passes see exactly the
// crossings the reference's one-hit-per-trace loop sees, in the same order, while an
// edge with h crossings costs about h / kLongChunk traversals instead of h.
constexpr int kLongChunk = 16;

__device__ __forceinline__ void segment_long(Ray r, const int32_t* __restrict__ src, int nsrc,
                                             const BNode* __restrict__ nodes, uint32_t max_steps,
                                             const float4* __restrict__ tris, int swap, const PairTable& table) {
    EdgeWalk w;
    int32_t last = INT_MIN;
    const float tmax0 = r.tmax;
    bool cursor = false;  // (ct, cid): the last crossing of the previous pass
    float ct = 0.0f;
    uint32_t cid = 0;
    while (!w.done) {
        r.tmin = w.thr;
        r.tmax = tmax0;
        float lt[kLongChunk];
        uint32_t lid[kLongChunk];
        int32_t lobj[kLongChunk];
        int n = 0;
        const bool ok = traverse<-1, kStack, true>(nodes, max_steps, r, [&](int first, int cnt) {
            for (int k = first; k < first + cnt; ++k) {
                float a[3], b[3], c[3];
                uint32_t tid;
                int32_t obj;
                load_tri(tris, k, a, b, c, tid, obj);
                float t;
                if (!hit_triangle<-1>(r, a, b, c, t)) continue;
                if (cursor && !hit_less(ct, cid, t, tid)) continue;  // walked in an earlier pass
                if (n == kLongChunk && !hit_less(t, tid, lt[kLongChunk - 1], lid[kLongChunk - 1])) continue;
                int j = n < kLongChunk ? n++ : kLongChunk - 1;
                while (j > 0 && hit_less(t, tid, lt[j - 1], lid[j - 1])) {
                    lt[j] = lt[j - 1];
                    lid[j] = lid[j - 1];
                    lobj[j] = lobj[j - 1];
                    --j;
                }
                lt[j] = t;
                lid[j] = tid;
                lobj[j] = obj;
                if (n == kLongChunk) r.tmax = lt[kLongChunk - 1];
            }
        });
        if (!ok) {
            atomicOr(table.status, ST_STACK_OVERFLOW);
            break;
        }
        for (int j = 0; j < n && !w.done; ++j) {
            if (!w.take(lt[j], table.max_hits, table.next_float)) continue;
            if (lobj[j] != last) {
                last = lobj[j];
                insert_sources(table, src, nsrc, last, swap);
            }
        }
        if (n < kLongChunk) break;
        cursor = true;
        ct = lt[kLongChunk - 1];
        cid = lid[kLongChunk - 1];
    }
    count_edge(table, w.n);
}

// Edge i of a .pre edge payload (starts/ends float3, offsets/counts into sources).
struct EdgePayload {
    const float* starts;
    const float* ends;
    const int32_t* offsets;
    const int32_t* counts;
    const int32_t* sources;
};

__device__ __forceinline__ void edge_ray_long(const EdgePayload& p, uint64_t i, const BNode* __restrict__ nodes,
                                              uint32_t max_steps, const float4* __restrict__ tris, int swap,
                                              const PairTable& table) {
    Ray r;
    if (!segment_ray_of(p.starts[3 * i], p.starts[3 * i + 1], p.starts[3 * i + 2], p.ends[3 * i], p.ends[3 * i + 1],
                        p.ends[3 * i + 2], r))
        return;
    segment_long(r, p.sources + p.offsets[i], p.counts[i], nodes, max_steps, tris, swap, table);
}

// ---------------------------------------------------------------------------
// Ray packets: up to 32 rays by one warp, every lane busy.  One thread per ray ran 9 of 32
// lanes an instruction (the rays of a warp visit different numbers of nodes and reach their
// leaves at different steps) and left whole joins waiting on the thread with the longest
// traversal.  Here the warp's (node, ray) pairs lie on one shared-memory stack and its
// (leaf, ray) pairs in a ring: each step pops up to 32 nodes of any of the rays and tests
// both children of each, and 32 leaves at a time are tested once there are so many.  The
// visits, and so the crossings, are those of one traversal per ray.  Bound by the latency of
// the scattered node loads at 24 warps an SM: 6.6 KB a warp leaves the L1 cache 70 KB, where
// 32 warps of 64 registers (no spills gained) took 15 % longer and 16 warps 25 %.
// ---------------------------------------------------------------------------
constexpr int kPacketStack = 384;  // (node, ray) pairs
constexpr int kPacketRing = 128;   // (leaf, ray) pairs: below 32 before a step, which adds at most 64
constexpr int kPacketHits = kHits; // crossings kept per ray

struct RayPacket {
    float4 o[32];    // origin, tmax
    float4 d[32];    // direction
    float4 inv[32];  // 1 / direction as make_ray defines it
    int node[kPacketStack];
    uint2 leaf[kPacketRing];  // first triangle; count << 5 | ray
    float t[kPacketHits][32];
    int tri[kPacketHits][32];  // leaf-ordered triangle: its id and object are read at the end
    int n[32];
    unsigned char own[kPacketStack];
};

// Traces every lane's ray r (valid false: none; r.tmin is `tmin` for all) from node `start`: sm.n
// has its number of crossings, sm.t and sm.tri the first kPacketHits found.  Returns the
// lanes whose rays are not finished, the packet having run out of stack or of `max_steps`.
template <int AXIS>
__device__ __forceinline__ unsigned int packet_trace(RayPacket& sm, const Ray& mine, bool valid, int start,
                                                     const BNode* __restrict__ nodes, uint32_t max_steps,
                                                     const float4* __restrict__ tris, float tmin = kEps) {
    constexpr unsigned int kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned int below = (1u << lane) - 1u;
    if (valid) {
        sm.o[lane] = make_float4(mine.o[0], mine.o[1], mine.o[2], mine.tmax);
        if (AXIS < 0) {
            sm.d[lane] = make_float4(mine.d[0], mine.d[1], mine.d[2], 0.0f);
            sm.inv[lane] = make_float4(mine.inv[0], mine.inv[1], mine.inv[2], 0.0f);
        }
    }
    sm.n[lane] = 0;
    const unsigned int traced = __ballot_sync(kAll, valid);
    if (valid) {
        const int at = __popc(traced & below);
        sm.node[at] = start;
        sm.own[at] = (unsigned char)lane;
    }
    __syncwarp();
    int sp = __popc(traced);
    uint32_t head = 0, queued = 0, steps = 0;
    unsigned int tests = 0;
    auto ray_of = [&](int e, bool direction) {
        const float4 o = sm.o[e];
        if (AXIS >= 0)
            return make_ray(o.x, o.y, o.z, AXIS == 0 ? 1.0f : 0.0f, AXIS == 1 ? 1.0f : 0.0f, AXIS == 2 ? 1.0f : 0.0f,
                            tmin, o.w);
        const float4 inv = sm.inv[e];
        Ray r;
        r.o[0] = o.x; r.o[1] = o.y; r.o[2] = o.z;
        r.inv[0] = inv.x; r.inv[1] = inv.y; r.inv[2] = inv.z;
        r.tmin = tmin;
        r.tmax = o.w;
        if (direction) {
            const float4 d = sm.d[e];
            r.d[0] = d.x; r.d[1] = d.y; r.d[2] = d.z;
        }
        return r;
    };
    while (sp > 0 || queued > 0) {
        if (queued >= 32u || sp == 0) {
            const uint32_t m = min(queued, 32u);
            const uint2 leaf = (uint32_t)lane < m ? sm.leaf[(head + lane) & (kPacketRing - 1)] : make_uint2(0u, 0u);
            head += m;
            queued -= m;
            const int cnt = (int)(leaf.y >> 5), e = (int)(leaf.y & 31u);
            tests += (unsigned int)cnt;
            const int rounds = __reduce_max_sync(kAll, cnt);
            for (int k = 0; k < rounds; ++k) {
                if (k >= cnt) continue;
                float a[3], b[3], c[3], t;
                uint32_t tid;
                int32_t obj;
                load_tri(tris, (int)leaf.x + k, a, b, c, tid, obj);
                if (!hit_triangle<AXIS>(ray_of(e, true), a, b, c, t)) continue;
                const int slot = atomicAdd(&sm.n[e], 1);
                if (slot < kPacketHits) {
                    sm.t[slot][e] = t;
                    sm.tri[slot][e] = (int)leaf.x + k;
                }
            }
            __syncwarp();
            continue;
        }
        // No more nodes than leave kStackRoom entries: a wide traversal turns into a depth-first one.
        const int take = min(min(sp, 32), max(kPacketStack - kStackRoom - sp, 1));
        if (++steps > max_steps) break;
        sp -= take;
        bool h0 = false, h1 = false;
        int e = 0;
        int4 nd = make_int4(0, 0, 0, 0);
        if (lane < take) {
            const int node = sm.node[sp + lane];
            e = sm.own[sp + lane];
            const BNode bn = load_node(nodes, node);
            const float4 na = bn.a, nb = bn.b, nc = bn.c;
            nd = bn.d;
            const Ray r = ray_of(e, false);
            const float lo0[3] = {na.x, na.y, na.z}, hi0[3] = {na.w, nb.x, nb.y};
            const float lo1[3] = {nb.z, nb.w, nc.x}, hi1[3] = {nc.y, nc.z, nc.w};
            float en, ex;
            h0 = slab<AXIS>(r, lo0, hi0, r.tmin, r.tmax, en, ex);
            h1 = slab<AXIS>(r, lo1, hi1, r.tmin, r.tmax, en, ex);
        }
        __syncwarp();  // popped entries are read before they are overwritten
        const bool l0 = h0 && nd.y > 0, l1 = h1 && nd.w > 0;
        const unsigned int ml0 = __ballot_sync(kAll, l0), ml1 = __ballot_sync(kAll, l1);
        if (ml0 | ml1) {
            const uint32_t at = head + queued;
            if (l0) sm.leaf[(at + __popc(ml0 & below)) & (kPacketRing - 1)] = make_uint2((uint32_t)nd.x, (uint32_t)nd.y << 5 | (uint32_t)e);
            if (l1)
                sm.leaf[(at + __popc(ml0) + __popc(ml1 & below)) & (kPacketRing - 1)] =
                    make_uint2((uint32_t)nd.z, (uint32_t)nd.w << 5 | (uint32_t)e);
            queued += __popc(ml0) + __popc(ml1);
        }
        const bool p0 = h0 && nd.y <= 0, p1 = h1 && nd.w <= 0;
        const unsigned int mp0 = __ballot_sync(kAll, p0), mp1 = __ballot_sync(kAll, p1);
        const int pushed = __popc(mp0) + __popc(mp1);
        if (sp + pushed > kPacketStack) {  // the popped nodes lie there still
            sp += take;
            break;
        }
        if (p0) {
            const int at = sp + __popc(mp0 & below);
            sm.node[at] = nd.x;
            sm.own[at] = (unsigned char)e;
        }
        if (p1) {
            const int at = sp + __popc(mp0) + __popc(mp1 & below);
            sm.node[at] = nd.z;
            sm.own[at] = (unsigned char)e;
        }
        sp += pushed;
        __syncwarp();
    }
    __syncwarp();
    add_tests(tests);
    unsigned int unfinished = 0;
    for (int i = lane; i < sp; i += 32) unfinished |= 1u << sm.own[i];
    for (uint32_t i = lane; i < queued; i += 32) unfinished |= 1u << (sm.leaf[(head + i) & (kPacketRing - 1)].y & 31u);
    return __reduce_or_sync(kAll, unfinished);
}

// The advance rule on the crossings that packet_trace left for this lane (at most
// kPacketHits).
__device__ __forceinline__ Chain packet_chain(const RayPacket& sm, const float4* __restrict__ tris, int n) {
    const int lane = threadIdx.x & 31;
    HitList hl;
#pragma unroll
    for (int q = 0; q < kHits; ++q)
        if (q < n) {
            const size_t k = 3 * (size_t)sm.tri[q][lane];
            hl.t[q] = sm.t[q][lane];
            hl.id[q] = __float_as_uint(__ldg(&tris[k].w));
            hl.obj[q] = __float_as_int(__ldg(&tris[k + 1].w));
        }
    hl.n = n;
    return n <= 2 ? hl.finish2() : hl.finish();
}

// The edge of every lane (valid false: none), traversed from node `start`.  True for a lane
// whose edge has to be traced by the long path: more than kPacketHits crossings, or not
// finished when the packet ran out of stack or steps; nothing is inserted for it.
__device__ __forceinline__ bool edge_packet(RayPacket& sm, const EdgePayload& p, bool valid, uint64_t i, int start,
                                            const BNode* __restrict__ nodes, uint32_t max_steps,
                                            const float4* __restrict__ tris, int swap, const PairTable& table) {
    const int lane = threadIdx.x & 31;
    Ray r;
    if (valid)
        valid = segment_ray_of(p.starts[3 * i], p.starts[3 * i + 1], p.starts[3 * i + 2], p.ends[3 * i],
                               p.ends[3 * i + 1], p.ends[3 * i + 2], r);
    const unsigned int unfinished = packet_trace<-1>(sm, r, valid, start, nodes, max_steps, tris);
    if (!valid) return false;
    const int n = sm.n[lane];
    if ((unfinished >> lane & 1u) || n > kPacketHits) return true;
    // The crossings in (t, id) order, each the least above the one before.
    EdgeWalk w;
    int32_t last = INT_MIN;
    float ct = -INFINITY;
    uint32_t cid = 0;
    for (int k = 0; k < n && !w.done; ++k) {
        float bt = INFINITY;
        uint32_t bid = 0xffffffffu;
        int bk = 0;
        for (int j = 0; j < n; ++j) {
            const float t = sm.t[j][lane];
            const uint32_t id = __float_as_uint(__ldg(&tris[3 * (size_t)sm.tri[j][lane]].w));
            if ((k == 0 || hit_less(ct, cid, t, id)) && hit_less(t, id, bt, bid)) {
                bt = t;
                bid = id;
                bk = sm.tri[j][lane];
            }
        }
        const int32_t bobj = __float_as_int(__ldg(&tris[3 * (size_t)bk + 1].w));
        ct = bt;
        cid = bid;
        if (!w.take(bt, table.max_hits, table.next_float) || bobj == last) continue;
        last = bobj;
        insert_sources(table, p.sources + p.offsets[i], p.counts[i], bobj, swap);
    }
    count_edge(table, w.n);
    return false;
}

// Record r = 3 t + e: edge e of triangle t of a source mesh, in the triangle's own
// orientation (v0v1, v1v2, v2v0), with the triangle's object as its one source -- the
// legacy per-triangle overlap (mesh_overlap.cu:126-179), which traces shared edges once
// per triangle.
__device__ __forceinline__ bool triangle_edge_of(const float* __restrict__ V, const uint32_t* __restrict__ I,
                                                 uint64_t r, Ray& ray) {
    const uint64_t t = r / 3;
    const int e = (int)(r % 3);
    const uint64_t a = I[3 * t + e], b = I[3 * t + (e == 2 ? 0 : e + 1)];
    return segment_ray_of(V[3 * a], V[3 * a + 1], V[3 * a + 2], V[3 * b], V[3 * b + 1], V[3 * b + 2], ray);
}

}  // namespace
}  // namespace rs
