// rs_pim.cu -- point-in-mesh parity and the fused bounding-box filter.
//
// Replaces __raygen__rg (query/src/cuda/raytracing.cu:9-78) + __closesthit__ch
// (optix_common_shaders.cuh:12-19), RayLauncher (query/src/raytracing/RayLauncher.cpp:14-64),
// FilterRefinePipeline (query/src/raytracing/FilterRefine.cpp:10-122) and ResultProcessor
// (query/src/raytracing/ResultProcessor.cpp:8-60).
//
// The reference re-traces a closest-hit query from t_min = t + 1e-6 until it misses
// (crossings + 1 traversals per ray).  Here every crossing with t in [1e-6, 1e16] is
// collected once, by the warp, and the reference's advance rule is applied to the crossings
// in (t, triangle id) order.  Rays of more crossings than the query keeps follow in a second
// launch, a warp each, in ranges of t (pim_range_ray).
//
// Candidates come from one of two structures with the same hit set:
//  * rays along +x, +y or +z use a column grid: a uniform 2D grid over the projection
//    of the leaf-ordered triangles.  Triangle boxes and query points go through the
//    same monotone cell formula, so every triangle whose projection can contain the
//    (perturbed) point is in the point's cell; up to 8 crossings a lane, 256 a warp;
//  * any other direction traverses the BVH in packets of 32 rays, up to 8 crossings each.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "rs_engine.h"
#include "rs_prims.cuh"
#include "rs_query_core.cuh"

namespace rs {
namespace {

constexpr int kT = 256;

// Bounds of all vertices, and the box of 12 triangles over them that the filter's parity is
// defined by (BoundingBox::createBoxMesh, query/src/geometry/BoundingBox.cpp:12-50): three
// corners a triangle, bits 0, 1 and 2 of a corner choose the maximum in x, y and z.
struct BoxBounds {
    float mn[3], mx[3];
    int finite;
};

__constant__ unsigned char kBoxCorners[12][3] = {{0, 3, 1}, {0, 2, 3}, {4, 5, 7}, {4, 7, 6}, {0, 1, 5}, {0, 5, 4},
                                                 {2, 7, 3}, {2, 6, 7}, {0, 4, 6}, {0, 6, 2}, {1, 3, 7}, {1, 7, 5}};

// Whether the ray's parity against the box is odd.
template <int AXIS>
__device__ __forceinline__ bool box_filter(const BoxBounds& box, const Ray& r) {
    if (AXIS >= 0 && box.finite && isfinite(r.o[0]) && isfinite(r.o[1]) && isfinite(r.o[2])) {
        // In closed form (12 exact triangle tests took 80 % of a filtered query's time): the
        // four sides project to segments, which no perturbed point is inside of, and the two
        // triangles of an end cover its rectangle exactly once, so the ray crosses both ends
        // when the perturbed point (moved up by delta in u, delta^2 in v) is inside it.  An
        // end's box is flat, so its t is the rounded difference whatever its triangle.
        constexpr int W = AXIS >= 0 ? AXIS : 0, U = (W + 1) % 3, V = (W + 2) % 3;
        if (!(r.o[U] >= box.mn[U] && r.o[U] < box.mx[U] && r.o[V] >= box.mn[V] && r.o[V] < box.mx[V])) return false;
        Chain ch;
        const float t0 = __fsub_rn(box.mn[W], r.o[W]), t1 = __fsub_rn(box.mx[W], r.o[W]);
        if (t0 >= r.tmin && t0 <= r.tmax) ch.step(t0, 0);
        if (t1 >= r.tmin && t1 <= r.tmax) ch.step(t1, 0);
        return (ch.count & 1) != 0;
    }
    HitList hl;
#pragma unroll 1
    for (int k = 0; k < 12; ++k) {
        float v[3][3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int q = 0; q < 3; ++q) v[c][q] = (kBoxCorners[k][c] >> q) & 1 ? box.mx[q] : box.mn[q];
        float t;
        if (hit_triangle<AXIS>(r, v[0], v[1], v[2], t)) hl.add(t, (uint32_t)k, 0);
    }
    // A ray crosses at most two of the 12 faces under the hit contract.
    const Chain ch = hl.finish();
    return (ch.count & 1) != 0;
}


// Leaves ray i to the fallback.  *left (pinned host memory, nullable) tells the host that
// there is one, so that a query without any needs no read-back of the count.
__device__ __forceinline__ void leave_ray(uint32_t* __restrict__ ovf_list, unsigned long long* __restrict__ ovf_count,
                                          volatile int* left, uint32_t i) {
    ovf_list[atomicAdd(ovf_count, 1ull)] = i;
    if (left) *left = 1;
}

// BVH traversal in ray packets, for directions without a column grid.  Rays of more
// crossings than a packet keeps, or of a packet without room, go to the fallback.
constexpr int kPimT = 128;

template <int AXIS, bool FILTER>
__global__ void __launch_bounds__(kPimT, 6) k_pim(const float* __restrict__ pts, uint64_t n, float dx, float dy,
                                                  float dz, const BNode* __restrict__ nodes, uint32_t max_steps,
                                                  const float4* __restrict__ tris, BoxBounds box,
                                                  int32_t* __restrict__ out_obj, uint8_t* __restrict__ out_in,
                                                  uint32_t* __restrict__ ovf_list,
                                                  unsigned long long* __restrict__ ovf_count,
                                                  volatile int* __restrict__ left) {
    __shared__ RayPacket packets[kPimT / 32];
    RayPacket& sm = packets[threadIdx.x >> 5];
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const bool valid = i < n;
    Ray r;
    bool keep = valid;
    if (valid) {
        r = make_ray(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], dx, dy, dz, kEps, kTmax);
        if (FILTER) keep = box_filter<AXIS>(box, r);
    }
    const bool ok = !(packet_trace<AXIS>(sm, r, keep, 0, nodes, max_steps, tris) >> (threadIdx.x & 31) & 1u);
    const int hits = keep ? sm.n[threadIdx.x & 31] : 0;
    if (!valid) return;
    if (keep && (!ok || hits > kPacketHits)) leave_ray(ovf_list, ovf_count, left, (uint32_t)i);
    else write_result(packet_chain(sm, tris, hits), i, out_obj, out_in);
}

// Column-grid query, 32 points a warp (pim_grid_warp).
constexpr int kWarps = kT / 32;
constexpr int kGridBlocks = 4;  // resident blocks an SM

template <int AXIS, bool FILTER>
__global__ void __launch_bounds__(kT, kGridBlocks) k_pim_grid(const float* __restrict__ pts, uint64_t n, GridView g,
                                                 const float4* __restrict__ tris, BoxBounds box,
                                                 int32_t* __restrict__ out_obj, uint8_t* __restrict__ out_in,
                                                 uint32_t* __restrict__ ovf_list,
                                                 unsigned long long* __restrict__ ovf_count,
                                                 volatile int* __restrict__ left) {
    __shared__ GridWarpSlots slots[kWarps];
    grid_points<AXIS>(
        g, tris, blockIdx.x * (uint64_t)kT + threadIdx.x, n, (uint64_t)gridDim.x * kT, out_obj, out_in,
        slots[threadIdx.x >> 5],
        [&](uint64_t i, float* p) {
#pragma unroll
            for (int q = 0; q < 3; ++q) p[q] = __ldcs(&pts[3 * i + q]);
        },
        [&](const float* p) {
            return !FILTER || box_filter<AXIS>(box, make_ray(p[0], p[1], p[2], AXIS == 0 ? 1.0f : 0.0f,
                                                             AXIS == 1 ? 1.0f : 0.0f, AXIS == 2 ? 1.0f : 0.0f, kEps,
                                                             kTmax));
        },
        [&](uint32_t i) { leave_ray(ovf_list, ovf_count, left, i); });
}

// The rays left over: of more than kDenseHits crossings on a column grid, of more than kPacketHits
// or of an unfinished packet otherwise.  80 registers and 6 blocks an SM: 10 % less than 126 and
// 4, or 72 and 7.
template <int AXIS>
__global__ void __launch_bounds__(32 * kRangeWarps, 6) k_pim_fallback(
    const float* __restrict__ pts, float dx, float dy, float dz, const BNode* __restrict__ nodes, uint32_t max_steps,
    const float4* __restrict__ tris, int32_t* __restrict__ out_obj, uint8_t* __restrict__ out_in,
    unsigned int* __restrict__ status, const uint32_t* __restrict__ ovf_list,
    const unsigned long long* __restrict__ ovf_count) {
    __shared__ RangeWarp warps[kRangeWarps];
    const unsigned long long cnt = *ovf_count;
    for (unsigned long long q = blockIdx.x * (unsigned long long)kRangeWarps + (threadIdx.x >> 5); q < cnt;
         q += (unsigned long long)gridDim.x * kRangeWarps) {
        const uint64_t i = ovf_list[q];
        const Ray r = make_ray(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], dx, dy, dz, kEps, kTmax);
        pim_range_ray<AXIS>(warps[threadIdx.x >> 5], nodes, max_steps, tris, r, status, out_obj, out_in, i);
        __syncwarp();
    }
}

// --- column grid build ---------------------------------------------------------------

// Box of triangle k: across the ray axis (u, v) and along it.
struct TriBox {
    float ul, uh, vl, vh, wl, wh;
    bool nan;  // a coordinate is not a number
};

template <int AXIS>
__device__ __forceinline__ TriBox tri_box(const float4* __restrict__ tris, int k) {
    const float4 a = __ldg(&tris[3 * (size_t)k]), b = __ldg(&tris[3 * (size_t)k + 1]),
                 c = __ldg(&tris[3 * (size_t)k + 2]);
    const float au = AXIS == 0 ? a.y : (AXIS == 1 ? a.z : a.x), av = AXIS == 0 ? a.z : (AXIS == 1 ? a.x : a.y);
    const float bu = AXIS == 0 ? b.y : (AXIS == 1 ? b.z : b.x), bv = AXIS == 0 ? b.z : (AXIS == 1 ? b.x : b.y);
    const float cu = AXIS == 0 ? c.y : (AXIS == 1 ? c.z : c.x), cv = AXIS == 0 ? c.z : (AXIS == 1 ? c.x : c.y);
    const float aw = AXIS == 0 ? a.x : (AXIS == 1 ? a.y : a.z), bw = AXIS == 0 ? b.x : (AXIS == 1 ? b.y : b.z);
    const float cw = AXIS == 0 ? c.x : (AXIS == 1 ? c.y : c.z);
    TriBox r;
    r.ul = fminf(fminf(au, bu), cu);
    r.uh = fmaxf(fmaxf(au, bu), cu);
    r.vl = fminf(fminf(av, bv), cv);
    r.vh = fmaxf(fmaxf(av, bv), cv);
    r.wl = fminf(fminf(aw, bw), cw);
    r.wh = fmaxf(fmaxf(aw, bw), cw);
    r.nan = isnan(au) || isnan(av) || isnan(aw) || isnan(bu) || isnan(bv) || isnan(bw) || isnan(cu) || isnan(cv) ||
            isnan(cw);
    return r;
}

__device__ __forceinline__ int ford(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}

// Bounds of all triangles (b: ordered ints: u, v, w ranges) and the sums of their projected
// boxes' widths, heights and areas (finite ones each), which choose the cell size.
template <int AXIS>
__global__ void k_cg_bounds(const float4* __restrict__ tris, int n, int* __restrict__ b, double* __restrict__ sums) {
    // [0..5] minima of u, -u, v, -v, w, -w, then the three sums (a thread sums a few dozen
    // boxes: the sizing needs no more digits).
    float v[9] = {INFINITY, INFINITY, INFINITY, INFINITY, INFINITY, INFINITY, 0.0f, 0.0f, 0.0f};
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const TriBox t = tri_box<AXIS>(tris, k);
        // A coordinate that is not a number may be crossed at any height: no height limit then.
        const float m[6] = {t.ul, -t.uh, t.vl, -t.vh, t.wl, t.nan ? -INFINITY : -t.wh};
#pragma unroll
        for (int q = 0; q < 6; ++q) v[q] = fminf(v[q], m[q]);
        const float w = t.uh - t.ul, h = t.vh - t.vl;
        v[6] += w < INFINITY ? w : 0.0f;
        v[7] += h < INFINITY ? h : 0.0f;
        v[8] += w * h < INFINITY ? w * h : 0.0f;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const float y = __shfl_xor_sync(0xffffffffu, v[q], o);
            v[q] = q < 6 ? fminf(v[q], y) : v[q] + y;
        }
    __shared__ float red[9][8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 9; ++q) red[q][warp] = v[q];
    __syncthreads();
    if (threadIdx.x >= 9) return;
    const int q = threadIdx.x;
    float x = red[q][0];
    for (int w = 1; w < 8; ++w) x = q < 6 ? fminf(x, red[q][w]) : x + red[q][w];
    if (q >= 6) atomicAdd(&sums[q - 6], (double)x);
    else if (q & 1) atomicMax(&b[q], ford(-x));
    else atomicMin(&b[q], ford(x));
}

// Counts (FILL false) or lists (FILL true, count holding each cell's length) the cells that
// every triangle's projected box touches.  A warp flattens the rectangles of its 32
// triangles into one work list, so a lane never walks a large rectangle alone; the fill
// takes its slots from the cell's end, and the counts are back at zero after it.
template <int AXIS, bool FILL>
__global__ void __launch_bounds__(256) k_cg_cells(const float4* __restrict__ tris, int n, GridView g,
                                                  uint32_t* __restrict__ count, uint2* __restrict__ list) {
    const int lane = threadIdx.x & 31;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t cells = 0, width = 1;
    int cu0 = 0, cv0 = 0;
    float ful = 0.0f, fuh = 0.0f, fvl = 0.0f, fvh = 0.0f;  // the box in cell units
    uint32_t high = 0;
    if (k < n) {
        const TriBox t = tri_box<AXIS>(tris, k);
        const int cu1 = cell_of(t.uh, g.u0, g.su, g.gu), cv1 = cell_of(t.vh, g.v0, g.sv, g.gv);
        cu0 = cell_of(t.ul, g.u0, g.su, g.gu);
        cv0 = cell_of(t.vl, g.v0, g.sv, g.gv);
        if (cu1 >= cu0 && cv1 >= cv0) {
            width = (uint32_t)(cu1 - cu0 + 1);
            cells = width * (uint32_t)(cv1 - cv0 + 1);
        }
        if (FILL) {
            // A triangle with a coordinate that is not a number covers its cells whole.
            ful = t.nan ? -INFINITY : cell_units(t.ul, g.u0, g.su);
            fuh = t.nan ? INFINITY : cell_units(t.uh, g.u0, g.su);
            fvl = t.nan ? -INFINITY : cell_units(t.vl, g.v0, g.sv);
            fvh = t.nan ? INFINITY : cell_units(t.vh, g.v0, g.sv);
            high = t.nan ? 255u : height_units(g, t.wh);
        }
    }
    uint32_t inc = cells;  // 32 rectangles of at most 2^26 cells fit
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    const uint32_t pre = inc - cells, total = __shfl_sync(0xffffffffu, inc, 31);
    for (uint32_t base = 0; base < total; base += 32) {
        const uint32_t j = base + lane;
        int owner = 0;  // the last lane whose prefix is <= j
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
            const uint32_t pc = __shfl_sync(0xffffffffu, pre, owner + step);
            if (pc <= j) owner += step;
        }
        const int ou = __shfl_sync(0xffffffffu, cu0, owner), ov = __shfl_sync(0xffffffffu, cv0, owner);
        const uint32_t ow = __shfl_sync(0xffffffffu, width, owner), op = __shfl_sync(0xffffffffu, pre, owner);
        const uint32_t r = j - op, row = r / ow;
        const int cu = ou + (int)(r - row * ow), cv = ov + (int)row;
        const size_t c = (size_t)cv * g.gu + cu;
        if (!FILL) {
            if (j < total) atomicAdd(&count[c], 1u);
            continue;
        }
        const int ok = __shfl_sync(0xffffffffu, k, owner);
        const float a0 = __shfl_sync(0xffffffffu, ful, owner), a1 = __shfl_sync(0xffffffffu, fuh, owner);
        const float a2 = __shfl_sync(0xffffffffu, fvl, owner), a3 = __shfl_sync(0xffffffffu, fvh, owner);
        const uint32_t oh = __shfl_sync(0xffffffffu, high, owner);
        if (j < total) {
            const uint32_t y = unit_in_cell(a0, cu) | unit_in_cell(a1, cu) << 6 | unit_in_cell(a2, cv) << 12 |
                               unit_in_cell(a3, cv) << 18 | oh << 24;
            list[g.start[c] + atomicSub(&count[c], 1u) - 1u] = make_uint2((uint32_t)ok, y);
        }
    }
}

std::mutex g_grid_mu;

float dec_ord(int i) {
    int x = i >= 0 ? i : i ^ 0x7fffffff;
    float f;
    std::memcpy(&f, &x, 4);
    return f;
}

// Cells of a grid over n triangles with the given projected extent and sums of box widths,
// heights and areas.  At most four per triangle (and 2^24): more would not shorten the
// lists of a mesh whose boxes are as small as its cells.  At s cells per unit of length a
// box of w x h touches about (s w + 1)(s h + 1) cells, so n boxes make about
// s^2 sum(w h) + s (sum w + sum h) + n list entries; cells are made larger until that is at
// most kEntries a triangle, since many small objects over a wide scene would otherwise list
// every triangle in a hundred cells and more.  20,000 level-2 spheres, 6.4 M triangles, asked
// for 500,009 points: 920 M entries took 27 ms to count and list and .57 ms to ask; at 12
// entries a triangle 0.93 + 0.99 ms, at 8 0.58 + 1.04, at 5 0.44 + 1.18.  Up to kFree entries
// the build takes no longer than its launches and stays at four cells a triangle.
constexpr double kEntries = 8.0;
constexpr double kFree = 4194304.0;

double grid_cells(double n, double w, double h, const double* sum) {
    const double finest = std::min(std::max(4.0 * n, 1.0), (double)(1 << 24));
    const double budget = std::max(kEntries * n, kFree);
    if (!(w > 0 && h > 0) || !std::isfinite(w * h)) return finest;
    const double s0 = std::sqrt(finest / (w * h)), lin = sum[0] + sum[1], area = sum[2];
    if (!(s0 * s0 * area + s0 * lin + n > budget)) return finest;
    const double room = budget - n;
    const double s = area > 0 ? (-lin + std::sqrt(lin * lin + 4.0 * area * room)) / (2.0 * area) : room / lin;
    return std::min(std::max(finest * (s / s0) * (s / s0), 1.0), finest);
}

struct GridSize {
    int gu, gv;
};

// Columns and rows of about `target` cells, shaped like the projected bounds (endless ones have a
// scale of zero, so one cell).
GridSize grid_shape(double target, double w, double h) {
    GridSize g{1, 1};
    if (!std::isfinite(w)) w = 0.0;
    if (!std::isfinite(h)) h = 0.0;
    if (w > 0 && h > 0) {
        g.gu = (int)std::lround(std::min(std::max(std::sqrt(target * w / h), 1.0), 8192.0));
        g.gv = (int)std::lround(std::min(std::max(target / g.gu, 1.0), 8192.0));
    } else if (w > 0) {
        g.gu = (int)std::min(std::max(target, 1.0), 8192.0);
    } else if (h > 0) {
        g.gv = (int)std::min(std::max(target, 1.0), 8192.0);
    }
    return g;
}

// The grid's size, halved until its own cells -- not square where the bounds are longer than
// 8,192 cells, or flat -- keep about the entries that grid_cells allows, and until no place of
// the boxes in them can make 2^32 (a box of w x h cells touches at most (w + 2)(h + 2); from
// 2^30 triangles on, that many around the same cells' corners, one in two is allowed for).
// Without it strips across a band a million times as long as wide lie in 408 rows each: 412 M
// entries for 1 M strips, and more than 2^32 for 10.5 M.
GridSize grid_size(double n, double w, double h, const double* sum) {
    const double budget = std::max(kEntries * n, kFree), slack = n < 1073741824.0 ? 4.0 : 2.0;
    // Areas that overflowed a float are not in the sum.
    const double area = w * h < 1e38 ? sum[2] : std::min(sum[0] * h, sum[1] * w);
    for (double target = grid_cells(n, w, h, sum);; target *= 0.5) {
        const GridSize g = grid_shape(target, w, h);
        const double su = w > 0 && std::isfinite(w) ? g.gu / w : 0.0, sv = h > 0 && std::isfinite(h) ? g.gv / h : 0.0;
        const double boxes = su > 0 && sv > 0 ? su * sv * area : 0.0, edges = su * sum[0] + sv * sum[1];
        if (g.gu * g.gv == 1 ||
            (boxes + edges + n <= 2.0 * budget && boxes + 2.0 * edges + slack * n < 4294967296.0))
            return g;
    }
}

template <int AXIS>
cudaError_t build_grid(rs_bvh* bvh, cudaStream_t s) {
    rs_column_grid& cg = bvh->cgrid[AXIS];
    const int n = (int)bvh->n_tris;
    int* b = nullptr;  // six ordered ints, then three sums
    constexpr size_t kBytes = 6 * sizeof(int) + 3 * sizeof(double);
    cudaError_t e = dmalloc((void**)&b, kBytes, s);
    if (e != cudaSuccess) return e;
    struct {
        int b[6] = {0x7fffffff, (int)0x80000000, 0x7fffffff, (int)0x80000000, 0x7fffffff, (int)0x80000000};
        double sum[3] = {0.0, 0.0, 0.0};
    } h;
    static_assert(sizeof(h) == kBytes, "bounds layout");
    cudaMemcpyAsync(b, &h, kBytes, cudaMemcpyHostToDevice, s);
    launch(k_cg_bounds<AXIS>, std::min(2 * sm_count(), (n + 255) / 256), 256, 0, s, (const float4*)bvh->tris, n, b,
           reinterpret_cast<double*>(b + 6));
    e = cudaMemcpyAsync(&h, b, kBytes, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFreeAsync(b, s);
    if (e != cudaSuccess) return e;
    cg.u0 = dec_ord(h.b[0]);
    cg.u1 = dec_ord(h.b[1]);
    cg.v0 = dec_ord(h.b[2]);
    cg.v1 = dec_ord(h.b[3]);
    cg.w0 = dec_ord(h.b[4]);
    cg.w1 = dec_ord(h.b[5]);
    const double depth = (double)cg.w1 - cg.w0;
    cg.sw = depth > 0 ? (float)(256.0 / depth) : 0.0f;
    const double w = (double)cg.u1 - cg.u0, hh = (double)cg.v1 - cg.v0;
    const GridSize size = grid_size(n, w, hh, h.sum);
    const int gu = size.gu, gv = size.gv;
    cg.gu = gu;
    cg.gv = gv;
    cg.su = w > 0 ? (float)gu / (float)w : 0.0f;
    cg.sv = hh > 0 ? (float)gv / (float)hh : 0.0f;
    const size_t ncell = (size_t)gu * gv;
    uint32_t* count = nullptr;
    e = dmalloc((void**)&count, ncell * sizeof(uint32_t), s);
    if (e == cudaSuccess) e = dmalloc((void**)&cg.start, (ncell + 1) * sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    const GridView gvw = grid_view(cg);
    cudaMemsetAsync(count, 0, ncell * sizeof(uint32_t), s);
    const unsigned grid = (unsigned)((n + 255) / 256);
    launch(k_cg_cells<AXIS, false>, grid, 256, 0, s, (const float4*)bvh->tris, n, gvw, count, (uint2*)nullptr);
    e = exclusive_scan_u32(count, cg.start, ncell, cg.start + ncell, s);
    uint32_t total = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&total, cg.start + ncell, sizeof(total), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = dmalloc((void**)&cg.list, (size_t)std::max<uint32_t>(total, 1) * sizeof(uint2), s);
    if (e == cudaSuccess) {
        launch(k_cg_cells<AXIS, true>, grid, 256, 0, s, (const float4*)bvh->tris, n, gvw, count, cg.list);
        e = cudaGetLastError();
    }
    cudaFreeAsync(count, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cg.nlist = total;
    if (e == cudaSuccess) cg.built = 1;
    return e;
}

// Blocks of k_pim_grid: one resident wave at most.
unsigned grid_blocks(uint64_t n) {
    return (unsigned)std::min<uint64_t>((n + kT - 1) / kT, (uint64_t)kGridBlocks * sm_count());
}

template <int AXIS, bool FILTER>
cudaError_t launch_pim(const rs_bvh* bvh, const float* pts, uint64_t n, float dx, float dy, float dz,
                       const BoxBounds& box, int32_t* obj, uint8_t* in, uint32_t* ovf_list,
                       unsigned long long* ovf_count, volatile int* left, cudaStream_t s) {
    constexpr int GA = AXIS < 0 ? 0 : AXIS;
    const int ptok = prof_begin(P_PIM, s);
    if (AXIS >= 0 && bvh->cgrid[GA].built) {
        const GridView g = grid_view(bvh->cgrid[GA]);
        launch(k_pim_grid<GA, FILTER>, grid_blocks(n), kT, 0, s, pts, n, g, (const float4*)bvh->tris, box, obj, in,
               ovf_list, ovf_count, left);
    } else {
        launch(k_pim<AXIS, FILTER>, (unsigned)((n + kPimT - 1) / kPimT), kPimT, 0, s, pts, n, dx, dy, dz, bvh->nodes,
               max_steps(bvh), (const float4*)bvh->tris, box, obj, in, ovf_list, ovf_count, left);
    }
    prof_end(P_PIM, s, ptok);
    return cudaGetLastError();
}

// Launches the query, waits for it, and resolves the rays it left in ovf_list (their count
// is known then, so a query without any pays for no second launch).  meta: status word,
// overflow count, both zero before the call; h: their host copy.  left: a pinned word, zero
// before the call, that says whether there is anything to read back (nullable: read back).
template <int AXIS>
int run_pim_axis(const rs_bvh* bvh, const float* pts, uint64_t n, float dx, float dy, float dz, bool filter,
                 const BoxBounds& box, int32_t* obj, uint8_t* in, unsigned long long* meta, unsigned long long* h,
                 volatile int* left, uint32_t* ovf, cudaStream_t s) {
    unsigned int* status = reinterpret_cast<unsigned int*>(meta);
    cudaError_t e = filter ? launch_pim<AXIS, true>(bvh, pts, n, dx, dy, dz, box, obj, in, ovf, meta + 1, left, s)
                           : launch_pim<AXIS, false>(bvh, pts, n, dx, dy, dz, box, obj, in, ovf, meta + 1, left, s);
    constexpr size_t kWords = 2 * sizeof(unsigned long long);
    cudaError_t e2 = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = e2;
    if (e == cudaSuccess && (!left || *left)) {
        e = cudaMemcpyAsync(h, meta, kWords, cudaMemcpyDeviceToHost, s);
        e2 = cudaStreamSynchronize(s);
        if (e == cudaSuccess) e = e2;
    }
    if (e == cudaSuccess && h[1]) {
        const uint64_t blocks = std::min<uint64_t>((h[1] + kRangeWarps - 1) / kRangeWarps, 16ull * sm_count());
        launch(k_pim_fallback<AXIS>, (unsigned)blocks, 32 * kRangeWarps, 0, s, pts, dx, dy, dz, bvh->nodes,
               max_steps(bvh), (const float4*)bvh->tris, obj, in, status, (const uint32_t*)ovf,
               (const unsigned long long*)(meta + 1));
        e = cudaMemcpyAsync(h, meta, kWords, cudaMemcpyDeviceToHost, s);
        e2 = cudaStreamSynchronize(s);
        if (e == cudaSuccess) e = e2;
    }
    prof_collect();
    return e == cudaSuccess ? status_from_bits((uint32_t)h[0]) : to_status(e);
}

int pim_axis(float dx, float dy, float dz) {
    const bool zx = dx == 0.0f, zy = dy == 0.0f, zz = dz == 0.0f;
    if (dz == 1.0f && zx && zy) return 2;
    if (dx == 1.0f && zy && zz) return 0;
    if (dy == 1.0f && zx && zz) return 1;
    return -1;
}

int run_pim(int axis, const rs_bvh* bvh, const float* pts, uint64_t n, float dx, float dy, float dz, bool filter,
            const BoxBounds& box, int32_t* obj, uint8_t* in, unsigned long long* meta, unsigned long long* h,
            volatile int* left, uint32_t* ovf, cudaStream_t s) {
    switch (axis) {
        case 0: return run_pim_axis<0>(bvh, pts, n, dx, dy, dz, filter, box, obj, in, meta, h, left, ovf, s);
        case 1: return run_pim_axis<1>(bvh, pts, n, dx, dy, dz, filter, box, obj, in, meta, h, left, ovf, s);
        case 2: return run_pim_axis<2>(bvh, pts, n, dx, dy, dz, filter, box, obj, in, meta, h, left, ovf, s);
        default: return run_pim_axis<-1>(bvh, pts, n, dx, dy, dz, filter, box, obj, in, meta, h, left, ovf, s);
    }
}

BoxBounds make_box(const rs_bvh* bvh) {
    BoxBounds b;
    b.finite = 1;
    for (int k = 0; k < 3; ++k) {
        b.mn[k] = bvh->vmin[k];
        b.mx[k] = bvh->vmax[k];
        if (!std::isfinite(b.mn[k]) || !std::isfinite(b.mx[k])) b.finite = 0;
    }
    return b;
}

// The status word and overflow count of a call, device memory that is zero while it waits in
// its device's pool, and pinned words for their copy and run_pim's `left`: a call then needs
// neither an allocation nor a memset for them, and a copy back only when rays were left.  A call
// has one to itself until it has synchronised, so calls on other streams and threads have others.
struct CallWords {
    unsigned long long* dev = nullptr;
    unsigned long long* host = nullptr;
};
std::mutex g_words_mu;
std::vector<CallWords> g_words[64];
size_t g_words_made[64];  // room in the vector for all of them, so that giving one back cannot throw

cudaError_t words_acquire(int device, CallWords* out, cudaStream_t s) {
    if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> g(g_words_mu);
    std::vector<CallWords>& pool = g_words[device];
    if (pool.empty()) {  // as many as are ever in flight together, kept until the process ends
        constexpr int kBlock = 32;
        unsigned long long *d = nullptr, *h = nullptr;
        try {
            pool.reserve(g_words_made[device] + kBlock);
        } catch (...) {
            return cudaErrorMemoryAllocation;
        }
        // Relaxed, and no work on the legacy stream: another thread may be capturing a stream.
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        cudaError_t e = cudaMalloc((void**)&d, kBlock * 256);
        if (e == cudaSuccess) e = cudaMallocHost((void**)&h, kBlock * 256);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e == cudaSuccess) e = cudaMemsetAsync(d, 0, kBlock * 256, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            if (d) cudaFree(d);
            if (h) cudaFreeHost(h);
            return e;
        }
        for (int k = 0; k < kBlock; ++k) pool.push_back(CallWords{d + 32 * k, h + 32 * k});
        g_words_made[device] += kBlock;
    }
    *out = pool.back();
    pool.pop_back();
    return cudaSuccess;
}

// After the call's stream has been synchronised; words that are not zero are zeroed first.
void words_release(int device, const CallWords& w, bool clean, cudaStream_t s) {
    if (!clean && (cudaMemsetAsync(w.dev, 0, 16, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess))
        return;  // not reused
    std::lock_guard<std::mutex> g(g_words_mu);
    g_words[device].push_back(w);
}

int pim_impl(const rs_bvh* cbvh, const float* pts, uint64_t n, float dx, float dy, float dz, int32_t* obj,
             uint8_t* in, bool filter, cudaStream_t s) {
    if (!cbvh || (n && !pts)) return RS_ERR_INVALID;
    if (n == 0) return RS_OK;
    if (n > 0xffffffffull) return RS_ERR_INVALID;
    rs_bvh* bvh = const_cast<rs_bvh*>(cbvh);
    int st = filter ? bvh_ready(bvh) : RS_OK;
    if (st == RS_OK) st = bvh_use(bvh, s);
    if (st != RS_OK) return st;
    if (filter && bvh->nV == 0) {
        cudaError_t e = cudaSuccess;
        if (obj) e = cudaMemsetAsync(obj, 0xff, n * sizeof(int32_t), s);
        if (e == cudaSuccess && in) e = cudaMemsetAsync(in, 0, n, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        return to_status(e);
    }
    const int axis = pim_axis(dx, dy, dz);
    if (axis >= 0) {
        st = ensure_grid(bvh, axis, s);
        if (st != RS_OK) return st;
    }
    int device = 0;
    CallWords words;
    uint32_t* ovf = nullptr;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = words_acquire(device, &words, s);
    if (e != cudaSuccess) return to_status(e);
    e = dmalloc((void**)&ovf, n * sizeof(uint32_t), s);
    if (e != cudaSuccess) {
        words_release(device, words, true, s);
        cudaStreamSynchronize(s);
        return to_status(e);
    }
    const BoxBounds box = filter ? make_box(bvh) : BoxBounds{};
    words.host[0] = words.host[1] = words.host[2] = 0;
    st = run_pim(axis, bvh, pts, n, dx, dy, dz, filter, box, obj, in, words.dev, words.host,
                 reinterpret_cast<volatile int*>(words.host + 2), ovf, s);
    cudaFreeAsync(ovf, s);
    words_release(device, words, st == RS_OK && words.host[0] == 0 && words.host[1] == 0, s);
    return st;
}

// Ordered compaction in one pass: a block takes the next tile of kHitTile points (in start
// order), counts its hits, learns the number before it by decoupled look-back over the
// earlier tiles' words (flag | count: a tile's own number, or the number through it), and
// writes ids and objects in order.  It reads the objects once -- the flags, scan and scatter
// passes it replaces moved 20 bytes a point (60 M points: 700 us; 4 bytes a point and 8 a
// hit: 175).  *total receives the number of hits (pinned host memory).  Look-back waits only
// on blocks that started earlier, and at most kHitSpins polls.
constexpr int kHitPer = 4;  // 16-byte loads a thread
constexpr int kHitTile = kT * kHitPer * 4;
constexpr unsigned long long kHitOwn = 1ull << 62, kHitThrough = 2ull << 62, kHitCount = (1ull << 62) - 1;
constexpr uint32_t kHitSpins = 1u << 22;

template <bool VEC>
__global__ void __launch_bounds__(kT) k_hits(const int32_t* __restrict__ obj, uint64_t n, int32_t* __restrict__ ids,
                                             int32_t* __restrict__ objs, uint64_t capacity,
                                             unsigned long long* __restrict__ words, unsigned int* __restrict__ next,
                                             volatile int* __restrict__ total) {
    constexpr unsigned int kAll = 0xffffffffu;
    __shared__ uint32_t s_cnt[kHitPer * kWarps];
    __shared__ unsigned int s_tile;
    __shared__ unsigned long long s_before;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = next ? atomicAdd(next, 1u) : 0u;
    __syncthreads();
    const uint64_t tile = s_tile, base = tile * kHitTile;
    // Element j of load k of this thread is point base + (k * kT + tid) * 4 + j.
    int32_t o[kHitPer][4];
    uint32_t before[kHitPer];  // hits of the warp before this thread's, in load k
#pragma unroll
    for (int k = 0; k < kHitPer; ++k) {
        const uint64_t i = base + ((uint64_t)k * kT + tid) * 4;
        if (VEC && i + 4 <= n) {
            const int4 v = __ldcs(reinterpret_cast<const int4*>(obj + i));
            o[k][0] = v.x; o[k][1] = v.y; o[k][2] = v.z; o[k][3] = v.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) o[k][j] = i + j < n ? obj[i + j] : -1;
        }
    }
#pragma unroll
    for (int k = 0; k < kHitPer; ++k) {
        uint32_t b = 0, all = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const unsigned int m = __ballot_sync(kAll, o[k][j] != -1);
            b += __popc(m & ((1u << lane) - 1u));
            all += __popc(m);
        }
        before[k] = b;
        if (lane == 0) s_cnt[k * kWarps + warp] = all;
    }
    __syncthreads();
    if (warp == 0) {
        static_assert(kHitPer * kWarps == 32, "one lane per warp and load");
        const uint32_t c = s_cnt[lane];
        uint32_t x = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kAll, x, d);
            if (lane >= d) x += y;
        }
        s_cnt[lane] = x - c;
        const uint32_t mine = __shfl_sync(kAll, x, 31);
        unsigned long long sum = 0;
        bool ok = true;
        if (words) {
            volatile unsigned long long* w = words;
            if (lane == 0) w[tile] = (tile == 0 ? kHitThrough : kHitOwn) | mine;
            // 32 earlier tiles at a time, nearest first.
            long long j = (long long)tile - 1;
            uint32_t spins = 0;
            while (j >= 0) {
                const unsigned long long v = j - lane >= 0 ? +w[j - lane] : 2ull << 62;
                const unsigned int absent = __ballot_sync(kAll, (v & ~kHitCount) == 0);
                const unsigned int through = __ballot_sync(kAll, (v & ~kHitCount) == kHitThrough);
                const int use = absent ? __ffs(absent) - 1 : 32, last = through ? __ffs(through) - 1 : 32;
                unsigned long long add = lane < use && lane <= last ? v & kHitCount : 0ull;
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) add += __shfl_xor_sync(kAll, add, d);
                sum += add;
                if (last < use) break;
                if (use == 0 && ++spins > kHitSpins) {
                    ok = false;
                    break;
                }
                j -= use;
            }
            if (tile > 0 && lane == 0) w[tile] = kHitThrough | (sum + mine);
        }
        if (lane == 0) {
            s_before = sum;
            if (!ok) total[1] = 1;
            if (base + kHitTile >= n) total[0] = (int)(uint32_t)(sum + mine);
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kHitPer; ++k) {
        unsigned long long p = s_before + s_cnt[k * kWarps + warp] + before[k];
        const uint64_t i = base + ((uint64_t)k * kT + tid) * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (o[k][j] == -1) continue;
            if (p < capacity) {
                if (ids) ids[p] = (int32_t)(i + j);
                if (objs) objs[p] = o[k][j];
            }
            ++p;
        }
    }
}

}  // namespace

// The column grid of one axis is built once per handle, like the index build of the
// reference (allocates and synchronises the stream).
int ensure_grid(const rs_bvh* cbvh, int axis, cudaStream_t s) {
    rs_bvh* bvh = const_cast<rs_bvh*>(cbvh);
    if (axis < 0 || axis > 2 || bvh->n_tris == 0 || bvh->cgrid[axis].built) return RS_OK;
    std::lock_guard<std::mutex> g(g_grid_mu);
    if (!bvh->cgrid[axis].built) {
        cudaError_t e = axis == 0 ? build_grid<0>(bvh, s) : (axis == 1 ? build_grid<1>(bvh, s) : build_grid<2>(bvh, s));
        if (e != cudaSuccess) return to_status(e);
    }
    return RS_OK;
}


int recheck_pim(int op, unsigned long long* out) { return recheck_op(op, out); }

}  // namespace rs

// ---------------------------------------------------------------------------
// Point-in-mesh without device allocation.
//
// Callers that cannot allocate device memory on their query path -- services whose
// own allocator has reserved the whole GPU, or hosts with a fixed device-memory budget
// checked per request -- use rs_pim_noalloc.  It waits for the stream and returns once
// the results are written.  Its per-call scratch (status word, overflow count and the list
// of points that the query leaves to the fallback) lives
// in the fixed array below instead of coming from an allocator.  Host code may not
// use the array's name as a device address, so its address is looked up with
// cudaGetSymbolAddress once per device (with that device current) and passed to
// the kernels.
// ---------------------------------------------------------------------------
constexpr uint64_t kNoAllocMaxPoints = 1ull << 20;  // 1,048,576 points per call
constexpr size_t kNoAllocMetaOffset = 0;            // u64 status, u64 overflow count
constexpr size_t kNoAllocListOffset = 1024;         // u32 per point
constexpr size_t kNoAllocBytes = kNoAllocListOffset + kNoAllocMaxPoints * sizeof(uint32_t);

static __device__ __align__(256) unsigned char g_pim_scratch[kNoAllocBytes];

namespace rs {
namespace {
std::mutex g_scratch_mu;
void* g_scratch_ptr[64] = {};

// Device address of g_pim_scratch on the current device (looked up on first use).
cudaError_t scratch_address(void** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> g(g_scratch_mu);
    if (!g_scratch_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_pim_scratch);
        if (e != cudaSuccess) return e;
        g_scratch_ptr[dev] = p;
    }
    *out = g_scratch_ptr[dev];
    return cudaSuccess;
}
}  // namespace
}  // namespace rs

using namespace rs;

extern "C" int rs_pim_noalloc(const rs_bvh* bvh, const float* d_points, uint64_t n, float dx, float dy, float dz,
                              int32_t* d_obj, uint8_t* d_inside, int filtered, void* stream) {
    if (!bvh || (n && !d_points)) return RS_ERR_INVALID;
    if (n > kNoAllocMaxPoints) return RS_ERR_TOO_LARGE;
    if (n == 0) return RS_OK;
    cudaStream_t s = (cudaStream_t)stream;
    int st = filtered ? bvh_ready(bvh) : RS_OK;
    if (st == RS_OK) st = bvh_use(bvh, s);
    if (st != RS_OK) return st;
    if (filtered && bvh->nV == 0) {
        cudaError_t e = cudaSuccess;
        if (d_obj) e = cudaMemsetAsync(d_obj, 0xff, n * sizeof(int32_t), s);
        if (e == cudaSuccess && d_inside) e = cudaMemsetAsync(d_inside, 0, n, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        return to_status(e);
    }
    void* base = nullptr;
    cudaError_t e = scratch_address(&base);
    if (e != cudaSuccess) return to_status(e);
    unsigned char* sc = static_cast<unsigned char*>(base);
    unsigned long long* meta = reinterpret_cast<unsigned long long*>(sc + kNoAllocMetaOffset);
    uint32_t* ovf = reinterpret_cast<uint32_t*>(sc + kNoAllocListOffset);
    // The array keeps the previous call's contents: the status word and overflow count
    // must start at zero (the list is written before it is read).
    e = cudaMemsetAsync(meta, 0, 2 * sizeof(unsigned long long), s);
    if (e != cudaSuccess) return to_status(e);
    const BoxBounds box = filtered ? make_box(bvh) : BoxBounds{};
    // The column grid is used when it already exists; it is never built here, because
    // building it allocates.  Without it the BVH path gives the same results.
    unsigned long long h[2] = {0, 0};
    return run_pim(pim_axis(dx, dy, dz), bvh, d_points, n, dx, dy, dz, filtered != 0, box, d_obj, d_inside, meta, h,
                   nullptr, ovf, s);
}

extern "C" int rs_pim(const rs_bvh* bvh, const float* d_points, uint64_t n, float dx, float dy, float dz,
                      int32_t* d_obj, uint8_t* d_inside, void* stream) {
    return pim_impl(bvh, d_points, n, dx, dy, dz, d_obj, d_inside, false, (cudaStream_t)stream);
}

extern "C" int rs_pim_filtered(const rs_bvh* bvh, const float* d_points, uint64_t n, float dx, float dy, float dz,
                               int32_t* d_obj, uint8_t* d_inside, void* stream) {
    return pim_impl(bvh, d_points, n, dx, dy, dz, d_obj, d_inside, true, (cudaStream_t)stream);
}

extern "C" int rs_compact_hits(const int32_t* d_obj, uint64_t n, int32_t* d_point_ids, int32_t* d_point_obj,
                               uint64_t capacity, uint64_t* h_count, void* stream) {
    if (!h_count || (n && !d_obj) || n > 0xffffffffull) return RS_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    *h_count = 0;
    if (n == 0) return RS_OK;
    // One tile needs no look-back words; more get theirs and the tile counter zeroed.
    const uint64_t tiles = (n + kHitTile - 1) / kHitTile;
    unsigned long long* words = nullptr;
    cudaError_t e = cudaSuccess;
    if (tiles > 1) {
        e = dmalloc((void**)&words, (tiles + 1) * sizeof(unsigned long long), s);
        if (e == cudaSuccess) e = cudaMemsetAsync(words, 0, (tiles + 1) * sizeof(unsigned long long), s);
    }
    int* slot = pinned_slot_acquire();
    if (!slot && e == cudaSuccess) e = cudaErrorMemoryAllocation;
    if (e == cudaSuccess) {
        slot[0] = slot[1] = 0;
        auto kern = (reinterpret_cast<uintptr_t>(d_obj) & 15u) == 0 ? k_hits<true> : k_hits<false>;
        launch(kern, (unsigned)tiles, kT, 0, s, d_obj, n, d_point_ids, d_point_obj, capacity, words,
               words ? reinterpret_cast<unsigned int*>(words + tiles) : (unsigned int*)nullptr, (volatile int*)slot);
        e = cudaGetLastError();
    }
    if (words) cudaFreeAsync(words, s);
    const cudaError_t e2 = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = e2;
    const uint32_t ht = slot ? (uint32_t)slot[0] : 0;
    const bool gave_up = slot && slot[1] != 0;
    pinned_slot_release(slot);
    if (e != cudaSuccess) return to_status(e);
    if (gave_up) return RS_ERR_ITER_LIMIT;
    *h_count = ht;
    return ht > capacity ? RS_ERR_OUTPUT_OVERFLOW : RS_OK;
}
