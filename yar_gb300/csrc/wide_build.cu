// wide_build.cu - builds the wide tree of an uploaded scene (wide_bvh.cuh) on
// the device, from the triangles the upload put there.
//
//   bounds   per (object, triangle): the world box (outward rounded), the
//            largest coordinate, the box of the centroids
//   order    48-bit Morton codes of the centroids, radix-sorted (6 passes of
//            8 bits, stable)
//   pairs    bottom-up clustering over the sorted order: every cluster finds
//            the neighbour within kReach places whose union box has the least
//            area, mutual choices merge, the survivors are compacted (parallel
//            locally-ordered clustering, Meister and Bittner, TVCG 2018); after
//            a round that merged few, neighbours in the order are paired; from
//            kSmall clusters on, one block finishes
//   costs    bottom up, which nodes of the pair tree become wide nodes, which
//            joins of two triangles leaf children, by least expected cost
//   collapse level by level, each wide node's children (at most eight)
//   encode   children placed in the slots of the corners they lie toward, boxes
//            quantised outward, triangle slots written
//
// The tree changes no result (the kd-tree settles every hit); its quality
// changes only the number of nodes a ray visits.
#include "context.hpp"
#include "wide_bvh.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

namespace yar {

namespace {

constexpr int kBuildBlock = 256;
constexpr int kReach = 16;    // neighbours searched on either side (8, 32 and 64: the same casts within 2%)
constexpr int kSmall = 1024;  // clusters one block finishes
// A round of merging that takes in fewer than 1/16 of the clusters (2.4M
// triangles merge about 1/6 a round) is followed by one that pairs every two
// neighbours in the order.  Copies of one box, rows of equal cells and boxes
// that grow steadily along the order choose each other one pair a round: 24,000
// triangles of equal cubes in a row were not through after 256 rounds, 11.0 ms;
// their upload now takes 1.9 ms.  (Breaking ties by the lesser XOR of the two
// places, so that equal neighbours pair up by themselves: 1.6 ms, but the
// 4.1M-triangle render takes 74.5 ms on that tree, 73.9 ms on this one.)
constexpr uint32_t kFewMerges = 16;
constexpr uint32_t kInnerBit = 0x80000000u;

constexpr uint32_t kPlanarTriangles = 16384;  // of a scene of tessellated planes (yar_gpu_ctx::wide_planar)

// Of a scene of twins (yar_gpu_ctx::wide_twins): one in this many triangles has one.
constexpr uint32_t kTwinShare = 4;

struct Build_Object {
    uint32_t first;       // of its primitives
    uint32_t tri_offset;  // in the scene's triangle array
    uint32_t node_offset; // of the mesh's kd-tree
    uint32_t object;
    uint32_t flags;       // kWideAlpha, kWideNoShadow
    float cx, cy, cz;     // translation (world to object)
};

struct Build_Totals {
    uint32_t lo[3], hi[3];  // centroid box, order-preserving unsigned
    uint32_t reach;         // bits of a non-negative float
    uint32_t valid;         // primitives in the tree
    uint32_t bad;           // a non-finite coordinate
};

__device__ __forceinline__ uint32_t ordered(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unordered(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__device__ __forceinline__ uint32_t object_of(const Build_Object* objects, uint32_t count, uint32_t prim) {
    uint32_t a = 0, b = count;  // the last object whose first primitive is not past prim
    while (b - a > 1u) {
        const uint32_t m = (a + b) >> 1;
        if (objects[m].first <= prim) a = m;
        else b = m;
    }
    return a;
}

// World box of each primitive (lo.w: 0 when it is not in the tree).
__global__ void __launch_bounds__(kBuildBlock)
wide_bounds_kernel(const float4* __restrict__ tris, const Build_Object* __restrict__ objects, uint32_t object_count,
                   uint32_t prims, float4* __restrict__ lo_out, float4* __restrict__ hi_out, Build_Totals* totals) {
    __shared__ uint32_t s_lo[3], s_hi[3], s_reach, s_valid, s_bad;
    if (threadIdx.x < 3) {
        s_lo[threadIdx.x] = 0xffffffffu;
        s_hi[threadIdx.x] = 0u;
    }
    if (threadIdx.x == 0) s_reach = s_valid = s_bad = 0u;
    __syncthreads();
    const uint32_t i = blockIdx.x * kBuildBlock + threadIdx.x;
    if (i < prims) {
        const Build_Object o = objects[object_of(objects, object_count, i)];
        const float4* p = tris + 3 * ((size_t)o.tri_offset + (i - o.first));
        const float4 v0 = p[0], v1 = p[1], v2 = p[2];
        // object space to world: minus the world-to-object translation
        const float x0 = fminf(v0.x, fminf(v1.x, v2.x)), x1 = fmaxf(v0.x, fmaxf(v1.x, v2.x));
        const float y0 = fminf(v0.y, fminf(v1.y, v2.y)), y1 = fmaxf(v0.y, fmaxf(v1.y, v2.y));
        const float z0 = fminf(v0.z, fminf(v1.z, v2.z)), z1 = fmaxf(v0.z, fmaxf(v1.z, v2.z));
        const float sum = (v0.x + v0.y + v0.z) + (v1.x + v1.y + v1.z) + (v2.x + v2.y + v2.z);
        const bool finite = isfinite(sum);
        const bool valid = finite && v0.w == 0.f;
        const float4 lo = make_float4(__fsub_rd(x0, o.cx), __fsub_rd(y0, o.cy), __fsub_rd(z0, o.cz), valid ? 1.f : 0.f);
        const float ex = v1.x - v0.x, ey = v1.y - v0.y, ez = v1.z - v0.z, gx = v2.x - v0.x, gy = v2.y - v0.y, gz = v2.z - v0.z;
        const float nx = ey * gz - ez * gy, ny = ez * gx - ex * gz, nz = ex * gy - ey * gx;
        const float dx = gx - ex, dy = gy - ey, dz = gz - ez;
        const float longest = sqrtf(fmaxf(ex * ex + ey * ey + ez * ez, fmaxf(gx * gx + gy * gy + gz * gz, dx * dx + dy * dy + dz * dz)));
        const float shape = longest * longest / (sqrtf(nx * nx + ny * ny + nz * nz) / longest);
        const float4 hi = make_float4(__fsub_ru(x1, o.cx), __fsub_ru(y1, o.cy), __fsub_ru(z1, o.cz),
                                      shape >= 0.f ? shape : __int_as_float(0x7f800000));
        lo_out[i] = lo;
        hi_out[i] = hi;
        if (!finite && v0.w == 0.f) atomicOr(&s_bad, 1u);
        if (valid) {
            auto reach3 = [](float r, float a, float b, float c) {
                return fmaxf(r, fmaxf(fabsf(a), fmaxf(fabsf(b), fabsf(c))));
            };
            float r = reach3(0.f, lo.x, lo.y, lo.z);
            r = reach3(r, hi.x, hi.y, hi.z);
            r = reach3(r, x0, y0, z0);
            r = reach3(r, x1, y1, z1);
            r = reach3(r, o.cx, o.cy, o.cz);
            atomicMax(&s_reach, __float_as_uint(r));
            atomicAdd(&s_valid, 1u);
            const float c[3] = {0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z)};
#pragma unroll
            for (int k = 0; k < 3; k++) {
                atomicMin(&s_lo[k], ordered(c[k]));
                atomicMax(&s_hi[k], ordered(c[k]));
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        atomicMin(&totals->lo[threadIdx.x], s_lo[threadIdx.x]);
        atomicMax(&totals->hi[threadIdx.x], s_hi[threadIdx.x]);
    }
    if (threadIdx.x == 0) {
        atomicMax(&totals->reach, s_reach);
        atomicAdd(&totals->valid, s_valid);
        if (s_bad) atomicOr(&totals->bad, 1u);
    }
}

__device__ __forceinline__ uint64_t spread16(uint32_t v) {  // 16 bits, two zeros between
    uint64_t x = v & 0xffffu;
    x = (x | (x << 32)) & 0x00ff00000000ffffull;
    x = (x | (x << 16)) & 0x00ff0000ff0000ffull;
    x = (x | (x << 8)) & 0xf00f00f00f00f00full;
    x = (x | (x << 4)) & 0x30c30c30c30c30c3ull;
    x = (x | (x << 2)) & 0x9249249249249249ull;
    return x;
}

__global__ void __launch_bounds__(kBuildBlock)
wide_morton_kernel(const float4* __restrict__ lo_in, const float4* __restrict__ hi_in, uint32_t prims,
                   const Build_Totals* totals, uint64_t* __restrict__ keys, uint32_t* __restrict__ index) {
    const uint32_t i = blockIdx.x * kBuildBlock + threadIdx.x;
    if (i >= prims) return;
    const float4 lo = lo_in[i], hi = hi_in[i];
    uint64_t key = (1ull << 48) - 1ull;  // primitives outside the tree go last (and are told apart by lo.w)
    if (lo.w != 0.f) {
        const float c[3] = {0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z)};
        uint32_t q[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float a = unordered(totals->lo[k]), b = unordered(totals->hi[k]);
            const float u = b > a ? (c[k] - a) / (b - a) : 0.f;
            q[k] = (uint32_t)fminf(fmaxf(u * 65535.f, 0.f), 65534.f);
        }
        key = spread16(q[0]) | (spread16(q[1]) << 1) | (spread16(q[2]) << 2);
    }
    keys[i] = key;
    index[i] = i;
}

// ---- stable radix sort, 8 bits a pass: per-block digit counts (digit-major),
// their exclusive scan, then each block's ranks
constexpr int kSortItems = 8;
constexpr int kSortTile = kBuildBlock * kSortItems;

__global__ void __launch_bounds__(kBuildBlock)
wide_sort_count_kernel(const uint64_t* __restrict__ keys, uint32_t n, int shift, uint32_t* __restrict__ counts,
                       uint32_t blocks) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t first = blockIdx.x * kSortTile;
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const uint32_t i = first + k * kBuildBlock + threadIdx.x;
        if (i < n) atomicAdd(&h[(uint32_t)(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    counts[threadIdx.x * blocks + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan of n words in place, one block; their sum to *total.
__global__ void __launch_bounds__(1024) wide_scan_kernel(uint32_t* __restrict__ v, uint32_t n, uint32_t* total) {
    __shared__ uint32_t warp_sum[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t base = 0; base < n; base += 1024u * 4u) {
        uint32_t x[4], sum = 0;
        const uint32_t i = base + threadIdx.x * 4u;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            x[k] = i + k < n ? v[i + k] : 0u;
            sum += x[k];
        }
        uint32_t inc = sum;
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += y;
        }
        if (lane == 31) warp_sum[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            uint32_t w = warp_sum[lane];
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, w, d);
                if (lane >= d) w += y;
            }
            warp_sum[lane] = w;
        }
        __syncthreads();
        uint32_t run = carry + (warp ? warp_sum[warp - 1] : 0u) + inc - sum;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (i + k < n) v[i + k] = run;
            run += x[k];
        }
        __syncthreads();
        if (threadIdx.x == 0) carry += warp_sum[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

// Each warp owns kSortTile / 8 consecutive items; the lanes that share a digit
// are ranked by lane, warps and rounds in order, so the pass is stable.
__global__ void __launch_bounds__(kBuildBlock)
wide_sort_scatter_kernel(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ index, uint32_t n, int shift,
                         const uint32_t* __restrict__ offsets, uint32_t blocks, uint64_t* __restrict__ keys_out,
                         uint32_t* __restrict__ index_out) {
    constexpr int kWarps = kBuildBlock / 32;
    __shared__ uint32_t next[kWarps][256];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int d = lane; d < 256; d += 32) next[warp][d] = 0u;
    __syncwarp();
    const uint32_t first = blockIdx.x * kSortTile + warp * (kSortTile / kWarps);
    uint64_t key[kSortItems];
    uint32_t rank[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const uint32_t i = first + k * 32 + lane;
        key[k] = i < n ? keys[i] : ~0ull;
        const uint32_t digit = i < n ? (uint32_t)(key[k] >> shift) & 255u : 256u;
        const uint32_t peers = __match_any_sync(0xffffffffu, digit);
        const uint32_t below = __popc(peers & ((1u << lane) - 1u));
        uint32_t old = 0;
        if (digit < 256u && below == 0) {
            old = next[warp][digit];
            next[warp][digit] = old + __popc(peers);
        }
        old = __shfl_sync(0xffffffffu, old, __ffs(peers) - 1);
        rank[k] = old + below;
        __syncwarp();
    }
    __syncthreads();
    {   // the warps' counts of a digit to its warps' first places
        const int d = threadIdx.x;
        uint32_t run = offsets[d * blocks + blockIdx.x];
        for (int w = 0; w < kWarps; w++) {
            const uint32_t c = next[w][d];
            next[w][d] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const uint32_t i = first + k * 32 + lane;
        if (i >= n) continue;
        const uint32_t to = next[warp][(uint32_t)(key[k] >> shift) & 255u] + rank[k];
        keys_out[to] = key[k];
        index_out[to] = index[i];
    }
}

// ---- clusters: box (lo, hi) and node id (lo.w bits): a primitive, or an inner
// node's index with kInnerBit
// (hi.w: the largest L^2 / h of its triangles, longest edge over height)
struct Cluster {
    float lx, ly, lz, hx, hy, hz;
    uint32_t id;
    float shape;
};

__device__ __forceinline__ Cluster load_cluster(const float4* lo, const float4* hi, uint32_t i) {
    const float4 a = lo[i], b = hi[i];
    return Cluster{a.x, a.y, a.z, b.x, b.y, b.z, __float_as_uint(a.w), b.w};
}
__device__ __forceinline__ Cluster join(const Cluster& a, const Cluster& b) {
    return Cluster{fminf(a.lx, b.lx), fminf(a.ly, b.ly), fminf(a.lz, b.lz),
                   fmaxf(a.hx, b.hx), fmaxf(a.hy, b.hy), fmaxf(a.hz, b.hz), 0u, fmaxf(a.shape, b.shape)};
}
__device__ __forceinline__ float half_area(const Cluster& c) {
    const float x = c.hx - c.lx, y = c.hy - c.ly, z = c.hz - c.lz;
    return x * y + y * z + z * x;
}

__global__ void __launch_bounds__(kBuildBlock)
wide_leaves_kernel(const float4* __restrict__ lo_in, const float4* __restrict__ hi_in, const uint32_t* __restrict__ index,
                   uint32_t n, float4* __restrict__ lo_out, float4* __restrict__ hi_out) {
    const uint32_t i = blockIdx.x * kBuildBlock + threadIdx.x;
    if (i >= n) return;
    const uint32_t p = index[i];
    float4 lo = lo_in[p];
    lo.w = __uint_as_float(p);
    lo_out[i] = lo;
    hi_out[i] = hi_in[p];
}

// The nearest neighbour of each cluster within kReach places: least area of the
// union, the lower place on equal areas (so a least pair is always mutual);
// `pair` pairs neighbours in the order instead.
__global__ void __launch_bounds__(kBuildBlock)
wide_nearest_kernel(const float4* __restrict__ lo, const float4* __restrict__ hi, uint32_t n, bool pair,
                    uint32_t* __restrict__ nearest) {
    if (pair) {
        const uint32_t i = blockIdx.x * kBuildBlock + threadIdx.x;
        if (i < n) nearest[i] = min(i ^ 1u, n - 1u);
        return;
    }
    __shared__ float box[6][kBuildBlock + 2 * kReach];
    const int first = (int)(blockIdx.x * kBuildBlock) - kReach;
    for (int k = threadIdx.x; k < kBuildBlock + 2 * kReach; k += kBuildBlock) {
        const int i = first + k;
        if (i >= 0 && i < (int)n) {
            const float4 a = lo[i], b = hi[i];
            box[0][k] = a.x; box[1][k] = a.y; box[2][k] = a.z;
            box[3][k] = b.x; box[4][k] = b.y; box[5][k] = b.z;
        }
    }
    __syncthreads();
    const uint32_t i = blockIdx.x * kBuildBlock + threadIdx.x;
    if (i >= n) return;
    const int me = threadIdx.x + kReach;
    const Cluster c{box[0][me], box[1][me], box[2][me], box[3][me], box[4][me], box[5][me], 0u, 0.f};
    float best = __int_as_float(0x7f800000);
    uint32_t at = i;
    for (int k = me - kReach; k <= me + kReach; k++) {
        const int j = first + k;
        if (k == me || j < 0 || j >= (int)n) continue;
        const Cluster o{box[0][k], box[1][k], box[2][k], box[3][k], box[4][k], box[5][k], 0u, 0.f};
        const float area = half_area(join(c, o));
        if (area < best) {
            best = area;
            at = (uint32_t)j;
        }
    }
    nearest[i] = at;
}

// 0: merged into its neighbour, 1: stays, 2: takes its neighbour in
__device__ __forceinline__ int fate(const uint32_t* nearest, uint32_t i) {
    const uint32_t j = nearest[i];
    if (j == i || nearest[j] != i) return 1;
    return i < j ? 2 : 0;
}

// Per block: survivors (low half) and merges (high half).
__global__ void __launch_bounds__(kBuildBlock)
wide_count_kernel(const uint32_t* __restrict__ nearest, uint32_t n, uint32_t* __restrict__ stays, uint32_t* __restrict__ merges) {
    const uint32_t i = blockIdx.x * kBuildBlock + threadIdx.x;
    const int f = i < n ? fate(nearest, i) : 0;
    const int s = __syncthreads_count(f != 0), m = __syncthreads_count(f == 2);
    if (threadIdx.x == 0) {
        stays[blockIdx.x] = (uint32_t)s;
        merges[blockIdx.x] = (uint32_t)m;
    }
}

struct Pair_Tree {
    uint2* child;  // per inner node
    float4* lo;    // its box
    float4* hi;
};

__device__ __forceinline__ void store_cluster(float4* lo, float4* hi, uint32_t i, const Cluster& c) {
    lo[i] = make_float4(c.lx, c.ly, c.lz, __uint_as_float(c.id));
    hi[i] = make_float4(c.hx, c.hy, c.hz, c.shape);
}

__device__ __forceinline__ Cluster merge_clusters(const Cluster& a, const Cluster& b, uint32_t inner, const Pair_Tree& t) {
    Cluster c = join(a, b);
    c.id = inner | kInnerBit;
    t.child[inner] = make_uint2(a.id, b.id);
    store_cluster(t.lo, t.hi, inner, c);
    return c;
}

// stays / merges: exclusive scans of wide_count_kernel's counts
__global__ void __launch_bounds__(kBuildBlock)
wide_merge_kernel(const float4* __restrict__ lo, const float4* __restrict__ hi, const uint32_t* __restrict__ nearest,
                  uint32_t n, const uint32_t* __restrict__ stays, const uint32_t* __restrict__ merges, uint32_t inner_base,
                  Pair_Tree tree, float4* __restrict__ lo_out, float4* __restrict__ hi_out) {
    __shared__ uint32_t warp_s[kBuildBlock / 32], warp_m[kBuildBlock / 32];
    const uint32_t i = blockIdx.x * kBuildBlock + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int f = i < n ? fate(nearest, i) : 0;
    const uint32_t s = __ballot_sync(0xffffffffu, f != 0), m = __ballot_sync(0xffffffffu, f == 2);
    if (lane == 0) {
        warp_s[warp] = __popc(s);
        warp_m[warp] = __popc(m);
    }
    __syncthreads();
    if (f == 0) return;
    const uint32_t lower = (1u << lane) - 1u;
    uint32_t to = stays[blockIdx.x] + __popc(s & lower), inner = inner_base + merges[blockIdx.x] + __popc(m & lower);
    for (int w = 0; w < warp; w++) {
        to += warp_s[w];
        inner += warp_m[w];
    }
    Cluster c = load_cluster(lo, hi, i);
    if (f == 2) c = merge_clusters(c, load_cluster(lo, hi, nearest[i]), inner, tree);
    store_cluster(lo_out, hi_out, to, c);
}

// The last kSmall clusters in one block, in shared memory.  root = the last id.
__global__ void __launch_bounds__(kSmall)
wide_finish_kernel(const float4* __restrict__ lo, const float4* __restrict__ hi, uint32_t n, uint32_t inner_base, Pair_Tree tree,
                   uint32_t* root) {
    __shared__ Cluster box[kSmall];
    __shared__ uint32_t nearest[kSmall];
    __shared__ uint32_t warp_s[32], warp_m[32];
    const uint32_t i = threadIdx.x;
    const int lane = i & 31, warp = i >> 5;
    if (i < n) box[i] = load_cluster(lo, hi, i);
    __syncthreads();
    uint32_t inner = inner_base;
    bool pair = false;
    while (n > 1u) {  // each round merges at least the least pair
        if (pair) {
            if (i < n) nearest[i] = min(i ^ 1u, n - 1u);
        } else if (i < n) {
            const Cluster c = box[i];
            float best = __int_as_float(0x7f800000);
            uint32_t at = i;
            const uint32_t from = i > (uint32_t)kReach ? i - kReach : 0u, to = min(n - 1u, i + (uint32_t)kReach);
            for (uint32_t j = from; j <= to; j++) {
                if (j == i) continue;
                const float area = half_area(join(c, box[j]));
                if (area < best) {
                    best = area;
                    at = j;
                }
            }
            nearest[i] = at;
        }
        __syncthreads();
        const int f = i < n ? fate(nearest, i) : 0;
        const uint32_t s = __ballot_sync(0xffffffffu, f != 0), m = __ballot_sync(0xffffffffu, f == 2);
        if (lane == 0) {
            warp_s[warp] = __popc(s);
            warp_m[warp] = __popc(m);
        }
        Cluster c;
        Cluster other;
        if (f != 0) c = box[i];
        if (f == 2) other = box[nearest[i]];
        __syncthreads();
        const uint32_t lower = (1u << lane) - 1u;
        uint32_t to = __popc(s & lower), id = inner + __popc(m & lower), total_s = 0, total_m = 0;
        for (int w = 0; w < 32; w++) {
            if (w == warp) {
                to += total_s;
                id += total_m;
            }
            total_s += warp_s[w];
            total_m += warp_m[w];
        }
        if (f == 2) c = merge_clusters(c, other, id, tree);
        if (f != 0) box[to] = c;
        if (total_m == 0u) break;  // (cannot happen with finite boxes)
        pair = total_m * kFewMerges < n;
        n = total_s;
        inner += total_m;
        __syncthreads();
    }
    if (i == 0) *root = n == 1u ? box[0].id : 0xffffffffu;
}

// ---- collapse: one thread per node of the level; its children, largest first
// opened, go to `children` (pair-tree ids, kWideNone when empty)
__device__ __forceinline__ Cluster node_box(uint32_t id, const Pair_Tree& t, const float4* lo, const float4* hi) {
    const uint32_t i = id & ~kInnerBit;
    return (id & kInnerBit) ? load_cluster(t.lo, t.hi, i) : load_cluster(lo, hi, i);
}

// What becomes of each pair-tree node, by expected cost (surface area
// heuristic; the dynamic programme of Ylitie, Karras and Laine): c(n, i) is the
// least cost of the triangles below n as at most i children of a wide node,
//   c(n, 1) = min(area * 2 kTestCost where n joins two triangles,
//                 area * kVisitCost + d(n, 8)),
//   c(n, i) = min(d(n, i), c(n, i - 1)),  d(n, j) = min over k of c(left, k) + c(right, j - k).
// A choice word holds the k of d(n, j) at bits 3 (j - 2) for j = 2..8 (0: as
// c(n, j - 1)), and kLeafChoice.
// (Opening the largest child until there are eight instead: 4.1M-triangle
// render 96.6 ms, so 92.8; test costs 0.15 to 0.8 of a visit within 1%.)
constexpr float kVisitCost = 1.f, kTestCost = 0.3f;
constexpr uint32_t kLeafChoice = 1u << 24;

__global__ void __launch_bounds__(kBuildBlock)
wide_parents_kernel(Pair_Tree tree, uint32_t inner, uint32_t* __restrict__ prim_parent, uint32_t* __restrict__ inner_parent) {
    const uint32_t i = blockIdx.x * kBuildBlock + threadIdx.x;
    if (i >= inner) return;
    const uint2 c = tree.child[i];
    ((c.x & kInnerBit) ? inner_parent : prim_parent)[c.x & ~kInnerBit] = i;
    ((c.y & kInnerBit) ? inner_parent : prim_parent)[c.y & ~kInnerBit] = i;
}

// One thread per triangle climbs; the second child to arrive computes its parent.
__global__ void __launch_bounds__(kBuildBlock)
wide_costs_kernel(Pair_Tree tree, const float4* __restrict__ prim_lo, const float4* __restrict__ prim_hi,
                  const uint32_t* __restrict__ index, uint32_t n, const uint32_t* __restrict__ prim_parent,
                  const uint32_t* __restrict__ inner_parent, uint32_t root, uint32_t* __restrict__ arrived,
                  float* __restrict__ costs, uint32_t* __restrict__ choice) {
    const uint32_t i = blockIdx.x * kBuildBlock + threadIdx.x;
    if (i >= n) return;
    uint32_t node = prim_parent[index[i]];
    for (;;) {
        __threadfence();
        if (atomicAdd(&arrived[node], 1u) == 0u) return;
        __threadfence();
        const uint2 c = tree.child[node];
        float l[8], r[8];  // [i], 1..7
#pragma unroll
        for (int k = 1; k < 8; k++) {
            l[k] = (c.x & kInnerBit) ? __ldcg(&costs[8 * (size_t)(c.x & ~kInnerBit) + k]) : 0.f;
            r[k] = (c.y & kInnerBit) ? __ldcg(&costs[8 * (size_t)(c.y & ~kInnerBit) + k]) : 0.f;
        }
        if (!(c.x & kInnerBit)) {
            const float a = kTestCost * half_area(load_cluster(prim_lo, prim_hi, c.x));
#pragma unroll
            for (int k = 1; k < 8; k++) l[k] = a;
        }
        if (!(c.y & kInnerBit)) {
            const float a = kTestCost * half_area(load_cluster(prim_lo, prim_hi, c.y));
#pragma unroll
            for (int k = 1; k < 8; k++) r[k] = a;
        }
        float d[9];
        uint32_t word = 0;
#pragma unroll
        for (int j = 2; j <= 8; j++) {
            d[j] = __int_as_float(0x7f800000);
            uint32_t best = 1;
#pragma unroll
            for (int k = 1; k < j; k++) {
                if (k > 7 || j - k > 7) continue;
                const float v = l[k] + r[j - k];
                if (v < d[j]) {
                    d[j] = v;
                    best = (uint32_t)k;
                }
            }
            word |= best << (3 * (j - 2));
        }
        const float area = half_area(load_cluster(tree.lo, tree.hi, node));
        float best = area * kVisitCost + d[8];
        if (!(c.x & kInnerBit) && !(c.y & kInnerBit) && area * 2.f * kTestCost <= best) {
            best = area * 2.f * kTestCost;
            word |= kLeafChoice;
        }
        __stcg(&costs[8 * (size_t)node + 1], best);
#pragma unroll
        for (int j = 2; j < 8; j++) {
            if (d[j] < best) best = d[j];
            else word &= ~(7u << (3 * (j - 2)));
            __stcg(&costs[8 * (size_t)node + j], best);
        }
        choice[node] = word;
        if (node == root) return;
        node = inner_parent[node];
    }
}

__global__ void __launch_bounds__(128)
wide_collapse_kernel(Pair_Tree tree, const uint32_t* __restrict__ choice, const float4* __restrict__ prim_lo,
                     const float4* __restrict__ prim_hi,
                     const uint2* __restrict__ todo, const uint32_t* __restrict__ todo_count, uint2* __restrict__ next,
                     uint32_t* next_count, uint32_t* node_count, uint4* __restrict__ children, uint2* __restrict__ bases) {
    const uint32_t count = *todo_count;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const uint2 item = todo[k];  // pair-tree id, node
        auto is_inner = [&](uint32_t x) { return (x & kInnerBit) && !(choice[x & ~kInnerBit] & kLeafChoice); };
        uint32_t id[8];
        bool open[8];  // an inner child
#pragma unroll
        for (int j = 0; j < 8; j++) {
            id[j] = kWideNone;
            open[j] = false;
        }
        int n = 0;
        auto add = [&](uint32_t x, bool inner_child) {
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (j == n) {
                    id[j] = x;
                    open[j] = inner_child;
                }
            n++;
        };
        if (is_inner(item.x)) {
            // expand d(n, 8): (node, places) still to be placed
            uint32_t todo_node[8], todo_places[8];
            int todo_n = 2;
            {
                const uint32_t w = choice[item.x & ~kInnerBit], k = (w >> 18) & 7u;
                const uint2 c = tree.child[item.x & ~kInnerBit];
                todo_node[0] = c.y;
                todo_places[0] = 8u - k;
                todo_node[1] = c.x;
                todo_places[1] = k;
            }
            while (todo_n > 0) {
                todo_n--;
                const uint32_t x = todo_node[todo_n];
                uint32_t places = todo_places[todo_n];
                if (!(x & kInnerBit)) {
                    add(x, false);
                    continue;
                }
                const uint32_t w = choice[x & ~kInnerBit];
                while (places > 1u && ((w >> (3u * (places - 2u))) & 7u) == 0u) places--;
                if (places == 1u) {
                    add(x, !(w & kLeafChoice));
                    continue;
                }
                const uint32_t k = (w >> (3u * (places - 2u))) & 7u;
                const uint2 c = tree.child[x & ~kInnerBit];
                todo_node[todo_n] = c.y;
                todo_places[todo_n] = places - k;
                todo_node[todo_n + 1] = c.x;
                todo_places[todo_n + 1] = k;
                todo_n += 2;
            }
        } else {
            add(item.x, false);
        }
        uint32_t inner = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) inner += open[j] ? 1u : 0u;
        // inner children get consecutive nodes, in slot order
        const uint32_t base = inner ? atomicAdd(node_count, inner) : 0u;
        const uint32_t at = inner ? atomicAdd(next_count, inner) : 0u;
        // the slot of each child: the corner of the node it lies toward, each
        // slot once, best fit first
        Cluster all{};
        float cx[8], cy[8], cz[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            cx[j] = cy[j] = cz[j] = 0.f;
            if (id[j] == kWideNone) continue;
            const Cluster c = node_box(id[j], tree, prim_lo, prim_hi);
            all = j == 0 ? c : join(all, c);
            cx[j] = c.lx + c.hx;
            cy[j] = c.ly + c.hy;
            cz[j] = c.lz + c.hz;
        }
        const float mx = all.lx + all.hx, my = all.ly + all.hy, mz = all.lz + all.hz;
        uint32_t slot_of = 0xffffffffu;  // 4 bits per child
        uint32_t taken = 0, placed = 0;
        for (int round = 0; round < n; round++) {
            float best = -__int_as_float(0x7f800000);
            int bj = 0, bs = 0;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if (id[j] == kWideNone || ((placed >> j) & 1u)) continue;
                const float dx = cx[j] - mx, dy = cy[j] - my, dz = cz[j] - mz;
                for (int s = 0; s < 8; s++) {
                    if ((taken >> s) & 1u) continue;
                    const float v = ((s & 1) ? dx : -dx) + ((s & 2) ? dy : -dy) + ((s & 4) ? dz : -dz);
                    if (v > best) {
                        best = v;
                        bj = j;
                        bs = s;
                    }
                }
            }
            // (a box so large that its sums are not finite leaves best at -inf: child and slot 0 may
            // then repeat; the first free ones are taken instead)
            if (((placed >> bj) & 1u) || ((taken >> bs) & 1u) || best == -__int_as_float(0x7f800000)) {
                for (bj = 0; (placed >> bj) & 1u; bj++) {
                }
                for (bs = 0; (taken >> bs) & 1u; bs++) {
                }
            }
            placed |= 1u << bj;
            taken |= 1u << bs;
            slot_of = (slot_of & ~(15u << (4 * bj))) | ((uint32_t)bs << (4 * bj));
        }
        uint32_t by_slot[8], inner_slots = 0;
#pragma unroll
        for (int s = 0; s < 8; s++) by_slot[s] = kWideNone;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t s = (slot_of >> (4 * j)) & 15u;
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (id[j] != kWideNone && s == (uint32_t)q) {
                    by_slot[q] = id[j];
                    if (open[j]) inner_slots |= 1u << q;
                }
        }
        children[2 * (size_t)item.y] = make_uint4(by_slot[0], by_slot[1], by_slot[2], by_slot[3]);
        children[2 * (size_t)item.y + 1] = make_uint4(by_slot[4], by_slot[5], by_slot[6], by_slot[7]);
        bases[item.y] = make_uint2(base, inner_slots);
        uint32_t r = 0;
#pragma unroll
        for (int s = 0; s < 8; s++)
            if ((inner_slots >> s) & 1u) {
                next[at + r] = make_uint2(by_slot[s], base + r);
                r++;
            }
    }
}

// ---- encode: one thread per node
__global__ void __launch_bounds__(128)
wide_encode_kernel(Pair_Tree tree, const float4* __restrict__ prim_lo, const float4* __restrict__ prim_hi,
                   const float4* __restrict__ tris, const Build_Object* __restrict__ objects, uint32_t object_count,
                   const uint4* __restrict__ children, const uint2* __restrict__ bases, uint32_t nodes, float reach, uint32_t* flat_triangles,
                   uint4* __restrict__ out, float4* __restrict__ out_tris) {
    const uint32_t node = blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= nodes) return;
    const uint4 c0 = children[2 * (size_t)node], c1 = children[2 * (size_t)node + 1];
    const uint32_t id[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const uint2 base = bases[node];
    uint32_t masks = base.y;
    Cluster box[8];
    Cluster all{};
    bool some = false;
#pragma unroll
    for (int s = 0; s < 8; s++) {
        if (id[s] == kWideNone) continue;
        box[s] = node_box(id[s], tree, prim_lo, prim_hi);
        all = some ? join(all, box[s]) : box[s];
        some = true;
        if (!((base.y >> s) & 1u)) masks |= (id[s] & kInnerBit) ? 0x10100u << s : 0x100u << s;
    }
    if (all.shape <= 0.25f * reach)
        masks |= (all.lx == all.hx ? 1u << 24 : 0u) | (all.ly == all.hy ? 2u << 24 : 0u) | (all.lz == all.hz ? 4u << 24 : 0u);
    if (masks >> 24) atomicAdd(flat_triangles, (uint32_t)(__popc(masks & 0xff00u) + __popc(masks & 0xff0000u)));
#pragma unroll
    for (int axis = 0; axis < 3; axis++) {
        const float lo = axis == 0 ? all.lx : (axis == 1 ? all.ly : all.lz);
        const float hi = axis == 0 ? all.hx : (axis == 1 ? all.hy : all.hz);
        // step q (2^k) and origin so that every plane, 1/16 of a step outward, fits 0..255
        int k = -100;
        if (hi > lo) k = max(k, ilogbf(hi - lo) - 8);
        const float away = fmaxf(fabsf(lo), fabsf(hi));
        if (away > 0.f) k = max(k, ilogbf(away) - 40);
        float origin = 0.f;
        double grid = 0.0, q = 0.0;
        for (;; k++) {
            q = ldexp(1.0, k);
            origin = __double2float_rd((double)lo - q * 0.0625 - 32768.0 * q);
            grid = (double)origin + 32768.0 * q;
            if (ceil(((double)hi - grid) / q + 0.0625) <= 255.0) break;
        }
        uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int s = 0; s < 8; s++) {
            uint32_t a = 255u, b = 0u;  // an empty slot; of a flat axis, the plane (visit reads slot 0's)
            if (id[s] != kWideNone || lo == hi) {
                const double l = lo == hi ? lo : axis == 0 ? box[s].lx : (axis == 1 ? box[s].ly : box[s].lz);
                const double h = lo == hi ? hi : axis == 0 ? box[s].hx : (axis == 1 ? box[s].hy : box[s].hz);
                a = (uint32_t)fmin(fmax(floor((l - grid) / q - 0.0625), 0.0), 255.0);
                b = (uint32_t)fmin(fmax(ceil((h - grid) / q + 0.0625), 0.0), 255.0);
            }
            w[s >> 2] |= a << (8 * (s & 3));
            w[2 + (s >> 2)] |= b << (8 * (s & 3));
        }
        uint4* p = out + 6 * (size_t)node + 2 * axis;
        p[0] = make_uint4(__float_as_uint(origin), __float_as_uint((float)(32768.0 * q)), w[0], w[1]);
        p[1] = make_uint4(w[2], w[3], base.x, masks);
    }
    for (int s = 0; s < 8; s++) {
        if (!((masks >> (8 + s)) & 1u)) continue;
        uint2 leaf = make_uint2(id[s], kWideNone);
        if (id[s] & kInnerBit) leaf = tree.child[id[s] & ~kInnerBit];
        for (int k = 0; k < 2; k++) {
            const uint32_t which = k == 0 ? leaf.x : leaf.y;
            if (which == kWideNone) continue;
            const Build_Object o = objects[object_of(objects, object_count, which)];
            const uint32_t prim = which - o.first;
            const float4* p = tris + 3 * ((size_t)o.tri_offset + prim);
            const float4 v0 = p[0], v1 = p[1], v2 = p[2];
            float4* t = out_tris + 4 * (16 * (size_t)node + 2 * s + k);
            t[0] = make_float4(v0.x, v1.x, v2.x, o.cx);
            t[1] = make_float4(v0.y, v1.y, v2.y, o.cy);
            t[2] = make_float4(v0.z, v1.z, v2.z, o.cz);
            t[3] = make_float4(__uint_as_float(prim), __uint_as_float(o.object), __uint_as_float(o.flags), __uint_as_float(which));
        }
    }
}

// ---- twins: triangles with the vertices of another one, in any order (faces
// modelled twice, an object placed twice).  Twins have one Morton code; those
// further than kReach places apart among equal codes are not found.
__device__ __forceinline__ bool same_vertices(const float4* a, const float4* b) {
    uint32_t found = 0;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
            if (a[i].x == b[j].x && a[i].y == b[j].y && a[i].z == b[j].z) found |= 1u << i | 8u << j;
    return found == 63u;
}

__global__ void __launch_bounds__(kBuildBlock)
wide_twins_kernel(const float4* __restrict__ prim_lo, const float4* __restrict__ prim_hi, const uint32_t* __restrict__ index,
                  uint32_t n, const float4* __restrict__ tris, const Build_Object* __restrict__ objects, uint32_t object_count,
                  uint32_t* twins) {
    __shared__ float box[6][kBuildBlock + kReach];
    const uint32_t first = blockIdx.x * kBuildBlock;
    for (uint32_t k = threadIdx.x; k < kBuildBlock + kReach; k += kBuildBlock)
        if (first + k < n) {
            const uint32_t p = index[first + k];
            const float4 a = prim_lo[p], b = prim_hi[p];
            box[0][k] = a.x; box[1][k] = a.y; box[2][k] = a.z;
            box[3][k] = b.x; box[4][k] = b.y; box[5][k] = b.z;
        }
    __syncthreads();
    const uint32_t me = threadIdx.x, i = first + me;
    bool twin = false;  // of a triangle further on
    for (uint32_t k = me + 1; k <= me + (uint32_t)kReach && first + k < n && !twin; k++) {
        bool same = true;
#pragma unroll
        for (int c = 0; c < 6; c++) same = same && box[c][k] == box[c][me];
        if (!same) continue;
        const uint32_t p = index[i], q = index[first + k];
        const Build_Object a = objects[object_of(objects, object_count, p)], b = objects[object_of(objects, object_count, q)];
        twin = a.cx == b.cx && a.cy == b.cy && a.cz == b.cz &&
               same_vertices(tris + 3 * ((size_t)a.tri_offset + (p - a.first)), tris + 3 * ((size_t)b.tri_offset + (q - b.first)));
    }
    const int found = __syncthreads_count(twin);
    if (threadIdx.x == 0 && found) atomicAdd(twins, (uint32_t)found);
}

// ---- entries: the deepest kd-tree node whose cell holds a box (a box that
// ends at a split belongs to the side it lies on), and whether that node is a
// leaf that holds primitive `prim`
__device__ __forceinline__ void write_entry(const uint2* nodes, float3 lo, float3 hi, uint32_t prim, float4* out) {
    const float inf = __int_as_float(0x7f800000);
    float c_lo[3] = {-inf, -inf, -inf}, c_hi[3] = {inf, inf, inf};
    uint32_t node = 0, holds = 0;
    for (;;) {  // (child indices increase: the upload checked the links)
        const uint2 n = nodes[node];
        const int axis = (int)(n.x & 3u);
        if (axis == 3) {
            const uint32_t* list = reinterpret_cast<const uint32_t*>(nodes + node) + 1;
            for (uint32_t i = 0; i < (n.x >> 2); i++)
                if (list[i] == prim) holds = kWideHolds;
            break;
        }
        const float split = __uint_as_float(n.y);
        const float a = sel3(lo.x, lo.y, lo.z, axis), b = sel3(hi.x, hi.y, hi.z, axis);
        const bool below = b <= split && a < split, above = a >= split && b > split;
        if (!below && !above) break;
#pragma unroll
        for (int k = 0; k < 3; k++)
            if (k == axis) {
                if (below) c_hi[k] = split;
                else c_lo[k] = split;
            }
        node = below ? node + 1 : n.x >> 2;
    }
    out[0] = make_float4(c_lo[0], c_lo[1], c_lo[2], __uint_as_float(node | holds));
    out[1] = make_float4(c_hi[0], c_hi[1], c_hi[2], 0.f);
}

__global__ void __launch_bounds__(kBuildBlock)
wide_entries_kernel(const float4* __restrict__ tris, const uint2* __restrict__ mesh_nodes, const uint2* __restrict__ scene_nodes,
                    const Build_Object* __restrict__ objects, uint32_t object_count, uint32_t prims, float4* __restrict__ out) {
    const uint32_t i = blockIdx.x * kBuildBlock + threadIdx.x;
    if (i >= prims) return;
    const Build_Object o = objects[object_of(objects, object_count, i)];
    const float4* p = tris + 3 * ((size_t)o.tri_offset + (i - o.first));
    const float4 v0 = p[0], v1 = p[1], v2 = p[2];
    const float3 lo = make_float3(fminf(v0.x, fminf(v1.x, v2.x)), fminf(v0.y, fminf(v1.y, v2.y)), fminf(v0.z, fminf(v1.z, v2.z)));
    const float3 hi = make_float3(fmaxf(v0.x, fmaxf(v1.x, v2.x)), fmaxf(v0.y, fmaxf(v1.y, v2.y)), fmaxf(v0.z, fmaxf(v1.z, v2.z)));
    write_entry(mesh_nodes + o.node_offset, lo, hi, i - o.first, out + 4 * (size_t)i);
    write_entry(scene_nodes, make_float3(lo.x - o.cx, lo.y - o.cy, lo.z - o.cz), make_float3(hi.x - o.cx, hi.y - o.cy, hi.z - o.cz),
                o.object, out + 4 * (size_t)i + 2);
}

// The build's device memory, one allocation, freed on every way out: laid out
// once without a base to learn its size, then again from it.
struct Scratch {
    unsigned char* base = nullptr;
    size_t used = 0;
    template <class T>
    T* take(size_t n) {
        used = (used + 255) & ~(size_t)255;
        T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
        used += n * sizeof(T);
        return p;
    }
    bool allocate() {
        void* p = nullptr;
        if (cudaMalloc(&p, used) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        base = static_cast<unsigned char*>(p);
        used = 0;
        return true;
    }
    ~Scratch() {
        if (base) cudaFree(base);
    }
};

bool identity_linear_part(const float* m) {
    const float want[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++) {
            uint32_t a, b;
            memcpy(&a, &m[4 * r + c], 4);
            memcpy(&b, &want[3 * r + c], 4);
            if (a != b) return false;
        }
    return true;
}

} // namespace

void wide_release(yar_gpu_ctx* ctx) {
    device_free(ctx->wide_nodes);
    device_free(ctx->wide_tris);
    device_free(ctx->wide_entries);
    ctx->ds.wide_nodes = nullptr;
    ctx->ds.wide_tris = nullptr;
    ctx->ds.wide_entries = nullptr;
    ctx->ds.wide_reach = 0.f;
    ctx->ds.wide_flags = 0u;
    ctx->wide_planar = ctx->wide_twins = false;
}

// Scenes without a wide tree (and every cast of theirs) use the kd-tree
// kernels: an object whose transform is more than a translation (the world
// boxes would have to cover the rounding of its linear part), coordinates
// beyond 2^30 or all below 2^-30, a tree too deep for the stack, no memory.
cudaError_t wide_build(yar_gpu_ctx* ctx, const yar_flat_scene* scene, const uint32_t* tri_offset, const uint32_t* node_offset) {
    wide_release(ctx);
    std::vector<Build_Object> objects;
    uint64_t prims64 = 0;
    uint32_t any_flags = 0;
    for (uint32_t i = 0; i < scene->object_count; i++) {
        const yar_object_desc& o = scene->objects[i];
        const yar_mesh_desc& mesh = scene->meshes[o.mesh_index];
        if (mesh.visibility == YAR_INVISIBLE) continue;
        const float* w = o.world_to_object;
        if (!identity_linear_part(w) || !std::isfinite(w[3]) || !std::isfinite(w[7]) || !std::isfinite(w[11]))
            return cudaSuccess;
        Build_Object b;
        b.first = (uint32_t)prims64;
        b.tri_offset = tri_offset[o.mesh_index];
        b.node_offset = node_offset[o.mesh_index];
        b.object = i;
        b.flags = (mesh.alpha_texture ? (uint32_t)kWideAlpha : 0u) |
                  (mesh.visibility != YAR_VISIBLE ? (uint32_t)kWideNoShadow : 0u);
        b.cx = w[3];
        b.cy = w[7];
        b.cz = w[11];
        any_flags |= b.flags;
        objects.push_back(b);
        prims64 += mesh.triangle_count;
        if (prims64 > (1u << 26)) return cudaSuccess;
    }
    if (prims64 == 0) return cudaSuccess;
    const uint32_t prims = (uint32_t)prims64;
    cudaStream_t st = ctx->stream;
    const uint32_t blocks = (prims + kBuildBlock - 1) / kBuildBlock;
    const uint32_t sort_blocks = (prims + kSortTile - 1) / kSortTile;

    Build_Object* d_objects;
    Build_Totals* d_totals;
    float4 *prim_lo, *prim_hi, *clusters;
    uint64_t* keys[2];
    uint32_t *index[2], *counts, *parents[2], *choice, *words;
    Pair_Tree tree;
    uint4* children;
    uint2* bases;  // first child node, inner slots
    Scratch S;
    for (int pass = 0; pass < 2; pass++) {
        if (pass == 1 && !S.allocate()) return cudaSuccess;
        d_objects = S.take<Build_Object>(objects.size());
        d_totals = S.take<Build_Totals>(1);
        prim_lo = S.take<float4>(prims);
        prim_hi = S.take<float4>(prims);
        for (int k = 0; k < 2; k++) {
            keys[k] = S.take<uint64_t>(prims);
            index[k] = S.take<uint32_t>(prims);
            parents[k] = S.take<uint32_t>(prims);
        }
        counts = S.take<uint32_t>(std::max<size_t>(256 * (size_t)sort_blocks, 2 * (size_t)blocks));
        clusters = S.take<float4>(4 * (size_t)prims);  // later the costs, 32 B per inner node
        tree.child = S.take<uint2>(prims);
        tree.lo = S.take<float4>(prims);
        tree.hi = S.take<float4>(prims);
        children = S.take<uint4>(2 * (size_t)prims);
        bases = S.take<uint2>(prims);
        choice = S.take<uint32_t>(prims);
        words = S.take<uint32_t>(kWideStackSize + 4);
    }
    float4* c_lo[2] = {clusters, clusters + prims};
    float4* c_hi[2] = {clusters + 2 * (size_t)prims, clusters + 3 * (size_t)prims};

    Build_Totals totals{{~0u, ~0u, ~0u}, {0u, 0u, 0u}, 0u, 0u, 0u};
    cudaError_t e = cudaMemcpyAsync(d_objects, objects.data(), objects.size() * sizeof(Build_Object), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_totals, &totals, sizeof(totals), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    const float4* tris = (const float4*)ctx->tris.ptr;
    const uint32_t n_objects = (uint32_t)objects.size();
    wide_bounds_kernel<<<blocks, kBuildBlock, 0, st>>>(tris, d_objects, n_objects, prims, prim_lo, prim_hi, d_totals);
    wide_morton_kernel<<<blocks, kBuildBlock, 0, st>>>(prim_lo, prim_hi, prims, d_totals, keys[0], index[0]);
    int cur = 0;
    for (int shift = 0; shift < 48; shift += 8, cur ^= 1) {
        wide_sort_count_kernel<<<sort_blocks, kBuildBlock, 0, st>>>(keys[cur], prims, shift, counts, sort_blocks);
        wide_scan_kernel<<<1, 1024, 0, st>>>(counts, 256u * sort_blocks, words);
        wide_sort_scatter_kernel<<<sort_blocks, kBuildBlock, 0, st>>>(keys[cur], index[cur], prims, shift, counts, sort_blocks,
                                                                      keys[cur ^ 1], index[cur ^ 1]);
    }
    e = cudaMemcpyAsync(&totals, d_totals, sizeof(totals), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    float reach;
    memcpy(&reach, &totals.reach, 4);
    if (totals.valid == 0u || totals.bad || !(reach <= 1073741824.f) || !(reach >= 9.313226e-10f)) return cudaSuccess;
    uint32_t n = totals.valid;
    wide_leaves_kernel<<<(n + kBuildBlock - 1) / kBuildBlock, kBuildBlock, 0, st>>>(prim_lo, prim_hi, index[cur], n, c_lo[0], c_hi[0]);
    uint32_t inner = 0;
    int side = 0;
    uint32_t* nearest = index[cur ^ 1];
    bool pair = false;
    while (n > (uint32_t)kSmall) {
        const uint32_t b = (n + kBuildBlock - 1) / kBuildBlock;
        wide_nearest_kernel<<<b, kBuildBlock, 0, st>>>(c_lo[side], c_hi[side], n, pair, nearest);
        wide_count_kernel<<<b, kBuildBlock, 0, st>>>(nearest, n, counts, counts + blocks);
        wide_scan_kernel<<<1, 1024, 0, st>>>(counts, b, words);
        wide_scan_kernel<<<1, 1024, 0, st>>>(counts + blocks, b, words + 1);
        uint32_t sums[2];
        e = cudaMemcpyAsync(sums, words, sizeof(sums), cudaMemcpyDeviceToHost, st);
        wide_merge_kernel<<<b, kBuildBlock, 0, st>>>(c_lo[side], c_hi[side], nearest, n, counts, counts + blocks, inner, tree,
                                                     c_lo[side ^ 1], c_hi[side ^ 1]);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
        const uint32_t stays = sums[0], merged = sums[1];
        if (merged == 0u) return cudaSuccess;  // (cannot happen with finite boxes)
        pair = (uint64_t)merged * kFewMerges < n;
        n = stays;
        inner += merged;
        side ^= 1;
    }
    // words: [0] root, [1] nodes, [2 + level] the level's nodes
    e = cudaMemsetAsync(words, 0, (kWideStackSize + 4) * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    wide_finish_kernel<<<1, kSmall, 0, st>>>(c_lo[side], c_hi[side], n, inner, tree, words);
    uint32_t root = 0;
    e = cudaMemcpyAsync(&root, words, 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    if (root == 0xffffffffu) return cudaSuccess;
    uint2* todo[2] = {reinterpret_cast<uint2*>(keys[0]), reinterpret_cast<uint2*>(keys[1])};
    const uint2 first = make_uint2(root, 0u);
    const uint32_t inner_count = totals.valid - 1u;
    if (inner_count) {
        const uint32_t inner_blocks = (inner_count + kBuildBlock - 1) / kBuildBlock;
        uint32_t* arrived = nearest;  // (the merging is done)
        e = cudaMemsetAsync(arrived, 0, (size_t)inner_count * sizeof(uint32_t), st);
        if (e != cudaSuccess) return e;
        wide_parents_kernel<<<inner_blocks, kBuildBlock, 0, st>>>(tree, inner_count, parents[0], parents[1]);
        wide_costs_kernel<<<(totals.valid + kBuildBlock - 1) / kBuildBlock, kBuildBlock, 0, st>>>(
            tree, prim_lo, prim_hi, index[cur], totals.valid, parents[0], parents[1], root & ~kInnerBit, arrived,
            reinterpret_cast<float*>(c_lo[0]), choice);
    }
    uint32_t h_words[kWideStackSize + 4] = {};
    h_words[1] = 1u;
    h_words[2] = 1u;
    e = cudaMemcpyAsync(todo[0], &first, sizeof(first), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(words, h_words, sizeof(h_words), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    // eight levels at a time (a level without nodes ends at its count), until one has none
    const uint32_t level_grid = std::min<uint32_t>((prims + 127u) / 128u, 152u * 8u);
    for (int level = 0; level < kWideStackSize && h_words[2 + level] != 0u;) {
        for (const int end = level + 8; level < end; level++)
            wide_collapse_kernel<<<level_grid, 128, 0, st>>>(tree, choice, prim_lo, prim_hi, todo[level & 1], words + 2 + level,
                                                             todo[(level & 1) ^ 1], words + 3 + level, words + 1, children,
                                                             bases);
        e = cudaMemcpyAsync(h_words, words, sizeof(h_words), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e == cudaSuccess) e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (h_words[2 + kWideStackSize] != 0u) return cudaSuccess;  // deeper than the stack
    const uint32_t nodes = h_words[1];
    if (device_alloc(ctx, ctx->wide_nodes, 96 * (size_t)nodes) != YAR_OK ||
        device_alloc(ctx, ctx->wide_tris, 1024 * (size_t)nodes) != YAR_OK ||
        device_alloc(ctx, ctx->wide_entries, 64 * (size_t)prims) != YAR_OK) {
        wide_release(ctx);
        return cudaSuccess;
    }
    e = cudaMemsetAsync(words, 0, 2 * sizeof(uint32_t), st);  // triangles of flat nodes, twins
    if (e != cudaSuccess) return e;
    wide_twins_kernel<<<(totals.valid + kBuildBlock - 1) / kBuildBlock, kBuildBlock, 0, st>>>(
        prim_lo, prim_hi, index[cur], totals.valid, tris, d_objects, n_objects, words + 1);
    wide_encode_kernel<<<(nodes + 127u) / 128u, 128, 0, st>>>(tree, prim_lo, prim_hi, tris, d_objects, n_objects, children, bases,
                                                              nodes, reach, words, (uint4*)ctx->wide_nodes.ptr, (float4*)ctx->wide_tris.ptr);
    wide_entries_kernel<<<blocks, kBuildBlock, 0, st>>>(tris, (const uint2*)ctx->mesh_nodes.ptr, (const uint2*)ctx->scene_nodes.ptr,
                                                        d_objects, n_objects, prims, (float4*)ctx->wide_entries.ptr);
    e = cudaGetLastError();
    uint32_t found[2] = {0u, 0u};
    if (e == cudaSuccess) e = cudaMemcpyAsync(found, words, sizeof(found), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    ctx->wide_planar = found[0] >= kPlanarTriangles && found[0] > totals.valid / 2u;
    ctx->wide_twins = 2ull * found[1] * kTwinShare > totals.valid;  // (of two, one was counted)
    ctx->ds.wide_entries = (const float4*)ctx->wide_entries.ptr;
    ctx->ds.wide_nodes = (const uint4*)ctx->wide_nodes.ptr;
    ctx->ds.wide_tris = (const float4*)ctx->wide_tris.ptr;
    ctx->ds.wide_reach = reach;
    ctx->ds.wide_flags = any_flags;
    return cudaSuccess;
}

} // namespace yar
