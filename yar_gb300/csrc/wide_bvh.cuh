// wide_bvh.cuh - the wide tree that answers a ray first, and the proof that
// its answer is the kd-tree's.
//
// The kd-tree decides what a cast returns: its closest hit is the nearest of
// the triangles in the leaves it visits, the first visited on equal t.  Walking
// it takes about 55 dependent 8-byte node fetches per ray on the 2.4M-triangle
// ray-cast scene, each with little arithmetic, so the walk is bound by
// latency and by idle lanes.  Here a ray first walks an 8-wide tree over the
// same triangles (about 12 nodes of 96 B), then its hit is settled against the
// kd-tree: one descent without a stack to the leaf that holds the hit.
//
// Why the results are the kd-tree's, bit for bit:
//   - triangles are tested with the same arithmetic on the same numbers
//     (watertight_edges on the object-space ray), so every candidate t is the
//     kd-tree's;
//   - a box is skipped only if no triangle inside it can be accepted nearer
//     than the best hit.  The watertight test accepts only when 0 lies in the
//     hull of the three computed sheared points: the signs of its edge
//     functions are exact (a float difference of two products has the exact
//     sign or is 0, and zeros are recomputed in FP64).  With e = 2^-24 and r =
//     reach + |origin|, the computed points are within 8 e r of the exact ones,
//     so the exact ray passes that close to the triangle; the slabs' own
//     arithmetic takes 4 e r more, and they are widened by 20 e r.  The
//     accepted t lies between the vertices' depths along the ray's largest
//     axis up to 11 e r, so only that axis's slab is compared with the best t
//     and with 0 (across the other axes the computed t of a triangle seen
//     edge-on may be far from the crossing);
//   - a node whose triangles all lie in one plane across axis a is skipped when
//     the ray has left that plane behind by more than 20 e r: the computed
//     weights then give sum(w x) within 3 e r of 0 (for triangles with
//     L^2 / h <= reach / 4, longest edge L over height h; the node is not
//     marked otherwise), so the computed t is negative and rejected.  Rays
//     that leave a tessellated wall skip it this way;
//   - a miss of the wide tree is therefore a miss of the kd-tree, which visits
//     no other triangles;
//   - a hit (t, triangle) is the kd-tree's when no other accepted triangle has
//     t' < t (1 + 2^-18) (otherwise the kd-tree walks the ray) and the kd-tree
//     visits a leaf holding the triangle with t_min < t (1 + 2^-19): until it
//     gets there its limit is another hit's t' or tmax, both larger.  The
//     interval with which the kd-tree visits a node depends only on the path
//     from the root (a subtree entered with [a, b] is left with t_max = b), so
//     one descent with the same arithmetic finds it.  The descent begins at the
//     triangle's entry, the deepest node whose cell holds it: with t strictly
//     inside the cell's slabs, computed as the splits are, every split on the
//     way there is decided toward the node (products with 1/d are monotonic
//     in the plane) and its interval is that of the cell's faces;
//   - any hit: an accepted triangle in a visited leaf with t_min < tmax.
// Rays that do not settle, and rays whose numbers the margins above do not
// cover (non-finite, origins beyond 64 x reach, direction components smaller
// than 2^-24 of the largest), walk the kd-tree.
//
// Node, 96 B (three 32-byte blocks, one per axis, each one 256-bit load; the
// ray reads them in the order of its own axes, so nothing is selected by axis):
//   {origin, step, lo bytes 0-3, 4-7, hi bytes 0-3, 4-7, child base, masks}
//   plane(q) = origin + (1 + q / 2^15) step: a byte placed in the mantissa of
//   1.0 is the multiplier (step = 2^15 quantisation steps, a power of two), so
//   a plane costs one byte permute and half a packed FMA.
//   masks: inner children 0-7, leaf children 8-15, of these with two triangles
//   16-23, all triangles below in one plane across x, y, z 24-26.
// Triangle, 64 B: {v0.a, v1.a, v2.a, translation.a} for a = x, y, z, then
//   {triangle, object, flags, primitive}; the triangles of child c of node i are
//   16 i + 2 c and, of a pair, 16 i + 2 c + 1.
// Children sit in the slot of the corner they lie toward; a ray visits the
// slots in the order (slot XOR octant), front to back (the child order of
// Ylitie, Karras and Laine, "Efficient Incoherent Ray Traversal on GPUs Through
// Compressed Wide BVHs", HPG 2017).
#pragma once

#include "device_scene.cuh"

namespace yar {

constexpr int kWideStackSize = 32;            // tree levels a ray can postpone a group on
constexpr float kWideMargin = 1.1920928955078125e-6f;  // 20 * 2^-24
constexpr float kWideNear = 1.f + 3.814697265625e-6f;   // near ties: 2^-18
constexpr float kWideSettle = 1.f + 1.9073486328125e-6f;
constexpr uint32_t kWideNone = 0xffffffffu;
constexpr uint32_t kWideTie = 0x80000000u;   // with a triangle
constexpr uint32_t kWideWalk = 0xfffffffeu;
constexpr uint32_t kWideHolds = 0x80000000u;  // with an entry's node: a leaf that holds the triangle
enum : uint32_t { kWideAlpha = 1u, kWideNoShadow = 2u };  // triangle flags

struct Wide_Block {
    float origin, step;
    uint32_t lo0, lo1, hi0, hi1, base, masks;
};

__device__ __forceinline__ Wide_Block wide_block(const uint4* node, int axis) {
    Wide_Block b;
    uint32_t r0, r1;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r0), "=r"(r1), "=r"(b.lo0), "=r"(b.lo1), "=r"(b.hi0), "=r"(b.hi1), "=r"(b.base), "=r"(b.masks)
        : "l"(node + 2 * axis));
    b.origin = __uint_as_float(r0);
    b.step = __uint_as_float(r1);
    return b;
}

// (x0 * y + c0, x1 * y + c1) in one packed instruction
__device__ __forceinline__ void fma_pair(float x0, float x1, float y, float c0, float c1, float& r0, float& r1) {
    unsigned long long a, b, c, d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(x0), "f"(x1));
    asm("mov.b64 %0, {%1, %1};" : "=l"(b) : "f"(y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(c) : "f"(c0), "f"(c1));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r0), "=f"(r1) : "l"(d));
}

// One axis of a node: the words of the near and far planes and the slab
// constants, t = q * step + near / far.
struct Wide_Axis {
    uint32_t n0, n1, f0, f1;
    float step, near, far;
};

__device__ __forceinline__ Wide_Axis wide_axis(const Wide_Block& b, float o, float inv, float margin) {
    Wide_Axis x;
    const bool negative = inv < 0.f;
    x.n0 = negative ? b.hi0 : b.lo0;
    x.n1 = negative ? b.hi1 : b.lo1;
    x.f0 = negative ? b.lo0 : b.hi0;
    x.f1 = negative ? b.lo1 : b.hi1;
    const float a = b.origin - o;
    x.step = b.step * inv;
    x.near = __fmaf_rn(a, inv, -margin);
    x.far = __fmaf_rn(a, inv, margin);
    return x;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// 1 + q / 2^15 of byte `k` of `word`
__device__ __forceinline__ float wide_plane(uint32_t word, int k) {
    return __uint_as_float(__byte_perm(word, 0x3f800000u, 0x7604u | ((uint32_t)k << 4)));
}

// The traversal of one ray (ANY: stops at the first accepted triangle).
// Axes are the ray's own: z is its largest direction component (Watertight_Ray).
template <bool ANY>
struct Wide_Traversal {
    float ox, oy, oz;  // object-space origin before the object's translation
    float ix, iy, iz;  // 1 / direction (a zero component: a large number)
    float mx, my, mz;  // slab margins in t
    float sx, sy;      // shear; the third factor is iz
    float t;           // closest: best accepted t (tmax without one); any: tmax
    float limit;       // boxes that begin past it are skipped
    uint32_t best;     // triangle of the best hit
    uint32_t base, hits;       // current group: first child; visit-order hits 0-7, inner children by slot 8-15
    uint32_t tri_node, tris;   // node whose leaf children hit; visit-order hits 0-7, pairs 8-15
    uint32_t flags;            // 0-1 kx, 2-3 ky, 4-5 kz, 8-10 octant, 16 near tie
    int sp;
    uint32_t ray;

    __device__ __forceinline__ uint32_t octant() const { return (flags >> 8) & 7u; }
    // what wide_settle takes (after a hit)
    __device__ __forceinline__ uint32_t answer() const { return best | ((flags << 15) & 0x80000000u); }

    // false: the ray is not one that the margins cover
    __device__ __forceinline__ bool begin(const Device_Scene& s, uint32_t index, float3 ro, float3 rd, float tmax) {
        ray = index;
        // transform_ray with an identity linear part, before the translation
        const float3 o = make_float3(1.f * ro.x + 0.f * ro.y + 0.f * ro.z, 0.f * ro.x + 1.f * ro.y + 0.f * ro.z,
                                     0.f * ro.x + 0.f * ro.y + 1.f * ro.z);
        const float3 d = make_float3(1.f * rd.x + 0.f * rd.y + 0.f * rd.z, 0.f * rd.x + 1.f * rd.y + 0.f * rd.z,
                                     0.f * rd.x + 0.f * rd.y + 1.f * rd.z);
        const float far = 64.f * s.wide_reach;
        if (!(fabsf(o.x) <= far && fabsf(o.y) <= far && fabsf(o.z) <= far)) return false;
        const float big = 1073741824.f;  // 2^30
        if (!(fabsf(d.x) <= big && fabsf(d.y) <= big && fabsf(d.z) <= big)) return false;
        const float dmax = fmaxf(fabsf(d.x), fmaxf(fabsf(d.y), fabsf(d.z)));
        const float dmin = dmax * 5.9604645e-8f;
        if (!(dmax >= 9.313226e-10f) || tmax != tmax) return false;
        if ((d.x != 0.f && fabsf(d.x) < dmin) || (d.y != 0.f && fabsf(d.y) < dmin) || (d.z != 0.f && fabsf(d.z) < dmin))
            return false;
        const float3 inv = make_float3(1.f / d.x, 1.f / d.y, 1.f / d.z);
        const Watertight_Ray w = watertight_setup(d, inv);
        ox = sel3(o.x, o.y, o.z, w.kx);
        oy = sel3(o.x, o.y, o.z, w.ky);
        oz = sel3(o.x, o.y, o.z, w.kz);
        const float none = 1.099511627776e12f / dmax;  // 2^40 / dmax
        const float dx = sel3(d.x, d.y, d.z, w.kx), dy = sel3(d.x, d.y, d.z, w.ky);
        ix = dx != 0.f ? sel3(inv.x, inv.y, inv.z, w.kx) : none;
        iy = dy != 0.f ? sel3(inv.x, inv.y, inv.z, w.ky) : none;
        iz = w.sz;
        const float margin = kWideMargin * (s.wide_reach + fmaxf(fabsf(o.x), fmaxf(fabsf(o.y), fabsf(o.z))));
        mx = margin * fabsf(ix);
        my = margin * fabsf(iy);
        mz = margin * fabsf(iz);
        sx = w.sx;
        sy = w.sy;
        t = tmax;
        limit = ANY ? tmax : tmax * kWideNear;
        best = kWideNone;
        base = 0u;
        hits = 0x80u;  // the root: child 0 of a group without inner children
        tris = 0u;
        sp = 0;
        flags = (uint32_t)w.kx | ((uint32_t)w.ky << 2) | ((uint32_t)w.kz << 4) | (d.x > 0.f ? 1u << 8 : 0u) |
                (d.y > 0.f ? 2u << 8 : 0u) | (d.z > 0.f ? 4u << 8 : 0u);
        return true;
    }

    // The next child of the current group: fetch its node, test its children.
    template <class STACK>
    __device__ __forceinline__ void visit(const Device_Scene& s, STACK& stack) {
        const uint32_t oct = octant();
        const int bit = 31 - __clz((int)(hits & 0xffu));
        const uint32_t slot = (uint32_t)bit ^ oct;
        const uint32_t node = base + (uint32_t)__popc((hits >> 8) & ((1u << slot) - 1u));
        hits &= ~(1u << bit);
        if (hits & 0xffu) {
            stack.push(sp, base, __uint_as_float(hits));
            sp++;
        }
        const uint4* p = s.wide_nodes + 6 * (size_t)node;
        const Wide_Block bx = wide_block(p, (int)(flags & 3u));
        const Wide_Block by = wide_block(p, (int)((flags >> 2) & 3u));
        const Wide_Block bz = wide_block(p, (int)((flags >> 4) & 3u));
        const Wide_Axis x = wide_axis(bx, ox, ix, mx), y = wide_axis(by, oy, iy, my), z = wide_axis(bz, oz, iz, mz);
        uint32_t h = 0;
#pragma unroll
        for (int c = 0; c < 8; c++) {  // (bit by bit from the left)
            const int k = c & 3;
            float nx, ny, nz, fx, fy, fz;
            fma_pair(wide_plane(c < 4 ? x.n0 : x.n1, k), wide_plane(c < 4 ? x.f0 : x.f1, k), x.step, x.near, x.far, nx, fx);
            fma_pair(wide_plane(c < 4 ? y.n0 : y.n1, k), wide_plane(c < 4 ? y.f0 : y.f1, k), y.step, y.near, y.far, ny, fy);
            fma_pair(wide_plane(c < 4 ? z.n0 : z.n1, k), wide_plane(c < 4 ? z.f0 : z.f1, k), z.step, z.near, z.far, nz, fz);
            const float tn = max3(nx, ny, nz), tf = min3(fx, fy, fz);
            // missed: the sign of a difference (exact) or of fz
            const uint32_t miss = __float_as_uint(tf - tn) | __float_as_uint(limit - nz) | __float_as_uint(fz);
            h = __funnelshift_l(miss, h, 1);
        }
        h = __brev(h) >> 24 ^ 0xffu;
        h = (h | (h << 8) | 0xff0000u) & bx.masks;  // inner | leaf << 8 | pair << 16, by slot
        // to visit order: bit i of each byte moves to i XOR octant
        if (oct & 1u) h = ((h & 0x555555u) << 1) | ((h >> 1) & 0x555555u);
        if (oct & 2u) h = ((h & 0x333333u) << 2) | ((h >> 2) & 0x333333u);
        if (oct & 4u) h = ((h & 0x0f0f0fu) << 4) | ((h >> 4) & 0x0f0f0fu);
        // every triangle below in one plane across a small axis of the ray, behind it
        const uint32_t flat = bx.masks >> 24;
        if (flat) {
            if (((flat >> (flags & 3u)) & 1u) && __fmaf_rn(wide_plane(x.f0, 0), x.step, x.far) < 0.f) h = 0u;
            if (((flat >> ((flags >> 2) & 3u)) & 1u) && __fmaf_rn(wide_plane(y.f0, 0), y.step, y.far) < 0.f) h = 0u;
        }
        base = bx.base;
        hits = (h & 0xffu) | ((bx.masks & 0xffu) << 8);
        tri_node = node;
        tris = h >> 8;
    }

    __device__ __forceinline__ bool pending() const { return (tris & 0xffu) != 0u; }

    // One pending leaf child, its one or two triangles.  True: the ray is done.
    __device__ __forceinline__ bool test(const Device_Scene& s) {
        const int bit = 31 - __clz((int)(tris & 0xffu));
        const uint32_t first = 16u * tri_node + 2u * ((uint32_t)bit ^ octant());
        const bool pair = (tris >> (8 + bit)) & 1u;
        tris &= ~(1u << bit);
        if (test_triangle(s, first)) return true;
        return pair && test_triangle(s, first + 1u);
    }

    __device__ __forceinline__ bool test_triangle(const Device_Scene& s, uint32_t triangle) {
        const float4* p = s.wide_tris + 4 * (size_t)triangle;
        const float4 X = __ldg(p + (flags & 3u)), Y = __ldg(p + ((flags >> 2) & 3u)), Z = __ldg(p + ((flags >> 4) & 3u));
        const float px = ox + X.w, py = oy + Y.w, pz = oz + Z.w;
        float b0, b1, b2;
        const float th = watertight_edges(X.x - px, Y.x - py, Z.x - pz, X.y - px, Y.y - py, Z.y - pz, X.z - px, Y.z - py,
                                          Z.z - pz, sx, sy, iz, b0, b1, b2);
        if (ANY ? (th >= t) : !(th < limit)) return false;
        if (s.wide_flags) {
            const float4 id = __ldg(p + 3);
            const uint32_t f = __float_as_uint(id.z), object = __float_as_uint(id.y);
            if (ANY && (f & kWideNoShadow)) return false;
            if ((f & kWideAlpha) &&
                alpha_rejects(s, object, __float_as_uint(__ldg(s.objects + 6 * (size_t)object + 4).w) + __float_as_uint(id.x),
                              b0, b1, b2))
                return false;
        }
        if (ANY) {
            best = triangle;
            t = th;
            return true;
        }
        if (th < t) {
            // (every triangle accepted so far is at t or beyond)
            flags = (flags & ~(1u << 16)) | (best != kWideNone && t <= th * kWideNear ? 1u << 16 : 0u);
            best = triangle;
            t = th;
            limit = th * kWideNear;
        } else if (best != kWideNone) {
            flags |= 1u << 16;
        }
        return false;
    }

    // With no triangle pending and the group empty: the group on the stack.
    // False: nothing is left.
    template <class STACK>
    __device__ __forceinline__ bool next_group(STACK& stack) {
        if (hits & 0xffu) return true;
        if (sp == 0) return false;
        sp--;
        const uint2 e = stack.pop(sp);
        base = e.x;
        hits = e.y;
        return true;
    }
};

// Where the kd-tree's descent to a triangle begins, in its mesh's tree and in
// the scene's: the deepest node whose cell holds the triangle, and the cell's
// faces (infinite where no split made one): {lo, node} {hi, -} each.  Where the
// node is a leaf that holds the triangle (kWideHolds, checked when the entry
// was made), a hit inside its interval is settled without reading the tree.

// Whether the kd-tree `nodes`, entered with [t_min, t_max] by the ray (o, 1/d,
// direction sign bits), visits a leaf below `node` that holds primitive `prim`
// with t_min < bound, looked for where the ray is at t.
__device__ __forceinline__ bool kd_visits(const uint2* nodes, uint32_t node, float3 o, float3 inv, uint32_t positive,
                                          float t_min, float t_max, float t, float bound, uint32_t prim) {
    constexpr int kAlternatives = 6;
    uint32_t alt_node[kAlternatives];
    float alt_min[kAlternatives], alt_max[kAlternatives];
    int alternatives = 0;
    const float before = t * (1.f - 7.62939453125e-6f), after = t * (1.f + 7.62939453125e-6f);  // 2^-17
    for (;;) {
        bool leaf = !(bound > t_min);
        if (!leaf) {
            const uint2 n = __ldg(nodes + node);
            leaf = (n.x & 3u) == 3u;
            if (leaf) {
                const uint32_t count = n.x >> 2;
                const uint32_t* list = reinterpret_cast<const uint32_t*>(nodes + node) + 1;
                bool found = count != 0u && n.y == prim;
                for (uint32_t i = 1; i < count && !found; i++) found = __ldg(list + i) == prim;
                if (found) return true;
            } else {
                const int axis = (int)(n.x & 3u);
                const float dist = __uint_as_float(n.y) - sel3(o.x, o.y, o.z, axis);
                const uint32_t below = node + 1, above = n.x >> 2;
                const float t_split = dist * sel3(inv.x, inv.y, inv.z, axis);
                const bool below_first = dist > 0.f;
                // the kd-tree visits only the first side, only the second, or both
                const bool only_first = t_split > t_max || t_split < 0.f;
                const bool only_second = t_split < t_min;
                const bool second = !only_first && (only_second || t_split < before);
                const bool both = !only_first && !only_second && dist != 0.f;
                if (both && !second && !(t_split > after)) {  // the hit lies on the plane: the far side too, if need be
                    if (alternatives == kAlternatives) return false;
                    alt_node[alternatives] = below_first ? above : below;
                    alt_min[alternatives] = t_split;
                    alt_max[alternatives] = t_max;
                    alternatives++;
                }
                t_min = both && second ? t_split : t_min;
                t_max = both && !second ? t_split : t_max;
                const bool to_above = dist != 0.f ? second == below_first : ((positive >> axis) & 1u) != 0u;
                node = to_above ? above : below;
            }
        }
        if (leaf) {
            if (alternatives == 0) return false;
            alternatives--;
            node = alt_node[alternatives];
            t_min = alt_min[alternatives];
            t_max = alt_max[alternatives];
        }
    }
}

// The interval at `entry` of a walk that enters the root with [t_min, t_max];
// false where t is not strictly inside the entry's cell.
__device__ __forceinline__ bool entry_interval(float4 lo, float4 hi, float3 o, float3 inv, float t, float& t_min, float& t_max) {
    float tn = -__int_as_float(0x7f800000), tf = __int_as_float(0x7f800000);
    bool inside = true;
    auto face = [&](float l, float h, float oa, float ia) {
        const float a = (l - oa) * ia, b = (h - oa) * ia;
        const bool parallel = !(fabsf(ia) <= 3.402823466e38f);
        tn = parallel ? tn : fmaxf(tn, fminf(a, b));
        tf = parallel ? tf : fminf(tf, fmaxf(a, b));
        inside = inside && (!parallel || (l < oa && oa < h));
    };
    face(lo.x, hi.x, o.x, inv.x);
    face(lo.y, hi.y, o.y, inv.y);
    face(lo.z, hi.z, o.z, inv.z);
    if (!(inside && tn < fminf(t, t_max) && tf > fmaxf(t, t_min))) return false;
    t_min = fmaxf(t_min, tn);
    t_max = fminf(t_max, tf);
    return true;
}

// The kd-tree's walk of one ray, for rays that the wide tree does not settle
// (added to *walked, if given).
template <bool ANY>
__device__ __noinline__ int kd_walk(const Device_Scene& s, const float4* rays, uint32_t ray, uint32_t* walked, Hit& hit) {
    if (walked) {
        const unsigned here = __activemask();
        if ((int)(threadIdx.x & 31u) == __ffs((int)here) - 1) atomicAdd(walked, (uint32_t)__popc(here));
    }
    const float4 r0 = __ldg(rays + 2 * (size_t)ray), r1 = __ldg(rays + 2 * (size_t)ray + 1);
    Traversal<ANY> tr;
    Local_Stack stack;
    tr.begin(s, ray, make_float3(r0.x, r0.y, r0.z), make_float3(r1.x, r1.y, r1.z), r0.w);
    while (tr.template step<1 << 30>(s, rays, stack)) {
    }
    hit = tr.hit;
    return tr.status();
}

// The wide tree's answer for a ray that may hit (a triangle; with kWideTie
// or kWideWalk for a near tie or a ray it does not cover), settled: the status
// and hit that the kd-tree gives.  A miss (kWideNone) needs no settling.

template <bool ANY>
__device__ __forceinline__ int wide_settle(const Device_Scene& s, const float4* rays, uint32_t ray, uint32_t answer,
                                           uint32_t* walked, Hit& hit) {
    if (!(answer & kWideTie)) {
        const float4 r0 = __ldg(rays + 2 * (size_t)ray), r1 = __ldg(rays + 2 * (size_t)ray + 1);
        const float4* p = s.wide_tris + 4 * (size_t)answer;
        const float4 id = __ldg(p + 3);
        hit.prim = __float_as_uint(id.x);
        hit.object = __float_as_uint(id.y);
        const float3 ro = make_float3(r0.x, r0.y, r0.z), rd = make_float3(r1.x, r1.y, r1.z);
        const float4* q = s.objects + 6 * (size_t)hit.object;
        float3 oo, od;
        transform_ray(__ldg(q), __ldg(q + 1), __ldg(q + 2), ro, rd, oo, od);
        const float4 lo = __ldg(q + 3), hi = __ldg(q + 4);
        const float3 oinv = make_float3(1.f / od.x, 1.f / od.y, 1.f / od.z);
        {
            const Watertight_Ray w = watertight_setup(od, oinv);
            const float4 X = __ldg(p + w.kx), Y = __ldg(p + w.ky), Z = __ldg(p + w.kz);
            const float px = sel3(oo.x, oo.y, oo.z, w.kx), py = sel3(oo.x, oo.y, oo.z, w.ky), pz = sel3(oo.x, oo.y, oo.z, w.kz);
            hit.t = watertight_edges(X.x - px, Y.x - py, Z.x - pz, X.y - px, Y.y - py, Z.y - pz, X.z - px, Y.z - py,
                                     Z.z - pz, w.sx, w.sy, w.sz, hit.b0, hit.b1, hit.b2);
        }
        const float bound = ANY ? r0.w : fminf(hit.t * kWideSettle, r0.w);
        // the mesh's tree, then the scene's; each from the entry, else from the root
        bool visited = hit.t == hit.t;  // (any hit accepts a NaN t: the kd-tree walks that ray)
#pragma unroll 1
        for (int level = 0; level < 2 && visited; level++) {
            const bool mesh = level == 0;
            const float3 o = mesh ? oo : ro, d = mesh ? od : rd;
            const float3 inv = mesh ? oinv : make_float3(1.f / rd.x, 1.f / rd.y, 1.f / rd.z);
            const uint2* nodes = mesh ? s.mesh_nodes + __float_as_uint(lo.w) : s.scene_nodes;
            const float4* entry = s.wide_entries + 4 * (size_t)__float_as_uint(id.w) + (mesh ? 0 : 2);
            const float4 e_lo = __ldg(entry), e_hi = __ldg(entry + 1);
            float r_min, r_max;
            visited = clip_ray_inv(mesh ? make_float3(lo.x, lo.y, lo.z)
                                        : make_float3(s.scene_bounds[0], s.scene_bounds[1], s.scene_bounds[2]),
                                   mesh ? make_float3(hi.x, hi.y, hi.z)
                                        : make_float3(s.scene_bounds[3], s.scene_bounds[4], s.scene_bounds[5]),
                                   o, d, inv, r_min, r_max);
            if (!visited) break;
            float t_min = r_min, t_max = r_max;
            uint32_t node = 0u;
            if (entry_interval(e_lo, e_hi, o, inv, hit.t, t_min, t_max)) {
                node = __float_as_uint(e_lo.w);
                if ((node & kWideHolds) && bound > t_min) continue;  // that leaf: visited
                node &= ~kWideHolds;
            }
            const uint32_t positive = (d.x > 0.f ? 1u : 0u) | (d.y > 0.f ? 2u : 0u) | (d.z > 0.f ? 4u : 0u);
#pragma unroll 1
            for (;;) {
                visited = kd_visits(nodes, node, o, inv, positive, t_min, t_max, hit.t, bound, mesh ? hit.prim : hit.object);
                if (visited || node == 0u) break;
                node = 0u;
                t_min = r_min;
                t_max = r_max;
            }
        }
        if (visited) return 1;
    }
    return kd_walk<ANY>(s, rays, ray, walked, hit);
}

} // namespace yar
