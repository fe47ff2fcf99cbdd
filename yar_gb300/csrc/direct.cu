// direct.cu - the reference's direct-lighting algorithm on the device
// (estimate_direct_lighting, src/ref/direct_lighting.cpp:415-520; render_scene's
// pixel loop, src/ref/reference_renderer.cpp:331-409).
//
// Per sample: the camera ray, then at its hit every point and directional
// light, every rectangular and sphere light over its k x k sample arrays, the
// environment light over its sample count, and the delta ray of a delta
// event.  The sample arrays are extra rows of the sample tables (2D array
// grids before 1D ones, as Stratified_Pixel_Sampler::next_pixel draws them).
// The draws past the tables (the scattering-type sample, the environment's
// light and BSDF samples) come from the pixel's pcg stream in sample order; a
// sample's share of them depends on what its camera ray hit, so the camera
// rays and the per-pixel prefix of their draw counts come first.
//
// What a sample adds up is a list of units, the same for every sample: a
// point or directional light, or one element of an area or environment
// light's samples (a light sample and a BSDF sample).  No unit needs another
// one's result, so a chunk of samples runs through a few kernels, each with
// one thread per (sample, unit): the light samples' shadow rays and the BSDF
// samples' probe rays go into queues with what they contribute if they
// arrive, the cast kernels (cast.cu) trace the queues, and one thread per
// sample then adds the contributions in the reference's order.
//
// The rays bound it: 10 per sample and a few hundred instructions for each.
// The Cornell box with a quad light of 4 samples, two delta lights and a spot,
// 512 x 512 samples of 16: 5.7 ms, of which the casts and their settling take
// 40%, the light and BSDF samples 35%.  One kernel that walked through a
// sample's units and traced their rays inline through the kd-tree took 25 ms
// (28 ms in all): at 230 registers 12% of the warps were resident, and lanes
// whose light sample was not worth a ray waited for those that traced one.
#include "wavefront.cuh"

namespace yar {

namespace {

// Samples in flight per chunk, and rays per queue of a launch.  Both bound
// memory: 240 B per sample (textured: 440 B) and 146 B per ray slot, 3.4 GB at
// the full size.  512 x 512 samples of 16: 6.2 ms as one chunk, 6.5 ms at half
// and 7.0 ms at a quarter of both (more launches, shorter queues).
constexpr uint64_t kDirectPaths = 4u << 20;
constexpr uint64_t kDirectRaySlots = 16u << 20;
// The two sampling kernels wait on loads and instruction fetches more than
// they issue: at 64 registers (8 blocks per SM, up to 88 B spilled) the render
// took 6.04 ms against 6.32 ms without the bound.
constexpr int kDirectBlocks = 8;
constexpr uint32_t kMaxUnits = 4096;  // units per launch (gridDim.y)
constexpr size_t kDirectBuffers = 33;

enum { kUnitNoSamples = 0, kUnitDelta, kUnitRect, kUnitSphere, kUnitEnvironment };

// One summand of every sample, in the order in which they are added.
struct Direct_Unit {
    int32_t kind, light;
    int32_t element, side;  // element of the side x side array (environment: of the sample count)
    int32_t grid2, grid1;   // the light's first 2D and 1D array grid
    int32_t count;          // elements of the light
    int32_t pad;
};

// What a sample keeps between the kernels (SoA over the chunk's samples).
// info: bit 0 lights are summed, bit 1 a delta ray, bit 2 the shading normal
// was flipped, then the material index.
constexpr uint32_t kLit = 1u, kDeltaRay = 2u, kFlipped = 4u;
struct Direct_State {
    uint32_t paths;
    uint32_t* info;
    float* shading;      // 21 rows: Shading's vectors
    uint32_t* bsdf;      // rows of Bsdf words (textured scenes: the textures are looked up once)
    uint4* rng;          // the pcg state behind the scattering-type sample
    float4* L;           // the sum so far
    float4* L2;          // a light's sum so far
    float4* delta;       // the delta ray's attenuation, then what it adds
    // per (unit, sample)
    float4* contrib;     // light sample: contribution if unoccluded, w = 1 if there is a ray
    uint8_t* occluded;   // its shadow ray's answer; second half: the environment's BSDF samples
    float4* probe;       // BSDF sample: Le * f, pdf (sphere and environment lights: the contribution)
    float2* probe2;      // cosine at the light (0: no ray), |cosine| here with the sign bit if the
                         // ray starts on the far side of the normal
    float4* hit4;        // the probe's hit
    uint2* hit2;
    // queues
    float4* shd_rays;
    uint32_t* shd_slot;
    float4* prb_rays;
    uint32_t* prb_slot;
    uint32_t* counters;  // [0] delta rays, [1] shadow, [2] probe
};

__device__ __forceinline__ void store_shading(const Direct_State& D, uint32_t i, const Shading& sc) {
    const V3 v[7] = {sc.wo, sc.position, sc.ng, sc.n, sc.dpdu_shading, sc.origin_pos, sc.origin_neg};
#pragma unroll
    for (int k = 0; k < 7; k++) {
        float* row = D.shading + (size_t)(3 * k) * D.paths + i;
        row[0] = v[k].x;
        row[D.paths] = v[k].y;
        row[2 * (size_t)D.paths] = v[k].z;
    }
}
__device__ __forceinline__ V3 load_vector(const Direct_State& D, uint32_t i, int k) {
    const float* row = D.shading + (size_t)(3 * k) * D.paths + i;
    return v3(__ldg(row), __ldg(row + D.paths), __ldg(row + 2 * (size_t)D.paths));
}
__device__ __forceinline__ void load_shading(const Direct_State& D, uint32_t i, uint32_t info, Shading& sc) {
    sc.wo = load_vector(D, i, 0);
    sc.position = load_vector(D, i, 1);
    sc.ng = load_vector(D, i, 2);
    sc.n = load_vector(D, i, 3);
    sc.dpdu_shading = load_vector(D, i, 4);
    sc.origin_pos = load_vector(D, i, 5);
    sc.origin_neg = load_vector(D, i, 6);
    sc.flipped = (info & kFlipped) != 0;
}
constexpr int kBsdfWords = sizeof(Bsdf) / 4;
static_assert(sizeof(Bsdf) % 4 == 0, "stored by words");
// The sample's BSDF: made again from its shading, or as stored.
template <bool TEXTURED>
__device__ __forceinline__ void load_bsdf(const Scene_Dev& S, const Direct_State& D, uint32_t i, uint32_t info,
                                          const Shading& sc, Bsdf& f) {
    if constexpr (TEXTURED) {
        uint32_t w[kBsdfWords];
        for (int k = 0; k < kBsdfWords; k++) w[k] = __ldg(D.bsdf + (size_t)k * D.paths + i);
        memcpy(&f, w, sizeof(Bsdf));
    } else {
        make_bsdf(sc, S.materials[info >> 3], S.materials, f);
    }
}

// Queue append by the whole block, one atomic per block and queue; every
// thread of the block calls it.
__device__ __forceinline__ uint32_t block_append(uint32_t* counter, bool want) {
    __shared__ uint32_t warp_base[kBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned mask = __ballot_sync(0xffffffffu, want);
    if (lane == 0) warp_base[warp] = (uint32_t)__popc(mask);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t total = 0;
        for (int k = 0; k < kBlock / 32; k++) {
            const uint32_t c = warp_base[k];
            warp_base[k] = total;
            total += c;
        }
        const uint32_t base = total ? atomicAdd(counter, total) : 0u;
        for (int k = 0; k < kBlock / 32; k++) warp_base[k] += base;
    }
    __syncthreads();
    return warp_base[warp] + (uint32_t)__popc(mask & ((1u << lane) - 1u));
}
__device__ __forceinline__ void write_ray(float4* rays, uint32_t* slots, uint32_t at, uint32_t slot, V3 o, V3 d,
                                          float tmax) {
    rays[2 * (size_t)at] = make_float4(o.x, o.y, o.z, tmax);
    rays[2 * (size_t)at + 1] = make_float4(d.x, d.y, d.z, 0.f);
    slots[at] = slot;
}

__device__ __forceinline__ int4 object_info(const Scene_Dev& S, uint32_t object) {
    const float4 f = __ldg(S.obj_render + 7 * (size_t)object + 6);
    return make_int4(__float_as_int(f.x), __float_as_int(f.y), __float_as_int(f.z), __float_as_int(f.w));
}

// get_emitted_radiance (direct_lighting.cpp:386-413) of a light object hit.
__device__ __forceinline__ Col emitted(const Scene_Dev& S, int4 oinfo, bool flipped) {
    if ((uint32_t)oinfo.z == YAR_LIGHT_DIFFUSE_RECTANGULAR) {
        const float4 le = __ldg(&S.lights[oinfo.w].le);
        return col(le.x, le.y, le.z);
    }
    if ((uint32_t)oinfo.z == YAR_LIGHT_DIFFUSE_SPHERE) {
        const float4 le = __ldg(&S.sphere_lights[oinfo.w].le);
        return col(le.x, le.y, le.z);
    }
    if ((uint32_t)oinfo.z == YAR_LIGHT_DIFFUSE_TRIANGLE_MESH && !flipped) {
        const float4 le = __ldg(&S.mesh_lights[oinfo.w].le);
        return col(le.x, le.y, le.z);
    }
    return col(0.f, 0.f, 0.f);
}

// How many raw pcg draws each sample's shading takes (the scattering-type
// sample, then 5 per environment sample when the hit has a BSDF), as the
// offset of each sample in its pixel's draws.  One warp per pixel.
__global__ void __launch_bounds__(kBlock)
direct_draws_kernel(Scene_Dev S, uint32_t pixels, int spp, const uint2* __restrict__ hit2, int env_samples,
                    uint32_t* __restrict__ draws) {
    const uint32_t lp = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x & 31;
    if (lp >= pixels) return;
    uint32_t before = 0;
    for (int base = 0; base < spp; base += 32) {
        const size_t i = (size_t)lp * spp + base + lane;
        uint32_t n = 0;
        if (base + lane < spp) {
            const uint2 h2 = hit2[i];
            if (h2.y != 0xffffffffu) {
                n = 1;
                if (S.env_map) {
                    const int4 oi = object_info(S, h2.y);
                    if ((uint32_t)oi.z == YAR_LIGHT_NULL && (uint32_t)oi.x != YAR_MATERIAL_NULL &&
                        S.materials[oi.y].has_bsdf)
                        n += 5u * (uint32_t)env_samples;
                }
            }
        }
        uint32_t sum = n;
        for (int d = 1; d < 32; d *= 2) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, sum, d);
            if (lane >= d) sum += v;
        }
        if (base + lane < spp) draws[i] = before + sum - n;
        before += __shfl_sync(0xffffffffu, sum, 31);
    }
}

// The camera hit of every sample: its shading, what it emits, its delta ray.
// TEXTURED: image textures or bump maps in the scene.
template <bool TEXTURED>
__global__ void __launch_bounds__(kBlock)
direct_site_kernel(Render_Params p, Scene_Dev S, uint32_t chunk_first, Direct_State D, const float4* cam_rays,
                   const float4* hit4, const uint2* hit2, const uint32_t* __restrict__ draw_offset,
                   uint32_t stream_base, const float2* __restrict__ image_samples) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    Col L = col(0.f, 0.f, 0.f);
    uint32_t info = 0;
    V3 delta_o = v3(0.f, 0.f, 0.f), delta_wi = delta_o;
    if (i < D.paths) {
        const uint32_t lp = i / (uint32_t)p.spp;
        const float4 r1 = cam_rays[2 * (size_t)i + 1];
        const V3 dir = v3(r1.x, r1.y, r1.z);
        const uint2 h2 = hit2[i];
        if (h2.y == 0xffffffffu) {
            if (S.env_map) L = env_radiance(S, dir, true);
        } else {
            int x, y;
            Pcg rng = pixel_pcg(p, pixel_stream(p, chunk_first + lp, x, y));
            pcg_advance(rng, stream_base + draw_offset[i]);
            const float4 h4 = hit4[i];
            Shading sc;
            int4 oinfo;
            init_shading(S, dir, h2.y, h2.x, h4.y, h4.z, h4.w, sc, oinfo);
            float u_sc = pcg_float(rng);
            float bsdf_prob = 1.f;
            Col delta_atten = col(1.f, 1.f, 1.f);
            int delta = 0;
            const bool is_light = (uint32_t)oinfo.z != YAR_LIGHT_NULL;
            const Material_Dev* mat = (uint32_t)oinfo.x != YAR_MATERIAL_NULL ? &S.materials[oinfo.y] : nullptr;
            // Image textures and bump maps at the camera hit, with the camera ray's
            // differentials (the delta ray's hit adds its emission only)
            Tex_Site site;
            const bool textured = TEXTURED && mat && !is_light && (mat->texture | mat->texture2 | mat->bump) != 0u;
            if (textured) {
                Path_State ps{};
                ps.image_samples = image_samples;
                ps.chunk_first = chunk_first;
                texture_site(p, S, ps, i, 0, 0u, sc, h4, h2, site);
                if (mat->bump) apply_bump(S, *mat, site, h2.y, h2.x, h4.y, h4.z, h4.w, sc);
            }
            float delta_kind = 0.f;
            if (mat && mat->delta != kDeltaNone) {
                delta = delta_scattering(sc, *mat, S.materials, u_sc, delta_wi, delta_atten, bsdf_prob, delta_kind);
                if (textured && delta == 1 && mat->delta == kDeltaGlass && (mat->texture | mat->texture2) != 0u)
                    delta_atten = textured_glass_attenuation(S, site, *mat, delta_kind, delta_atten);
            }
            if (is_light) {
                L = emitted(S, oinfo, sc.flipped);
            } else if (mat && (delta == 0 || bsdf_prob != 0.f)) {
                info |= kLit | (sc.flipped ? kFlipped : 0u) | (uint32_t)oinfo.y << 3;
                store_shading(D, i, sc);
                if constexpr (TEXTURED) {
                    Bsdf f;
                    make_bsdf(sc, *mat, S.materials, f);
                    if (textured && (mat->texture | mat->texture2) != 0u) textured_bsdf_params(S, site, *mat, f);
                    uint32_t w[kBsdfWords];
                    memcpy(w, &f, sizeof(Bsdf));
                    for (int k = 0; k < kBsdfWords; k++) D.bsdf[(size_t)k * D.paths + i] = w[k];
                }
                if (S.env_map)
                    D.rng[i] = make_uint4((uint32_t)rng.state, (uint32_t)(rng.state >> 32), (uint32_t)rng.inc,
                                          (uint32_t)(rng.inc >> 32));
            }
            if (delta == 1) {
                info |= kDeltaRay;
                delta_o = origin_for_direction(sc, delta_wi);
                D.delta[i] = make_float4(delta_atten.r, delta_atten.g, delta_atten.b, 0.f);
            }
        }
        D.info[i] = info;
        D.L[i] = make_float4(L.r, L.g, L.b, 0.f);
    }
    const bool ray = (info & kDeltaRay) != 0;
    const uint32_t at = block_append(D.counters, ray);
    if (ray) write_ray(D.prb_rays, D.prb_slot, at, i, delta_o, delta_wi, __int_as_float(0x7f800000));
}

// What the delta rays' hits add (their hits replace the camera hits).
__global__ void __launch_bounds__(kBlock)
direct_delta_kernel(Scene_Dev S, Direct_State D, const float4* __restrict__ hit4, const uint2* __restrict__ hit2,
                    unsigned long long* rays) {
    const uint32_t n = D.counters[0];
    if (blockIdx.x == 0 && threadIdx.x == 0) rays[0] += D.paths + n;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t i = D.prb_slot[k];
        const float4 r1 = D.prb_rays[2 * (size_t)k + 1], h4 = hit4[i];
        const uint2 h2 = hit2[i];
        const V3 wi = v3(r1.x, r1.y, r1.z);
        Col em = col(0.f, 0.f, 0.f);
        if (h2.y != 0xffffffffu) {
            Shading sc;
            int4 oi;
            init_shading(S, wi, h2.y, h2.x, h4.y, h4.z, h4.w, sc, oi);
            em = emitted(S, oi, sc.flipped);
        } else if (S.env_map) {
            em = env_radiance(S, wi, true);
        }
        const float4 a = D.delta[i];
        const Col c = col(a.x, a.y, a.z) * em;
        D.delta[i] = make_float4(c.r, c.g, c.b, 0.f);
    }
}

// Stratified_Pixel_Sampler's array element of this sample
// (pixel_sampling.cpp:100-141): grid `grid` at the sample's position.
__device__ __forceinline__ float2 array_sample_2d(const Render_Params& p, const Direct_Unit& u, uint32_t i, int grid,
                                                  const float2* __restrict__ s2d) {
    const uint32_t lp = i / (uint32_t)p.spp, sample = i - lp * (uint32_t)p.spp;
    const float2 g = __ldg(s2d + ((size_t)lp * p.n2d + grid + u.element) * p.spp + sample);
    const float d = 1.f / (float)u.side;
    return make_float2(one_minus_eps_min(((float)(u.element % u.side) + g.x) * d),
                       one_minus_eps_min(((float)(u.element / u.side) + g.y) * d));
}
__device__ __forceinline__ Pcg unit_pcg(const Direct_State& D, uint32_t i, const Direct_Unit& u, uint32_t skip) {
    const uint4 r = __ldg(D.rng + i);
    Pcg rng;
    rng.state = (uint64_t)r.x | (uint64_t)r.y << 32;
    rng.inc = (uint64_t)r.z | (uint64_t)r.w << 32;
    pcg_advance(rng, 5u * (uint32_t)u.element + skip);
    return rng;
}

// The light sample of every (unit, sample): its shadow ray and what it adds if
// that is unoccluded (direct_lighting.cpp:26-107 point and directional lights,
// :109-194 rectangular, :196-260 sphere, :324-384 environment).
template <bool TEXTURED>
__global__ void __launch_bounds__(kBlock, kDirectBlocks)
direct_light_kernel(Render_Params p, Scene_Dev S, Direct_State D, const Direct_Unit* __restrict__ units,
                    const float2* __restrict__ s2d) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const Direct_Unit u = units[blockIdx.y];
    if (u.kind == kUnitNoSamples) return;  // the whole block
    const uint32_t slot = blockIdx.y * D.paths + i;
    bool ray = false;
    V3 wi = v3(0.f, 0.f, 0.f), position = wi;
    float tmax = __int_as_float(0x7f800000);
    const uint32_t info = i < D.paths ? __ldg(D.info + i) : 0u;
    if (info & kLit) {
        Shading sc;
        load_shading(D, i, info, sc);
        Bsdf f;
        load_bsdf<TEXTURED>(S, D, i, info, sc, f);
        Col c = col(0.f, 0.f, 0.f);
        if (u.kind == kUnitDelta) {
            const Delta_Light_Dev& T = S.delta_lights[u.light];
            const float4 da = __ldg(&T.a), db = __ldg(&T.b), dc = __ldg(&T.c);
            float scale;
            if (__float_as_uint(da.w) == YAR_LIGHT_DIRECTIONAL) {
                wi = v3(db.x, db.y, db.z);
                const float n_dot_l = dot(sc.n, wi);
                ray = !(n_dot_l <= 0.f);
                position = origin_for_direction(sc, wi);
                scale = n_dot_l;
            } else {
                const V3 lp = v3(da.x, da.y, da.z);
                position = origin_for_point(sc, lp);
                const V3 lv = lp - position;
                const float dist = len(lv);
                wi = divs(lv, dist);
                const float n_dot_l = dot(sc.n, wi);
                ray = !(n_dot_l <= 0.f);
                tmax = dist * (1.f - 1e-5f);
                scale = n_dot_l / (dist * dist);
            }
            if (ray) c = mul(col(dc.x, dc.y, dc.z) * bsdf_evaluate(f, sc.wo, wi), scale);
        } else {
            Col Le;
            float light_pdf = 0.f, ndw = 0.f;
            bool faces = true;
            if (u.kind == kUnitEnvironment) {
                Pcg rng = unit_pcg(D, i, u, 0u);
                const float u0 = pcg_float(rng), u1 = pcg_float(rng);
                Le = env_light_sample(S, u0, u1, wi, light_pdf);
                ndw = dot(sc.n, wi);
                position = origin_for_direction(sc, wi);
            } else {
                const float2 ul = array_sample_2d(p, u, i, u.grid2, s2d);
                V3 lp;
                Sphere_Sampler ss;
                if (u.kind == kUnitRect) {
                    const Rect_Light_Dev& T = S.lights[u.light];
                    lp = xform_point(__ldg(&T.r0), __ldg(&T.r1), __ldg(&T.r2),
                                     v3(__ldg(&T.le).w * (ul.x - 0.5f), __ldg(&T.sz).x * (ul.y - 0.5f), 0.0f));
                } else {
                    const float4 sa = __ldg(&S.sphere_lights[u.light].a);
                    sphere_sampler_init(ss, v3(sa.x, sa.y, sa.z), sa.w, sc.position);
                    lp = sphere_sampler_sample(ss, ul.x, ul.y);
                }
                position = origin_for_point(sc, lp);
                const V3 lv = lp - position;
                const float dist = len(lv);
                wi = divs(lv, dist);
                tmax = dist * (1.f - 1e-5f);
                ndw = dot(sc.n, wi);
                if (u.kind == kUnitRect) {
                    const Rect_Light_Dev& T = S.lights[u.light];
                    const float4 le = __ldg(&T.le);
                    Le = col(le.x, le.y, le.z);
                    const float lndw = dot(v3(__ldg(&T.r0).z, __ldg(&T.r1).z, __ldg(&T.r2).z), -wi);
                    faces = lndw > 1e-4f;
                    light_pdf = (dist * dist) / (le.w * __ldg(&T.sz).x * lndw);
                } else {
                    const float4 le = __ldg(&S.sphere_lights[u.light].le);
                    Le = col(le.x, le.y, le.z);
                    light_pdf = ss.cone_pdf;
                }
            }
            if (faces && ((ndw > 0.f && f.reflection) || (ndw < 0.f && f.transmission))) {
                float bpdf;
                const Col fv = bsdf_value(f, sc.wo, wi, bpdf);
                if (!black(fv)) {
                    ray = true;
                    const float w = mis_power(light_pdf, bpdf);
                    c = mul(Le * fv, w * fabsf(ndw) / light_pdf);
                }
            }
        }
        D.contrib[slot] = make_float4(c.r, c.g, c.b, ray ? 1.f : 0.f);
    }
    const uint32_t at = block_append(D.counters + 1, ray);
    if (ray) write_ray(D.shd_rays, D.shd_slot, at, slot, position, wi, tmax);
}

// The BSDF sample of every (unit, sample): its probe ray, and what it adds if
// that reaches the light (for an environment light: if it is unoccluded).
template <bool TEXTURED>
__global__ void __launch_bounds__(kBlock, kDirectBlocks)
direct_bsdf_kernel(Render_Params p, Scene_Dev S, Direct_State D, const Direct_Unit* __restrict__ units,
                   const float* __restrict__ s1d, const float2* __restrict__ s2d) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const Direct_Unit u = units[blockIdx.y];
    if (u.kind <= kUnitDelta) return;  // the whole block
    const uint32_t slot = blockIdx.y * D.paths + i;
    bool ray = false;
    V3 wi = v3(0.f, 0.f, 0.f), position = wi;
    const uint32_t info = i < D.paths ? __ldg(D.info + i) : 0u;
    if (info & kLit) {
        Shading sc;
        load_shading(D, i, info, sc);
        Bsdf f;
        load_bsdf<TEXTURED>(S, D, i, info, sc, f);
        float2 ub;
        float us;
        if (u.kind == kUnitEnvironment) {
            Pcg rng = unit_pcg(D, i, u, 2u);
            ub.x = pcg_float(rng);
            ub.y = pcg_float(rng);
            us = pcg_float(rng);
        } else {
            const uint32_t lp = i / (uint32_t)p.spp, sample = i - lp * (uint32_t)p.spp;
            ub = array_sample_2d(p, u, i, u.grid2 + u.count, s2d);
            us = one_minus_eps_min(((float)u.element +
                                    __ldg(s1d + ((size_t)lp * p.n1d + u.grid1 + u.element) * p.spp + sample)) *
                                   (1.f / (float)u.count));
        }
        Bsdf_Sample bs;
        const bool alive = bsdf_direction(f, ub.x, ub.y, us, sc.wo, bs);
        wi = bs.wi;
        float bpdf = 0.f, lndw = 1.f;
        float4 probe = make_float4(0.f, 0.f, 0.f, 0.f);
        // towards the light, then the value: most samples go elsewhere
        if (alive && u.kind == kUnitRect) {
            const Rect_Light_Dev& T = S.lights[u.light];
            lndw = dot(v3(__ldg(&T.r0).z, __ldg(&T.r1).z, __ldg(&T.r2).z), -wi);
            if (lndw > 1e-4f) {
                const Col fv = bsdf_sampled_value(f, sc.wo, bs, bpdf);
                const float4 le = __ldg(&T.le);
                const Col c = col(le.x, le.y, le.z) * fv;
                ray = !black(fv);
                probe = make_float4(c.r, c.g, c.b, bpdf);
            }
        } else if (alive && u.kind == kUnitSphere) {
            const float4 sa = __ldg(&S.sphere_lights[u.light].a), le = __ldg(&S.sphere_lights[u.light].le);
            Sphere_Sampler ss;
            sphere_sampler_init(ss, v3(sa.x, sa.y, sa.z), sa.w, sc.position);
            if (dot(-ss.axes[2], wi) >= ss.cos_theta_max) {
                const Col fv = bsdf_sampled_value(f, sc.wo, bs, bpdf);
                const float w = mis_power(bpdf, ss.cone_pdf);
                const Col c = mul(col(le.x, le.y, le.z) * fv, w * fabsf(dot(sc.n, wi)) / bpdf);
                ray = !black(fv);
                probe = make_float4(c.r, c.g, c.b, 0.f);
            }
        } else if (alive) {
            const Col fv = bsdf_sampled_value(f, sc.wo, bs, bpdf);
            if (!black(fv)) {
                const Col Le = env_radiance(S, wi, false);
                ray = !black(Le);
                const float w = mis_power(bpdf, env_light_pdf(S, wi));
                const Col c = mul(Le * fv, w * fabsf(dot(sc.n, wi)) / bpdf);
                probe = make_float4(c.r, c.g, c.b, 0.f);
            }
        }
        const bool behind = !(dot(wi, sc.ng) > 0.f);
        position = behind ? sc.origin_neg : sc.origin_pos;
        if (ray) D.probe[slot] = probe;
        D.probe2[slot] = make_float2(ray ? lndw : 0.f, behind ? -fabsf(dot(sc.n, wi)) : fabsf(dot(sc.n, wi)));
    }
    const bool env = u.kind == kUnitEnvironment;  // the whole block
    const uint32_t at = block_append(D.counters + (env ? 1 : 2), ray);
    if (!ray) return;
    const float inf = __int_as_float(0x7f800000);
    if (env) write_ray(D.shd_rays, D.shd_slot, at, gridDim.y * D.paths + slot, position, wi, inf);
    else write_ray(D.prb_rays, D.prb_slot, at, slot, position, wi, inf);
}

// Every sample's sum over `n` units, in their order; the last launch of a
// chunk adds the delta ray's part and writes the radiance.
__global__ void __launch_bounds__(kBlock)
direct_sum_kernel(Scene_Dev S, Direct_State D, const Direct_Unit* __restrict__ units, uint32_t n, bool first,
                  bool last, float4* __restrict__ radiance, unsigned long long* rays) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0 && n) {
        rays[0] += D.counters[2];
        rays[1] += D.counters[1];
    }
    if (i >= D.paths) return;
    const uint32_t info = D.info[i];
    const float4 l = D.L[i];
    Col L = col(l.x, l.y, l.z), L2 = col(0.f, 0.f, 0.f);
    if ((info & kLit) && n) {
        if (!first) {
            const float4 l2 = D.L2[i];
            L2 = col(l2.x, l2.y, l2.z);
        }
        for (uint32_t k = 0; k < n; k++) {
            const Direct_Unit u = units[k];
            const size_t slot = (size_t)k * D.paths + i;
            Col out = col(0.f, 0.f, 0.f);
            if (u.kind == kUnitNoSamples) {  // a mean of nothing
                L = L + mul(out, __int_as_float(0x7f800000));
                continue;
            }
            const float4 c = __ldg(D.contrib + slot);
            if (c.w != 0.f && !D.occluded[slot])
                out = u.kind == kUnitDelta ? col(c.x, c.y, c.z) : out + col(c.x, c.y, c.z);
            if (u.kind == kUnitDelta) {
                L = L + out;
                continue;
            }
            const float2 s = __ldg(D.probe2 + slot);
            if (s.x != 0.f) {
                bool arrives;
                if (u.kind == kUnitEnvironment) {
                    arrives = !D.occluded[(size_t)n * D.paths + slot];
                } else {
                    const uint2 h2 = __ldg(D.hit2 + slot);
                    arrives = false;
                    if (h2.y != 0xffffffffu) {
                        const int4 oi = object_info(S, h2.y);
                        arrives = (uint32_t)oi.z == (u.kind == kUnitRect ? YAR_LIGHT_DIFFUSE_RECTANGULAR
                                                                         : YAR_LIGHT_DIFFUSE_SPHERE) &&
                                  oi.w == u.light;
                    }
                }
                if (arrives) {
                    const float4 pr = __ldg(D.probe + slot);
                    Col add = col(pr.x, pr.y, pr.z);
                    if (u.kind == kUnitRect) {
                        const uint2 h2 = __ldg(D.hit2 + slot);
                        const float4 h4 = __ldg(D.hit4 + slot);
                        const uint32_t tri_offset = __float_as_uint(__ldg(S.ds.objects + 6 * (size_t)h2.y + 4).w);
                        const size_t g = (size_t)tri_offset + h2.x;
                        const float4 q0 = __ldg(S.ds.tris + 3 * g), q1 = __ldg(S.ds.tris + 3 * g + 1),
                                     q2 = __ldg(S.ds.tris + 3 * g + 2);
                        const V3 hp = bary(v3(q0.x, q0.y, q0.z), v3(q1.x, q1.y, q1.z), v3(q2.x, q2.y, q2.z), h4.y,
                                           h4.z, h4.w);
                        const V3 position = load_vector(D, i, signbit(s.y) ? 6 : 5);
                        const float d = len(hp - position);
                        const float4 le = __ldg(&S.lights[u.light].le), sz = __ldg(&S.lights[u.light].sz);
                        const float light_pdf = (d * d) / (le.w * sz.x * s.x);
                        const float w = mis_power(pr.w, light_pdf);
                        add = mul(add, w * fabsf(s.y) / pr.w);
                    }
                    out = out + add;
                }
            }
            L2 = L2 + out;
            if (u.element == u.count - 1) {
                L = L + mul(L2, 1.f / (float)u.count);  // ColorRGB::operator/= multiplies by 1/v
                L2 = col(0.f, 0.f, 0.f);
            }
        }
    }
    if (last) {
        if (info & kDeltaRay) {
            const float4 c = D.delta[i];
            L = L + col(c.x, c.y, c.z);
        }
        radiance[i] = make_float4(L.r, L.g, L.b, 0.f);
    } else if (info & kLit) {
        D.L[i] = make_float4(L.r, L.g, L.b, 0.f);
        D.L2[i] = make_float4(L2.r, L2.g, L2.b, 0.f);
    }
}

} // namespace

int render_direct(yar_gpu_ctx* ctx, float* rgb_out, yar_render_stats* stats) {
    Render_Params p;
    if (int rc0 = prepare_render_params(ctx, p)) return rc0;
    cudaSetDevice(ctx->device);
    const Render_Scene& R = ctx->render;
    const auto t_start = std::chrono::steady_clock::now();
    const uint64_t pixels = (uint64_t)p.sw * p.sh;
    const uint64_t samples = pixels * p.spp;
    // k x k arrays per rectangular, then sphere light (reference_renderer.cpp:101-128)
    const int env_samples = R.has_environment ? R.environment.sample_count : 0;
    if (R.has_environment && env_samples < 1) return fail(ctx, YAR_ERR_UNSUPPORTED, "environment light without samples");
    // the pixel stream after the sample tables: image, 2D array grids, 1D array grids
    const uint64_t base = 2ull * p.spp + (uint64_t)p.n2d * (3 * p.spp - 1) + (uint64_t)p.n1d * (2 * p.spp - 1);
    if (base > 0xffffffffull) return fail(ctx, YAR_ERR_UNSUPPORTED, "too many sample arrays");

    // what every sample adds up, in this order (direct_lighting.cpp:415-520)
    std::vector<Direct_Unit> units;
    for (uint32_t type : {(uint32_t)YAR_LIGHT_POINT, (uint32_t)YAR_LIGHT_DIRECTIONAL})
        for (size_t l = 0; l < R.host_delta_lights.size(); l++)
            if (R.host_delta_lights[l].type == type) units.push_back({kUnitDelta, (int32_t)l, 0, 1, 0, 0, 1, 0});
    int grid2 = 0, grid1 = 0;
    auto add_arrays = [&](int kind, size_t l, int sample_count) {  // k x k (reference_renderer.cpp:101-128)
        const int k = (int)std::ceil(std::sqrt((double)sample_count));
        if (k < 1) units.push_back({kUnitNoSamples, (int32_t)l, 0, 1, 0, 0, 1, 0});
        for (int e = 0; e < k * k; e++) units.push_back({kind, (int32_t)l, e, k, grid2, grid1, k * k, 0});
        grid2 += 2 * k * k;
        grid1 += k * k;
    };
    for (size_t l = 0; l < R.host_rect_lights.size(); l++) add_arrays(kUnitRect, l, R.host_rect_lights[l].sample_count);
    for (size_t l = 0; l < R.host_sphere_lights.size(); l++)
        add_arrays(kUnitSphere, l, R.host_sphere_lights[l].sample_count);
    for (int k = 0; k < env_samples; k++) units.push_back({kUnitEnvironment, 0, k, 1, 0, 0, env_samples, 0});

    // scratch: a buffer of the last call is kept when it is large enough;
    // without the memory for a full chunk, smaller chunks, and without the
    // memory for the least one, the wide tree's
    std::vector<Device_Buffer>& B = ctx->render_scratch;
    if (B.size() != kDirectBuffers) {
        for (Device_Buffer& b : B) device_free(b);
        B.assign(kDirectBuffers, Device_Buffer{});
    }
    int rc = YAR_OK;
    auto alloc = [&](int i, size_t bytes) {
        if (rc == YAR_OK && !(B[i].ptr && B[i].bytes >= bytes)) rc = device_alloc(ctx, B[i], bytes);
    };
    uint64_t chunk_pixels = 0, cap = 0, slots = 0, per_launch = 0;
    const uint64_t most_units = std::max<uint64_t>(1, std::min<uint64_t>(units.size(), kMaxUnits));
    for (uint64_t shrink = 1;;) {
        rc = YAR_OK;
        chunk_pixels = std::max<uint64_t>(1, std::min<uint64_t>(pixels, kDirectPaths / shrink / p.spp));
        cap = chunk_pixels * p.spp;  // samples per chunk
        per_launch = std::max<uint64_t>(1, std::min<uint64_t>(most_units, kDirectRaySlots / shrink / cap));
        slots = std::max(cap, cap * per_launch);  // rays per queue
        alloc(0, samples * sizeof(float4));                   // radiance
        alloc(1, samples * sizeof(float2));                   // image-plane samples
        alloc(2, cap * std::max(1, p.n1d) * sizeof(float));   // s1d: 1D array grids
        alloc(3, cap * std::max(1, p.n2d) * sizeof(float2));  // s2d: 2D array grids
        alloc(4, cap * sizeof(float4));                       // camera kernel's coeff, then the delta rays' part
        alloc(5, cap * sizeof(float4));                       // L
        alloc(6, cap * sizeof(uint32_t));                     // info
        alloc(7, cap * sizeof(uint4));                        // rng
        alloc(8, cap * 2 * sizeof(float4));                   // camera rays
        alloc(9, cap * sizeof(uint32_t));                     // camera ray slots
        alloc(10, cap * 21 * sizeof(float));                  // shading
        alloc(11, cap * sizeof(float4));                      // hit4 of camera and delta rays
        alloc(12, cap * sizeof(uint2));                       // hit2
        alloc(13, cap * sizeof(uint32_t));                    // draw offsets
        alloc(14, pixel_film_bytes(pixels));                  // pixel variance, film sums
        alloc(15, (size_t)p.tiles_x * p.tiles_y * sizeof(double));
        alloc(16, (size_t)p.rw * p.rh * 3 * sizeof(float));   // rgb
        alloc(17, 2 * sizeof(unsigned long long) + 4 * sizeof(int));  // ray counts, traversal error
        alloc(18, std::max<size_t>(1, units.size()) * sizeof(Direct_Unit));
        alloc(19, cap * sizeof(float4));                      // L2
        if (p.textured) alloc(20, cap * sizeof(Bsdf));
        alloc(21, slots * sizeof(float4));                    // contrib
        alloc(22, 2 * slots * sizeof(uint8_t));               // occluded
        alloc(23, slots * sizeof(float4));                    // probe
        alloc(24, slots * sizeof(float2));                    // probe2
        alloc(25, slots * sizeof(float4));                    // probe hit4
        alloc(26, slots * sizeof(uint2));                     // probe hit2
        alloc(27, (env_samples ? 2 : 1) * slots * 2 * sizeof(float4));  // shadow rays
        alloc(28, (env_samples ? 2 : 1) * slots * sizeof(uint32_t));    // shadow slots
        alloc(29, slots * 2 * sizeof(float4));                // probe and delta rays
        alloc(30, slots * sizeof(uint32_t));                  // probe and delta slots
        alloc(31, (env_samples ? 2 : 1) * slots * sizeof(uint32_t));    // the wide tree's answers
        alloc(32, 8 * sizeof(uint32_t));                      // queue counters, ray hand-out
        const bool least = chunk_pixels == 1 && per_launch == 1;
        if (rc != YAR_ERR_NOMEM || (least && !wide_leave(ctx))) break;
        for (Device_Buffer& b : B) device_free(b);
        shrink = least ? 1 : 4 * shrink;
    }
    if (rc != YAR_OK) return rc;
    Path_State ps{};
    ps.coeff = dptr<float4>(B[4]);
    ps.L = dptr<float4>(B[5]);
    ps.info = dptr<uint32_t>(B[6]);
    ps.rng = dptr<uint4>(B[7]);
    Queues q{};
    q.ext_rays[0] = dptr<float4>(B[8]);
    q.ext_slot[0] = dptr<uint32_t>(B[9]);
    float4* hit4 = dptr<float4>(B[11]);
    uint2* hit2 = dptr<uint2>(B[12]);
    unsigned long long* rays_dev = dptr<unsigned long long>(B[17]);
    int* err = reinterpret_cast<int*>(rays_dev + 2);
    const Direct_Unit* units_dev = dptr<Direct_Unit>(B[18]);
    Direct_State D{};
    D.info = ps.info;
    D.shading = dptr<float>(B[10]);
    D.bsdf = dptr<uint32_t>(B[20]);
    D.rng = ps.rng;
    D.L = ps.L;
    D.L2 = dptr<float4>(B[19]);
    D.delta = ps.coeff;
    D.contrib = dptr<float4>(B[21]);
    D.occluded = dptr<uint8_t>(B[22]);
    D.probe = dptr<float4>(B[23]);
    D.probe2 = dptr<float2>(B[24]);
    D.hit4 = dptr<float4>(B[25]);
    D.hit2 = dptr<uint2>(B[26]);
    D.shd_rays = dptr<float4>(B[27]);
    D.shd_slot = dptr<uint32_t>(B[28]);
    D.prb_rays = dptr<float4>(B[29]);
    D.prb_slot = dptr<uint32_t>(B[30]);
    D.counters = dptr<uint32_t>(B[32]);
    Scene_Dev S = scene_dev(ctx->ds, ctx->render);
    cudaStream_t st = ctx->stream;
    cudaError_t e = cudaMemsetAsync(rays_dev, 0, B[17].bytes, st);
    if (e == cudaSuccess && !units.empty())
        e = cudaMemcpyAsync(B[18].ptr, units.data(), units.size() * sizeof(Direct_Unit), cudaMemcpyHostToDevice, st);
    uint32_t launches = 0;
    const int closest_kernel = render_choice(ctx, 0, 0), any_kernel = render_choice(ctx, 1, 0);
    Cast_Args cast;
    cast.next_ray_zeroed = true;
    cast.err = err;
    cast.answers = dptr<uint32_t>(B[31]);
    auto trace_closest = [&](const float4* rays, uint32_t n, const uint32_t* count, const uint32_t* slot, float4* h4,
                             uint2* h2, int hand_out) {
        Cast_Args a = cast;
        a.rays = rays;
        (count ? a.n_max : a.n) = n;
        a.count = count;
        a.perm = slot;
        a.next_ray = D.counters + hand_out;
        a.hit4 = h4;
        a.hit2 = h2;
        launches += closest_kernel == kCastWide ? 2 : 1;
        return launch_extend(ctx->ds, a, closest_kernel, st);
    };
    for (uint64_t first = 0; first < pixels && e == cudaSuccess; first += chunk_pixels) {
        const uint32_t cp = (uint32_t)std::min<uint64_t>(chunk_pixels, pixels - first);
        const uint32_t paths = cp * (uint32_t)p.spp, blocks = (paths + kBlock - 1) / kBlock;
        D.paths = paths;
        e = launch_generate(p, (uint32_t)first, cp, dptr<float>(B[2]), dptr<float>(B[3]), dptr<float2>(B[1]), ps, q,
                            st);
        if (e == cudaSuccess) e = cudaMemsetAsync(D.counters, 0, 8 * sizeof(uint32_t), st);
        if (e == cudaSuccess) e = trace_closest(q.ext_rays[0], paths, nullptr, nullptr, hit4, hit2, 4);
        if (e != cudaSuccess) break;
        direct_draws_kernel<<<(uint32_t)(((uint64_t)cp * 32 + kBlock - 1) / kBlock), kBlock, 0, st>>>(
            S, cp, p.spp, hit2, env_samples, dptr<uint32_t>(B[13]));
        (p.textured ? direct_site_kernel<true> : direct_site_kernel<false>)<<<blocks, kBlock, 0, st>>>(
            p, S, (uint32_t)first, D, q.ext_rays[0], hit4, hit2, dptr<uint32_t>(B[13]), (uint32_t)base,
            dptr<float2>(B[1]));
        e = trace_closest(D.prb_rays, paths, D.counters, D.prb_slot, hit4, hit2, 5);
        if (e != cudaSuccess) break;
        direct_delta_kernel<<<std::min(blocks, 152u * 16u), kBlock, 0, st>>>(S, D, hit4, hit2, rays_dev);
        launches += 5;
        size_t u0 = 0;
        do {
            const uint32_t n = (uint32_t)std::min<uint64_t>(per_launch, units.size() - u0);
            if (n) {
                const dim3 grid(blocks, n);
                const bool arrays = std::any_of(units.begin() + u0, units.begin() + u0 + n,
                                                [](const Direct_Unit& u) { return u.kind > kUnitDelta; });
                e = cudaMemsetAsync(D.counters, 0, 8 * sizeof(uint32_t), st);
                if (e != cudaSuccess) break;
                (p.textured ? direct_light_kernel<true> : direct_light_kernel<false>)<<<grid, kBlock, 0, st>>>(
                    p, S, D, units_dev + u0, dptr<float2>(B[3]));
                if (arrays)
                    (p.textured ? direct_bsdf_kernel<true> : direct_bsdf_kernel<false>)<<<grid, kBlock, 0, st>>>(
                        p, S, D, units_dev + u0, dptr<float>(B[2]), dptr<float2>(B[3]));
                Cast_Args a = cast;
                a.rays = D.shd_rays;
                a.count = D.counters + 1;
                a.n_max = (env_samples ? 2 : 1) * n * paths;
                a.perm = D.shd_slot;
                a.next_ray = D.counters + 4;
                a.occluded = D.occluded;
                e = launch_shadow(ctx->ds, a, any_kernel, st);
                if (e == cudaSuccess && arrays)
                    e = trace_closest(D.prb_rays, n * paths, D.counters + 2, D.prb_slot, D.hit4, D.hit2, 5);
                launches += (arrays ? 2 : 1) + (any_kernel == kCastWide ? 2 : 1);
                if (e != cudaSuccess) break;
            }
            direct_sum_kernel<<<blocks, kBlock, 0, st>>>(S, D, units_dev + u0, n, u0 == 0, u0 + n == units.size(),
                                                         dptr<float4>(B[0]) + first * p.spp, rays_dev);
            launches++;
            u0 += n;
        } while (u0 < units.size());
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        const Pixel_Film pf = pixel_film(p, B[14].ptr, pixels);
        launch_samples(p, dptr<float4>(B[0]), dptr<float2>(B[1]), pf, st);
        tile_variance_kernel<<<p.tiles_x * p.tiles_y, kTileVarThreads, 0, st>>>(p, pf.variance, dptr<double>(B[15]));
        film_kernel<<<(uint32_t)(((uint64_t)p.rw * p.rh + kBlock - 1) / kBlock), kBlock, 0, st>>>(
            p, dptr<float4>(B[0]), dptr<float2>(B[1]), pf, dptr<float>(B[16]));
        launches += 3;
        e = cudaGetLastError();
    }
    std::vector<double> tile_var((size_t)p.tiles_x * p.tiles_y);
    unsigned long long rays[3] = {0, 0, 0};  // closest, any, then the error word
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(rgb_out, B[16].ptr, (size_t)p.rw * p.rh * 3 * sizeof(float), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(tile_var.data(), B[15].ptr, tile_var.size() * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(rays, rays_dev, sizeof(rays), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "direct-lighting render");
    if (rays[2]) return fail(ctx, YAR_ERR_CAPACITY, "kd-tree traversal stack overflow");
    if (stats) {
        double acc = 0.0;
        int64_t count = 0;
        for (int t = 0; t < p.tiles_x * p.tiles_y; t++) {
            acc += tile_var[t];
            const int tx = t % p.tiles_x, ty = t / p.tiles_x;
            count += (int64_t)std::min(kTile, p.sw - tx * kTile) * std::min(kTile, p.sh - ty * kTile);
        }
        stats->variance = p.spp > 1 ? acc / (double)count : 0.0;
        stats->seconds = (float)std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count();
        stats->paths = samples;
        stats->rays_closest = rays[0];
        stats->rays_any = rays[1];
        stats->kernel_launches = launches;
    }
    return YAR_OK;
}

} // namespace yar
