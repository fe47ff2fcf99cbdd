// guide_mlp.cu - the network of the learned directional proposal: a BF16
// MLP with FP32 accumulation on the tensor cores (tcgen05, accumulators in
// tensor memory), with hand-written inference and training kernels.
//
// Network: 128 inputs (16-frequency sin/cos encoding of the normalised
// position, frequencies pi f_k, f_k = (2^((k mod 3)/3) in float32) 2^(k div 3),
// k = 0..15: 96; shading normal 3,
// outgoing direction 3, zeros, input 127 = constant 1) -> 3 hidden layers of 64 ReLU units (unit 63 of each is the
// constant 1, so every bias is an ordinary weight column) -> 64 outputs, of
// which 40 parameterise a mixture of 8 von Mises-Fisher lobes in world space:
// per lobe an unnormalised mean direction m (3), log-concentration r and a
// mixture logit l.  kappa = exp(clamp(r, -3, 8)), pi = softmax(l).
//
// A group of 128 threads handles a tile of 128 rows (= TMEM lanes = threads):
// one thread issues the MMAs (M = 128, N = 64, K = 16 per instruction), all
// threads run the epilogues (tcgen05.ld of their lane, bias-free ReLU, BF16
// pack into the next layer's operand tile).  Several groups share a CTA and
// its copy of the weights, so that one group's epilogue runs while another's
// MMA is in flight.  Training fuses the forward pass, the loss gradient, the
// backward pass and the weight gradients: the weight gradients dW^T = A^T dY
// accumulate in tensor memory over all tiles a CTA processes, and each CTA
// writes one partial gradient; adam_kernel sums the partials.
//
// Loss for a sample direction w drawn with pdf p at (x, n, wo) with target
// value t (incident radiance x BSDF x cosine, as luminance): -(t / p) log q(w),
// whose expectation is the KL divergence from the normalised target to the
// mixture q up to a constant (the estimator of neural importance sampling).
#include "context.hpp"
#include "tc.cuh"

#include <cuda_bf16.h>

#include <cmath>
#include <random>
#include <vector>

namespace yar {

namespace {

constexpr int kRows = 128;
constexpr int kIn = 128;
constexpr int kHid = 64;
constexpr int kOut = 64;
constexpr uint32_t kWaitLimit = 1u << 20;  // mbarrier polls before a tile is abandoned

// parameter vector, fp32, row-major [out][in]
constexpr int kW1 = 0;
constexpr int kW2 = kW1 + kHid * kIn;
constexpr int kW3 = kW2 + kHid * kHid;
constexpr int kW4 = kW3 + kHid * kHid;
static_assert(kW4 + kOut * kHid == kGuideParams, "parameter count");

// bf16 operand images in tile layout: W1 (64 x 128), W2..W4 (64 x 64), rows =
// output unit.  Every tile serves as a K-major operand (rows x columns) and,
// with the MN-major bit, as its transpose: its 8 x 8 core matrices are the
// same in both, only the roles of the two strides change.  So the backward
// pass reads W as W^T, and the weight gradients read the activation and
// gradient rows as A^T and dY, without transposed copies.
constexpr uint32_t kImgW1 = 0, kImgW2 = 16384, kImgW3 = 24576, kImgW4 = 32768, kImgBytes = 40960;
constexpr int kGradOut = 48;  // columns of the output gradient's tile: the 40 outputs, then zeros

// shared memory, training: images | per group: X (32 KB), H1 H2 H3 (16 KB
// each; each is overwritten by its gradient), dOut (12 KB) | misc.  H tiles
// hold 64 columns but the transposed M = 128 operand reads 128: columns 64 to
// 127 come from the following rows, at the end of a tile from the tile behind
// it (their products land in TMEM lanes that are never read).
constexpr int kTrGroups = 2;
constexpr uint32_t kTrX = 0, kTrH = 32768, kTrDOut = kTrH + 3 * 16384, kTrGroupBytes = kTrDOut + kRows * kGradOut * 2;
constexpr uint32_t kTrMisc = kImgBytes + kTrGroups * kTrGroupBytes;
constexpr int kTrThreads = kTrGroups * kRows + 32;  // and a warp that issues the MMAs
// shared memory, inference: images | per group 32 KB of rows | misc
constexpr int kInGroups = 5;
constexpr uint32_t kInMisc = kImgBytes + kInGroups * 32768u;
constexpr int kInThreads = kInGroups * kRows;
constexpr uint32_t kMiscBytes = 192;  // 0: barriers, 96: TMEM address, 100: abort flag, 128: drain barriers
static_assert(kTrMisc + kMiscBytes <= 232448 && kInMisc + kMiscBytes <= 232448, "227 KB of shared memory");

// kind::f16 instruction descriptors: operands K-major, or read as their transpose
constexpr uint32_t kTransA = 1u << 15, kTransB = 1u << 16;

struct Mlp_Args {
    const uint8_t* images;
    const float4* rows;  // 3 float4 per query row, 4 per training row
    uint32_t n;
    const uint32_t* count;
    uint32_t stride, offset;  // row r of this launch is input row offset + r * stride
    float3 lo, inv_ext;
    float* lobes;          // inference: kGuideLobeFloats per row
    float* partials;       // training: kGuideParams per CTA
    const float* w_scale;  // training
    float* loss;           // training
    int* err;
};

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Encoding frequencies f_k = f_(k mod 3) 2^(k div 3), k = 0..15 (1 to 32
// half-periods across the scene box), from the float32 values of 2^(b/3),
// b = 0, 1, 2: three chains of doublings.
__constant__ float kFreq[3] = {1.000000000e+00f, 1.259921074e+00f, 1.587401032e+00f};

// Input features j and j + 1 (j even), visited in increasing j.  j < 96: sin
// and cos of pi f_k p_axis, k = j / 6, axis = (j % 6) / 2: a sincospif for
// k < 3, then each chain (axis, k mod 3) doubles its angle (sin 2x =
// 2 sin x cos x, cos 2x = (cos x - sin x)(cos x + sin x)), which leaves the
// features within 1e-6 of sincospif's, far below their BF16 rounding.  Then
// the normal, wo, zeros and the constant 1 at 127.
struct Encoding {
    float s[3][3], c[3][3];  // running sin and cos per (axis, chain)
};
__device__ __forceinline__ void feature_pair(int j, float3 p, float3 nrm, float3 wo, Encoding& e, float& f0,
                                             float& f1) {
    if (j < 96) {
        const int k = j / 6, a = (j % 6) / 2, b = k % 3;
        if (k < 3) {
            const float x = (a == 0) ? p.x : (a == 1 ? p.y : p.z);
            sincospif(x * kFreq[b], &e.s[a][b], &e.c[a][b]);
        } else {
            const float sn = e.s[a][b], cs = e.c[a][b];
            e.s[a][b] = 2.f * sn * cs;
            e.c[a][b] = (cs - sn) * (cs + sn);
        }
        f0 = e.s[a][b];
        f1 = e.c[a][b];
        return;
    }
    auto fixed = [&](int i) -> float {
        switch (i) {
            case 96: return nrm.x;
            case 97: return nrm.y;
            case 98: return nrm.z;
            case 99: return wo.x;
            case 100: return wo.y;
            case 101: return wo.z;
            case 127: return 1.f;
            default: return 0.f;
        }
    };
    f0 = fixed(j);
    f1 = fixed(j + 1);
}

__device__ __forceinline__ void store_row8(uint8_t* tile, int r, int k0, int K, const float* v) {
    uint4 q;
    q.x = pack_bf16(v[0], v[1]);
    q.y = pack_bf16(v[2], v[3]);
    q.z = pack_bf16(v[4], v[5]);
    q.w = pack_bf16(v[6], v[7]);
    *reinterpret_cast<uint4*>(tile + tc::tile_offset(r, k0, K)) = q;
}

// An MMA operand over K = 16 * n: a tile of `cols` columns, its rows the M or
// N dimension (K-major), or its columns (MN-major, `trans`).
struct Operand {
    uint32_t addr, cols;
    bool trans;
};
__device__ __forceinline__ uint64_t operand_desc(const Operand& o, int k16) {
    const uint32_t rows8 = o.cols * 16u;  // from 8 rows to the next 8
    return o.trans ? tc::smem_desc(o.addr + 2u * rows8 * (uint32_t)k16, rows8, 128u)
                   : tc::smem_desc(o.addr + 256u * (uint32_t)k16, 128u, rows8);
}
__device__ __forceinline__ void gemm(uint32_t d_tmem, Operand a, Operand b, int K, int N, bool accumulate) {
    const uint32_t idesc = tc::idesc_bf16_f32(128, N) | (a.trans ? kTransA : 0u) | (b.trans ? kTransB : 0u);
    for (int s = 0; s < K / 16; s++)
        tc::mma(d_tmem, operand_desc(a, s), operand_desc(b, s), idesc, (accumulate || s > 0) ? 1u : 0u);
}

template <int N>
__device__ __forceinline__ void load_row(uint32_t taddr, float (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N; i += 16) tc::tmem_ld16(taddr + i, *reinterpret_cast<float(*)[16]>(v + i));
    tc::tmem_wait_ld();
}

// Before an MMA: the generic-proxy shared-memory writes of this thread become
// visible to the tensor core, and its tensor-memory reads are ordered before
// the MMA; `ready` counts the group's threads.
__device__ __forceinline__ void arrive_ready(uint32_t ready) {
    tc::fence_proxy_async();
    tc::fence_before_sync();
    tc::mbar_arrive(ready);
}

// Bounded wait; gives up at once when another thread has given up.
__device__ __forceinline__ bool wait_or_abort(uint32_t mbar, uint32_t parity, volatile int* abort) {
    for (uint32_t i = 0; i < kWaitLimit / 64u; i++) {
        if (tc::mbar_wait(mbar, parity, 64u)) return true;
        if (*abort) return false;
    }
    *abort = 1;
    return false;
}

// After giving up: the MMAs that this thread has issued finish (or the wait's
// limit runs out) before the tensor memory is freed.
__device__ __forceinline__ void drain(uint32_t mbar) {
    tc::commit(mbar);
    tc::mbar_wait(mbar, 0u, kWaitLimit);
}

// A row of the input (3 float4 a query, 4 a training sample).
struct Input {
    float3 p, nrm, wo, wdir;
    float wt;
};
template <bool TRAIN>
__device__ __forceinline__ Input load_input(const Mlp_Args& a, uint32_t row, bool valid, float w_scale) {
    Input x;
    x.p = x.nrm = x.wo = x.wdir = make_float3(0.f, 0.f, 0.f);
    x.wt = 0.f;
    if (valid) {
        const float4* q = a.rows + ((size_t)a.offset + (size_t)row * a.stride) * (TRAIN ? 4 : 3);
        const float4 q0 = __ldg(q), q1 = __ldg(q + 1), q2 = __ldg(q + 2);
        x.p = make_float3((q0.x - a.lo.x) * a.inv_ext.x, (q0.y - a.lo.y) * a.inv_ext.y,
                          (q0.z - a.lo.z) * a.inv_ext.z);
        x.nrm = make_float3(q0.w, q1.x, q1.y);
        x.wo = make_float3(q1.z, q1.w, q2.x);
        if (TRAIN) {
            x.wdir = make_float3(q2.y, q2.z, q2.w);
            x.wt = __ldg(q + 3).x * w_scale;
        }
    }
    return x;
}

// The input features of this thread's row into the tile X.
__device__ __forceinline__ void store_features(uint8_t* X, int r, const Input& x) {
    Encoding enc;
#pragma unroll
    for (int c = 0; c < 16; c++) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; i += 2) feature_pair(8 * c + i, x.p, x.nrm, x.wo, enc, v[i], v[i + 1]);
        store_row8(X, r, 8 * c, kIn, v);
    }
}

// ReLU of a row of 64 sums into the operand tile H; unit 63 is the constant 1.
// The maximum is taken on the rounded pairs (rounding keeps the order).
__device__ __forceinline__ void store_hidden(uint8_t* H, int r, const float (&v)[64]) {
    const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
    for (int c = 0; c < 8; c++) {
        uint32_t q[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int j = 8 * c + 2 * i;
            const __nv_bfloat162 h = __hmax2(__floats2bfloat162_rn(v[j], j == 62 ? 1.f : v[j + 1]), zero);
            q[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(H + tc::tile_offset(r, 8 * c, kHid)) = make_uint4(q[0], q[1], q[2], q[3]);
    }
}

// A row of 64 gradients, zero where the unit's ReLU is (and for the constant
// unit), over that unit's activations in the tile H.
__device__ __forceinline__ void store_hidden_grad(uint8_t* H, int r, const float (&v)[64]) {
    const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
    for (int c = 0; c < 8; c++) {
        uint4* at = reinterpret_cast<uint4*>(H + tc::tile_offset(r, 8 * c, kHid));
        const uint4 h4 = *at;
        const uint32_t h[4] = {h4.x, h4.y, h4.z, h4.w};
        uint32_t q[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int j = 8 * c + 2 * i;
            const uint32_t on = __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&h[i]), zero);
            q[i] = pack_bf16(v[j], v[j + 1]) & (j == 62 ? on & 0xffffu : on);
        }
        *at = make_uint4(q[0], q[1], q[2], q[3]);
    }
}

// Mixture parameters and the loss gradient of one row (training) from the 40
// raw outputs; `d` receives d(loss)/d(raw).
__device__ __forceinline__ float mixture_grad(const float (&o)[kGradOut], float3 w_dir, float wt,
                                              float (&d)[kGradOut]) {
    float lp[8], lv[8], kap[8], len[8], cdot[8], inrange[8];
    float3 mu[8];
    float lmax = -1e30f;
#pragma unroll
    for (int k = 0; k < 8; k++) lmax = fmaxf(lmax, o[5 * k + 4]);
    float lsum = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) lsum += __expf(o[5 * k + 4] - lmax);
    const float llse = lmax + __logf(lsum);
    float qmax = -1e30f;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const float mx = o[5 * k], my = o[5 * k + 1], mz = o[5 * k + 2];
        len[k] = sqrtf(mx * mx + my * my + mz * mz) + 1e-6f;
        mu[k] = make_float3(mx / len[k], my / len[k], mz / len[k]);
        const float r = o[5 * k + 3];
        const float rc = fminf(fmaxf(r, -3.f), 8.f);
        inrange[k] = (r > -3.f && r < 8.f) ? 1.f : 0.f;
        kap[k] = __expf(rc);
        cdot[k] = mu[k].x * w_dir.x + mu[k].y * w_dir.y + mu[k].z * w_dir.z;
        lp[k] = o[5 * k + 4] - llse;
        // log C(kappa) = log kappa - log(2 pi) - log(1 - exp(-2 kappa))
        lv[k] = rc - 1.8378770664f - log1pf(-__expf(-2.f * kap[k])) + kap[k] * (cdot[k] - 1.f);
        qmax = fmaxf(qmax, lp[k] + lv[k]);
    }
    float qs = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) qs += __expf(lp[k] + lv[k] - qmax);
    const float logq = qmax + __logf(qs);
#pragma unroll
    for (int j = 40; j < kGradOut; j++) d[j] = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const float gam = __expf(lp[k] + lv[k] - logq);
        const float pik = __expf(lp[k]);
        d[5 * k + 4] = -wt * (gam - pik);
        const float e2 = __expf(-2.f * kap[k]);
        const float dlv = 1.f / kap[k] - 2.f * e2 / (1.f - e2) + (cdot[k] - 1.f);
        d[5 * k + 3] = -wt * gam * dlv * kap[k] * inrange[k];
        const float s = -wt * gam * kap[k] / len[k];
        d[5 * k + 0] = s * (w_dir.x - cdot[k] * mu[k].x);
        d[5 * k + 1] = s * (w_dir.y - cdot[k] * mu[k].y);
        d[5 * k + 2] = s * (w_dir.z - cdot[k] * mu[k].z);
    }
    return -wt * logq;
}

// Weight images into shared memory, barriers, tensor memory; returns its address.
template <int GROUPS>
__device__ __forceinline__ uint32_t mlp_begin(const Mlp_Args& a, uint8_t* sm, uint32_t misc, uint32_t ready_count) {
    const uint32_t base = tc::smem_addr(sm);
    for (uint32_t i = threadIdx.x; i < kImgBytes / 16; i += blockDim.x)
        reinterpret_cast<uint4*>(sm)[i] = __ldg(reinterpret_cast<const uint4*>(a.images) + i);
    if (threadIdx.x < 32) tc::tmem_alloc(base + misc + 96, 512u);
    if (threadIdx.x == 0) {
        for (int g = 0; g < GROUPS; g++) {
            tc::mbar_init(base + misc + 16 * g, ready_count);
            tc::mbar_init(base + misc + 16 * g + 8, 1);
            tc::mbar_init(base + misc + 128 + 8 * g, 1);
        }
        *reinterpret_cast<int*>(sm + misc + 100) = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    return *reinterpret_cast<uint32_t*>(sm + misc + 96);
}
__device__ __forceinline__ uint32_t mlp_rows(const Mlp_Args& a) {
    return a.count ? (*a.count > a.offset ? (*a.count - a.offset + a.stride - 1) / a.stride : 0u) : a.n;
}

// Inference.  A tile is a serial chain (features, 4 MMAs, 4 epilogues; 1,500
// instructions per row), so the tiles in flight per SM set the rate: 5 groups
// on one copy of the weights, where 3 CTAs of one group with their own copies
// fitted.  The results leave through shared memory (16-byte stores 160 bytes
// apart took 320 of the 480 shared-memory and store cycles of a warp's rows).
// 1M rows: 137 us with 3 CTAs per SM, 120 us with 5 groups, 92 us with both;
// 52% of the issue slots, 32 us at the copy bandwidth.
__global__ void __launch_bounds__(kInThreads, 1) mlp_infer_kernel(Mlp_Args a) {
    extern __shared__ __align__(1024) uint8_t sm[];
    const uint32_t tmem = mlp_begin<kInGroups>(a, sm, kInMisc, kRows);
    const int group = threadIdx.x / kRows, tid = threadIdx.x % kRows;
    const uint32_t base = tc::smem_addr(sm);
    const uint32_t ready = base + kInMisc + 16 * group, done = ready + 8;
    volatile int* abort = reinterpret_cast<volatile int*>(sm + kInMisc + 100);
    const uint32_t d_tmem = tmem + 64u * group;
    const uint32_t lane_addr = d_tmem + ((uint32_t)(tid & ~31) << 16);
    const uint32_t r_off = kImgBytes + 32768u * group;
    uint8_t* R = sm + r_off;  // X, then the hidden layers' rows in its halves
    // a warp's results on their way out: where its own rows of X are
    constexpr uint32_t kLobeBytes = kGuideLobeFloats * 4u;
    static_assert(kGuideLobeFloats == 40 && 32u * kLobeBytes <= 32u * kIn * 2u, "a warp's rows");
    uint8_t* out = R + (tid / 32) * (32 * kIn * 2);
    const uint32_t n = mlp_rows(a), tiles = (n + kRows - 1) / kRows;
    uint32_t parity = 0;
    bool ok = true;
    // D = A * W^T of the group's tile
    auto product = [&](uint32_t a_off, uint32_t w_off, uint32_t K) {
        arrive_ready(ready);
        if (tid == 0 && wait_or_abort(ready, parity, abort)) {
            tc::fence_after_sync();
            gemm(d_tmem, Operand{base + a_off, K, false}, Operand{base + w_off, K, false}, (int)K, kHid, false);
            tc::commit(done);
        }
        const bool got = __all_sync(0xffffffffu, wait_or_abort(done, parity, abort));
        parity ^= 1u;
        tc::fence_after_sync();
        return got;
    };
    for (uint32_t t = group; ok; t += kInGroups) {
        const uint64_t tile = blockIdx.x + (uint64_t)t * gridDim.x;
        if (tile >= tiles) break;
        const uint32_t row = (uint32_t)tile * kRows + tid;
        const bool valid = row < n;
        const Input x = load_input<false>(a, row, valid, 0.f);
        if ((tid & 31) == 0) tc::bulk_wait_read();  // the last tile's results have left `out`
        __syncwarp();
        store_features(R, tid, x);
        ok = product(r_off, kImgW1, kIn);
        uint32_t w_off = kImgW2;
#pragma unroll 1
        for (int l = 0; l < 3 && ok; l++) {
            float v[64];
            load_row(lane_addr, v);
            store_hidden(R + 16384 * (l & 1), tid, v);
            ok = product(r_off + 16384u * (l & 1), w_off, kHid);
            w_off += 8192u;
        }
        if (!ok) break;
        float o[kGradOut];
        load_row(lane_addr, o);
        if (valid) {
            float lmax = -1e30f;
#pragma unroll
            for (int k = 0; k < 8; k++) lmax = fmaxf(lmax, o[5 * k + 4]);
            float e[8], es = 0.f;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                e[k] = __expf(o[5 * k + 4] - lmax);
                es += e[k];
            }
            float f[40];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const float mx = o[5 * k], my = o[5 * k + 1], mz = o[5 * k + 2];
                const float il = 1.f / (sqrtf(mx * mx + my * my + mz * mz) + 1e-6f);
                f[5 * k + 0] = mx * il;
                f[5 * k + 1] = my * il;
                f[5 * k + 2] = mz * il;
                f[5 * k + 3] = __expf(fminf(fmaxf(o[5 * k + 3], -3.f), 8.f));
                f[5 * k + 4] = e[k] / es;
            }
#pragma unroll
            for (int i = 0; i < 10; i++)
                reinterpret_cast<float4*>(out + (tid & 31) * kLobeBytes)[i] =
                    make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
        }
        tc::fence_proxy_async();
        __syncwarp();
        const uint32_t row0 = (uint32_t)tile * kRows + (tid & ~31);
        if ((tid & 31) == 0 && row0 < n)
            tc::bulk_store(a.lobes + (size_t)row0 * kGuideLobeFloats, tc::smem_addr(out),
                           min(n - row0, 32u) * kLobeBytes);
    }
    if ((tid & 31) == 0) tc::bulk_wait_all();
    __syncwarp();
    if (!ok) {
        atomicOr(a.err, 2);
        if (tid == 0) drain(base + kInMisc + 128 + 8 * group);
        __syncwarp();
    }
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) tc::tmem_dealloc(tmem, 512u);
}

// Training.  Two groups per CTA, each on every other tile of the CTA's, and a
// warp that issues the MMAs of both in a fixed order: the weight gradients of
// both accumulate in the same tensor-memory columns, tile after tile.  With
// transposed copies of every operand (shuffles and 4-byte stores, 40% of the
// instructions, and shared memory for one tile only) 262,144 rows took 219 us;
// now 98 us: 3,400 instructions per row at 2 warps per scheduler, 26% of the
// issue slots.
__global__ void __launch_bounds__(kTrThreads, 1) mlp_train_kernel(Mlp_Args a) {
    extern __shared__ __align__(1024) uint8_t sm[];
    const uint32_t tmem = mlp_begin<kTrGroups>(a, sm, kTrMisc, kRows);
    const int group = threadIdx.x / kRows, tid = threadIdx.x % kRows;
    const uint32_t base = tc::smem_addr(sm);
    volatile int* abort = reinterpret_cast<volatile int*>(sm + kTrMisc + 100);
    const uint32_t n = mlp_rows(a), tiles = (n + kRows - 1) / kRows;
    // this CTA's tiles: blockIdx.x, blockIdx.x + gridDim.x, ...
    const uint32_t mine = blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;
    const uint32_t grads = tmem + 64u * kTrGroups;  // dW1^T, then dW2^T, dW3^T, dW4^T: 64 columns each
    bool ok = true;
    float loss_sum = 0.f;
    if (group == kTrGroups) {
        // the issuing warp: the steps of the groups' tiles in turn
        const bool issuer = tid == 0;
        uint32_t parity = 0;
        for (uint32_t t = 0; t < mine && ok; t += kTrGroups) {
#pragma unroll 1
            for (int step = 0; step < 8 && ok; step++) {
#pragma unroll 1
                for (uint32_t g = 0; g < (uint32_t)kTrGroups && t + g < mine && ok; g++) {
                    const uint32_t ready = base + kTrMisc + 16 * g;
                    const uint32_t tile = base + kImgBytes + kTrGroupBytes * g;
                    const uint32_t d = tmem + 64u * g;
                    const bool acc = t + g > 0;
                    ok = __all_sync(0xffffffffu, wait_or_abort(ready, parity, abort));
                    if (ok && issuer) {
                        tc::fence_after_sync();
                        const uint32_t h = tile + kTrH;
                        if (step == 0) {
                            gemm(d, Operand{tile + kTrX, kIn, false}, Operand{base + kImgW1, kIn, false}, kIn, kHid,
                                 false);
                        } else if (step < 4) {
                            gemm(d, Operand{h + 16384u * (step - 1), kHid, false},
                                 Operand{base + kImgW2 + 8192u * (step - 1), kHid, false}, kHid, kHid, false);
                        } else if (step < 7) {
                            // layer l's input gradient dY W and weight gradient A^T dY; dY of the output
                            // layer in its own tile, else in the tile of the layer's activations
                            const uint32_t l = 6u - (uint32_t)step;  // weights W(l + 2), input H(l + 1)
                            const uint32_t dy = l == 2u ? tile + kTrDOut : h + 16384u * (l + 1u);
                            const uint32_t cols = l == 2u ? (uint32_t)kGradOut : (uint32_t)kHid;
                            gemm(d, Operand{dy, cols, false}, Operand{base + kImgW2 + 8192u * l, kHid, true},
                                 (int)cols, kHid, false);
                            gemm(grads + 64u * (l + 1u), Operand{h + 16384u * l, kHid, true},
                                 Operand{dy, cols, true}, kRows, (int)cols, acc);
                        } else {
                            gemm(grads, Operand{tile + kTrX, kIn, true}, Operand{h, kHid, true}, kRows, kHid, acc);
                        }
                        tc::commit(ready + 8);
                    }
                    __syncwarp();
                }
                parity ^= 1u;
            }
        }
        if (!ok && issuer) drain(base + kTrMisc + 128);
        __syncwarp();
    } else {
        const uint32_t ready = base + kTrMisc + 16 * group, done = ready + 8;
        const uint32_t lane_addr = tmem + 64u * group + ((uint32_t)(tid & ~31) << 16);
        uint8_t* tile_sm = sm + kImgBytes + kTrGroupBytes * group;
        const float w_scale = __ldg(a.w_scale);
        uint32_t parity = 0;
        auto step = [&]() {
            arrive_ready(ready);
            const bool got = __all_sync(0xffffffffu, wait_or_abort(done, parity, abort));
            parity ^= 1u;
            tc::fence_after_sync();
            return got;
        };
        for (uint32_t t = group; t < mine && ok; t += kTrGroups) {
            const uint32_t row = (blockIdx.x + t * gridDim.x) * kRows + tid;
            const bool valid = row < n;
            const Input x = load_input<true>(a, row, valid, w_scale);
            store_features(tile_sm + kTrX, tid, x);
            ok = step();
#pragma unroll 1
            for (int l = 0; l < 3 && ok; l++) {
                float v[64];
                load_row(lane_addr, v);
                store_hidden(tile_sm + kTrH + 16384 * l, tid, v);
                ok = step();
            }
            if (!ok) break;
            {
                float o[kGradOut], d[kGradOut];
                load_row(lane_addr, o);
                const float l = mixture_grad(o, x.wdir, x.wt, d);
                if (valid) loss_sum += l;
#pragma unroll
                for (int c = 0; c < kGradOut / 8; c++)
                    store_row8(tile_sm + kTrDOut, tid, 8 * c, kGradOut, d + 8 * c);
            }
            ok = step();
#pragma unroll 1
            for (int l = 2; l >= 0 && ok; l--) {
                float v[64];
                load_row(lane_addr, v);
                store_hidden_grad(tile_sm + kTrH + 16384 * l, tid, v);
                ok = step();
            }
        }
    }
    const bool drained = !ok;
    ok = !__syncthreads_or(!ok);
    tc::fence_after_sync();
    if (!ok) {
        if (threadIdx.x == 0) atomicOr(a.err, 2);
        // a group gave up on a step that the issuing warp had issued as its last
        if (threadIdx.x == kTrGroups * kRows && !drained) drain(base + kTrMisc + 128);
    }

    // partial gradients of this CTA, in the parameter layout [out][in]
    float* part = a.partials + (size_t)blockIdx.x * kGuideParams;
    if (group == 0) {
        if (mine > 0 && ok) {
            const uint32_t lane_grads = grads + ((uint32_t)(tid & ~31) << 16);
            float v[64];
            load_row(lane_grads, v);
#pragma unroll
            for (int j = 0; j < 64; j++) part[kW1 + j * kIn + tid] = v[j];
            if (tid < kHid) {
#pragma unroll 1
                for (int l = 0; l < 3; l++) {
                    load_row(lane_grads + 64u * (uint32_t)(l + 1), v);
                    const int off = l == 0 ? kW2 : (l == 1 ? kW3 : kW4);
#pragma unroll
                    for (int j = 0; j < 64; j++) part[off + j * kHid + tid] = l == 2 && j >= kGradOut ? 0.f : v[j];
                }
            }
        } else {
            for (int i = tid; i < kGuideParams; i += kRows) part[i] = 0.f;
        }
    }
    if (group < kTrGroups) {
        float s = loss_sum;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
        if ((tid & 31) == 0 && s != 0.f) atomicAdd(a.loss, s);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) tc::tmem_dealloc(tmem, 512u);
}

// The MLP kernels' bounded mbarrier wait on a barrier that nothing arrives
// at: the limit runs out, the error word is set and the kernel returns, with
// no copy or MMA in flight.  Exercises the expiry path of the wait.
__global__ void wait_selftest_kernel(uint32_t limit, int* err) {
    __shared__ __align__(8) uint64_t mbar;
    if (threadIdx.x == 0) {
        const uint32_t a = (uint32_t)__cvta_generic_to_shared(&mbar);
        tc::mbar_init(a, 1);
        if (!tc::mbar_wait(a, 0, limit)) atomicExch(err, 1);
    }
}

// fp32 parameters -> bf16 operand images.
__global__ void images_kernel(const float* __restrict__ params, uint8_t* __restrict__ img) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kGuideParams) return;
    const float w = params[i];
    const __nv_bfloat16 b = __float2bfloat16_rn(w);
    auto put = [&](uint32_t off) { *reinterpret_cast<__nv_bfloat16*>(img + off) = b; };
    if (i < kW2) {
        const int nn = i / kIn, k = i % kIn;
        put(kImgW1 + tc::tile_offset(nn, k, kIn));
        return;
    }
    const int l = (i - kW2) / (kHid * kHid);  // 0: W2, 1: W3, 2: W4
    const int j = (i - kW2) % (kHid * kHid);
    const int nn = j / kHid, k = j % kHid;
    const uint32_t fwd = l == 0 ? kImgW2 : (l == 1 ? kImgW3 : kImgW4);
    put(fwd + tc::tile_offset(nn, k, kHid));
}

// Sum of the per-CTA partial gradients; Adam step when `lr` > 0, else the
// summed gradient is written to `grad_out`.
__global__ void adam_kernel(const float* __restrict__ partials, int parts, float* __restrict__ params,
                            float* __restrict__ m, float* __restrict__ v, float lr, float beta1, float beta2,
                            float eps, float c1, float c2, float* __restrict__ grad_out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kGuideParams) return;
    float g = 0.f;
#pragma unroll 16
    for (int c = 0; c < parts; c++) g += partials[(size_t)c * kGuideParams + i];
    if (grad_out) {
        grad_out[i] = g;
        return;
    }
    const float mi = beta1 * m[i] + (1.f - beta1) * g;
    const float vi = beta2 * v[i] + (1.f - beta2) * g * g;
    m[i] = mi;
    v[i] = vi;
    params[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
}

// The current device's SM count (the partial-gradient slots and the grids),
// cached per device.
int sm_count() {
    static int sms[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (sms[dev] == 0) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    return sms[dev];
}

} // namespace

int guide_ensure(yar_gpu_ctx* ctx) {
    Guide& g = ctx->guide;
    if (g.params.ptr) return YAR_OK;
    int rc = YAR_OK;
    const size_t pb = kGuideParams * sizeof(float);
    cudaSetDevice(ctx->device);
    if (sm_count() <= 0) return fail(ctx, YAR_ERR_INVALID, "guide: no SM count for the device");
    if ((rc = work_alloc(ctx, g.params, pb)) != YAR_OK) return rc;
    if ((rc = work_alloc(ctx, g.adam_m, pb)) != YAR_OK) return rc;
    if ((rc = work_alloc(ctx, g.adam_v, pb)) != YAR_OK) return rc;
    if ((rc = work_alloc(ctx, g.images, kImgBytes)) != YAR_OK) return rc;
    if ((rc = work_alloc(ctx, g.partials, (size_t)sm_count() * pb)) != YAR_OK) return rc;
    if ((rc = work_alloc(ctx, g.scalars, 64)) != YAR_OK) return rc;
    cudaError_t e = cudaMemsetAsync(g.images.ptr, 0, kImgBytes, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "guide init");
    static bool attr[64] = {};  // per device
    if (ctx->device < 0 || ctx->device >= 64) return fail(ctx, YAR_ERR_INVALID, "guide: device index");
    if (!attr[ctx->device]) {
        e = cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(kTrMisc + kMiscBytes));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(mlp_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(kInMisc + kMiscBytes));
        if (e != cudaSuccess) return cuda_fail(ctx, e, "guide kernel attributes");
        attr[ctx->device] = true;
    }
    return guide_reset(ctx, 1);
}

int guide_reset(yar_gpu_ctx* ctx, uint64_t seed) {
    // He-uniform hidden weights, small output weights (broad, even lobes at
    // the start), zero bias columns.
    std::vector<float> w(kGuideParams, 0.f);
    std::mt19937_64 rng(seed);
    std::uniform_real_distribution<float> u(-1.f, 1.f);
    auto fill = [&](int off, int rows, int cols, int fan_in, float gain, int used_rows, int used_cols) {
        const float b = gain * std::sqrt(6.f / (float)fan_in);
        for (int r = 0; r < rows; r++)
            for (int c = 0; c < cols; c++)
                w[off + r * cols + c] = (r < used_rows && c < used_cols) ? b * u(rng) : 0.f;
    };
    fill(kW1, kHid, kIn, 102, 1.f, kHid - 1, 102);
    fill(kW2, kHid, kHid, kHid - 1, 1.f, kHid - 1, kHid - 1);
    fill(kW3, kHid, kHid, kHid - 1, 1.f, kHid - 1, kHid - 1);
    fill(kW4, kOut, kHid, kHid - 1, 0.1f, kGuideLobeFloats, kHid - 1);
    return guide_set_params(ctx, w.data());
}

int guide_set_params(yar_gpu_ctx* ctx, const float* host_params) {
    Guide& g = ctx->guide;
    const size_t pb = kGuideParams * sizeof(float);
    cudaError_t e = cudaMemcpyAsync(g.params.ptr, host_params, pb, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(g.adam_m.ptr, 0, pb, ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(g.adam_v.ptr, 0, pb, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "guide parameters");
    g.step = 0;
    images_kernel<<<(kGuideParams + 255) / 256, 256, 0, ctx->stream>>>((const float*)g.params.ptr,
                                                                        (uint8_t*)g.images.ptr);
    e = cudaStreamSynchronize(ctx->stream);  // the host vector may die at return
    if (e != cudaSuccess) return cuda_fail(ctx, e, "guide parameters");
    return YAR_OK;
}

cudaError_t guide_infer(yar_gpu_ctx* ctx, const float4* queries, uint32_t n_max, const uint32_t* count,
                        const float* box, float* lobes, cudaStream_t st) {
    Guide& g = ctx->guide;
    if (n_max == 0) return cudaSuccess;
    Mlp_Args a{};
    a.images = (const uint8_t*)g.images.ptr;
    a.rows = queries;
    a.n = n_max;
    a.count = count;
    a.stride = 1;
    a.offset = 0;
    a.lo = make_float3(box[0], box[1], box[2]);
    a.inv_ext = make_float3(1.f / std::max(box[3] - box[0], 1e-20f), 1.f / std::max(box[4] - box[1], 1e-20f),
                            1.f / std::max(box[5] - box[2], 1e-20f));
    a.lobes = lobes;
    a.err = ctx->d_error;
    const uint32_t tiles = (n_max + kRows - 1) / kRows;
    const uint32_t grid = std::min<uint32_t>(tiles, (uint32_t)sm_count());
    mlp_infer_kernel<<<grid, kInThreads, kInMisc + kMiscBytes, st>>>(a);
    return cudaGetLastError();
}

cudaError_t guide_train(yar_gpu_ctx* ctx, const float4* samples, uint32_t n_max, const uint32_t* count,
                        uint32_t stride, uint32_t offset, const float* box, const float* w_scale_dev, float lr,
                        float* grad_out, cudaStream_t st) {
    Guide& g = ctx->guide;
    if (n_max == 0) return cudaSuccess;
    Mlp_Args a{};
    a.images = (const uint8_t*)g.images.ptr;
    a.rows = samples;
    a.n = n_max;
    a.count = count;
    a.stride = stride;
    a.offset = offset;
    a.lo = make_float3(box[0], box[1], box[2]);
    a.inv_ext = make_float3(1.f / std::max(box[3] - box[0], 1e-20f), 1.f / std::max(box[4] - box[1], 1e-20f),
                            1.f / std::max(box[5] - box[2], 1e-20f));
    a.partials = (float*)g.partials.ptr;
    a.w_scale = w_scale_dev;
    a.loss = (float*)g.scalars.ptr;
    a.err = ctx->d_error;
    const uint32_t tiles = (n_max + kRows - 1) / kRows;
    const int grid = (int)std::min<uint32_t>(tiles, (uint32_t)sm_count());
    mlp_train_kernel<<<grid, kTrThreads, kTrMisc + kMiscBytes, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    float c1 = 1.f, c2 = 1.f;
    if (!grad_out) {
        g.step++;
        c1 = 1.f / (1.f - std::pow(g.beta1, (float)g.step));
        c2 = 1.f / (1.f - std::pow(g.beta2, (float)g.step));
    }
    adam_kernel<<<(kGuideParams + 255) / 256, 256, 0, st>>>((const float*)g.partials.ptr, grid, (float*)g.params.ptr,
                                                            (float*)g.adam_m.ptr, (float*)g.adam_v.ptr, lr, g.beta1,
                                                            g.beta2, g.eps, c1, c2, grad_out);
    if (!grad_out)
        images_kernel<<<(kGuideParams + 255) / 256, 256, 0, st>>>((const float*)g.params.ptr, (uint8_t*)g.images.ptr);
    return cudaGetLastError();
}

void guide_release(yar_gpu_ctx* ctx) {
    Guide& g = ctx->guide;
    for (Device_Buffer* b : {&g.params, &g.adam_m, &g.adam_v, &g.images, &g.partials, &g.scalars}) device_free(*b);
}


// ---------------------------------------------------------------- C ABI
namespace {

int guide_call_prologue(yar_gpu_ctx* ctx) {
    if (!ctx) return YAR_ERR_INVALID;
    cudaSetDevice(ctx->device);
    return guide_ensure(ctx);
}

int guide_finish(yar_gpu_ctx* ctx, cudaError_t e, const char* what, float* loss) {
    struct {
        int err;
        float loss;
    } h = {0, 0.f}, *words = &h;  // (pageable without the context's page-locked block)
    if (char* p = pinned_block(ctx)) words = reinterpret_cast<decltype(words)>(p);
    if (e == cudaSuccess && loss)
        e = cudaMemcpyAsync(&words->loss, ctx->guide.scalars.ptr, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&words->err, ctx->d_error, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, what);
    if (loss) *loss = words->loss;
    if (words->err) {
        cudaMemset(ctx->d_error, 0, sizeof(int));
        return fail(ctx, YAR_ERR_TIMEOUT, "tensor-core wait gave up");
    }
    return YAR_OK;
}

int guide_step(yar_gpu_ctx* ctx, const float* samples, uint32_t n, const float* box, float weight_scale, float lr,
               float* grad, float* loss) {
    int rc = guide_call_prologue(ctx);
    if (rc != YAR_OK) return rc;
    if (!box || (n && !samples) || (((uintptr_t)samples & 15u) != 0)) return fail(ctx, YAR_ERR_INVALID, "guide step");
    float* scal = (float*)ctx->guide.scalars.ptr;
    const float h[2] = {0.f, weight_scale};
    cudaError_t e = cudaMemcpyAsync(scal, h, sizeof(h), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess)
        e = guide_train(ctx, (const float4*)samples, n, nullptr, 1, 0, box, scal + 1, lr, grad, ctx->stream);
    return guide_finish(ctx, e, "guide training step", loss);
}

} // namespace

extern "C" int yar_guide_set_params(yar_gpu_ctx* ctx, const float* params) {
    int rc = guide_call_prologue(ctx);
    if (rc != YAR_OK) return rc;
    if (!params) return fail(ctx, YAR_ERR_INVALID, "null parameters");
    return guide_set_params(ctx, params);
}

extern "C" int yar_guide_get_params(yar_gpu_ctx* ctx, float* params) {
    int rc = guide_call_prologue(ctx);
    if (rc != YAR_OK) return rc;
    if (!params) return fail(ctx, YAR_ERR_INVALID, "null parameters");
    cudaError_t e = cudaMemcpyAsync(params, ctx->guide.params.ptr, kGuideParams * sizeof(float),
                                    cudaMemcpyDeviceToHost, ctx->stream);
    return guide_finish(ctx, e, "guide parameters", nullptr);
}

extern "C" int yar_gpu_wait_selftest(yar_gpu_ctx* ctx, uint32_t limit) {
    if (!ctx) return YAR_ERR_INVALID;
    if (limit == 0 || limit > (1u << 24)) return fail(ctx, YAR_ERR_INVALID, "wait self-test: limit in [1, 2^24]");
    cudaSetDevice(ctx->device);
    wait_selftest_kernel<<<1, 32, 0, ctx->stream>>>(limit, ctx->d_error);
    return guide_finish(ctx, cudaGetLastError(), "wait self-test", nullptr);
}

extern "C" int yar_guide_infer(yar_gpu_ctx* ctx, const float* queries, uint32_t n, const float* box, float* lobes) {
    int rc = guide_call_prologue(ctx);
    if (rc != YAR_OK) return rc;
    if (!box || (n && (!queries || !lobes)) || (((uintptr_t)queries & 15u) != 0) || (((uintptr_t)lobes & 15u) != 0))
        return fail(ctx, YAR_ERR_INVALID, "guide inference");
    cudaError_t e = guide_infer(ctx, (const float4*)queries, n, nullptr, box, lobes, ctx->stream);
    return guide_finish(ctx, e, "guide inference", nullptr);
}

extern "C" int yar_guide_gradient(yar_gpu_ctx* ctx, const float* samples, uint32_t n, const float* box,
                                  float weight_scale, float* grad, float* loss) {
    if (ctx && !grad) return fail(ctx, YAR_ERR_INVALID, "null gradient buffer");
    return guide_step(ctx, samples, n, box, weight_scale, 0.f, grad, loss);
}

extern "C" int yar_guide_train_step(yar_gpu_ctx* ctx, const float* samples, uint32_t n, const float* box,
                                    float weight_scale, float learning_rate, float* loss) {
    return guide_step(ctx, samples, n, box, weight_scale, learning_rate, nullptr, loss);
}

} // namespace yar
