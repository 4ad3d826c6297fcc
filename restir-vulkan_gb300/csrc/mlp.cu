// mlp.cu -- kernels of the learned light-cluster proposal (network in mlp.cuh).
//
// The forward pass of a 128-pixel tile is one CTA on the tcgen05 tensor cores:
// features -> x tile (shared memory, bf16) -> three 64-wide layers (MMA into
// tensor memory, bias + ReLU + bf16 epilogue back into shared memory) -> the
// cluster logit layer in chunks of 64 clusters, double-buffered in tensor
// memory so that the MMA of chunk c+1 runs under the epilogue of chunk c.
// Weight tiles arrive by cp.async from bf16 images that are already in the MMA
// operand layout.  Logits never leave the SM.  Exponentials are 2^x on the MUFU
// unit with the log2(e) scale folded into one FMA per logit.  Bound by issue
// slots and by the latency of the epilogues (55-60 % of the slots, 15 warps an
// SM), so they read b4 from shared memory (global loads, even from L1, were
// most of the stalls), and kSample draws a row's uniforms before its search
// and kLse finds an arg-max by triples; tile addresses are arithmetic (a pointer
// array would live in local memory, a load from L2 a chunk) and tile copies have
// compile-time sizes.  2,073,600 rows and 4096 clusters, both passes: 5.66 ms,
// 7.38 without these.  Two epilogues:
//   kLse     log-sum-exp, arg-max and its probability per row;
//   kSample  the learned-branch candidates: each row walks its softmax CDF
//            once with its uniforms drawn as ascending order statistics; a
//            uniform's column inside the 32-column piece that holds it is
//            found by binary search over the piece's running sums, and its
//            probability is the width of its interval.  (The uniform-branch
//            candidates, a light and q of its cluster, are written at the
//            end of kLse.)
// Training runs kLse with the hidden activations saved, then from h3:
//   k_mlp_grad  dz = d(loss)/d(logits) = (softmax - onehot) / n per chunk into
//            a bf16 tile, then dh3 += dz W4^T on the tensor cores, and the
//            cross-entropy loss;
//   k_mlp_dw4   dW4 and db4, from the logits recomputed chunk by chunk (dz
//            never leaves the SM);
//   k_mlp_backward_rows  the hidden layers.
// Every wait on the tensor core is bounded; a CTA whose wait runs out records
// an error, waits (bounded) for its last MMA, frees its tensor memory and
// leaves.  At most four CTAs share an SM: each holds 128 tensor-memory
// columns and uses more than a fifth of the shared memory.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "mlp.cuh"
#include "rg_math.cuh"
#include "umma.cuh"

using namespace rgm;

namespace {

constexpr int kRows = 128;                 // rows (pixels) per CTA
constexpr int kChunkN = mlp::kChunkN;      // clusters per logit MMA chunk
constexpr uint32_t kMaxPolls = 1u << 26;   // bounded mbarrier waits
constexpr int kTmemCols = 2 * kChunkN;    // two chunk accumulators; the hidden layers use them first

// shared-memory map (bytes)
constexpr int kOffX = 0;                               // x tile, 128 x 16 bf16
constexpr int kOffH = kOffX + kRows * mlp::kIn * 2;    // h tile, 128 x 64 bf16
constexpr int kOffW1 = kOffH + kRows * mlp::kH * 2;    // W1^T image, 64 x 16
constexpr int kOffW2 = kOffW1 + mlp::kH * mlp::kIn * 2;
constexpr int kOffW3 = kOffW2 + mlp::kH * mlp::kH * 2;
constexpr int kOffB = kOffW3 + mlp::kH * mlp::kH * 2;  // two chunk tiles, 128 x 64
constexpr int kChunkBytes = kChunkN * mlp::kH * 2;
constexpr int kOffBias = kOffB + 2 * kChunkBytes;      // b1 | b2 | b3
static_assert(kOffB - kOffW1 >= (mlp::kCand + 1) * kRows * 4, "kSample's uniforms lie over the hidden weights");
constexpr int kSmemUsed = kOffBias + 3 * mlp::kH * 4;
// b4 of three chunks, in turn, over the x tile once layer 1 has read it
constexpr int kOffB4 = kOffX;
constexpr int kB4Bytes = kChunkN * 4;
static_assert(3 * kB4Bytes <= kRows * mlp::kIn * 2, "three chunks' biases fit the x tile");
constexpr int kWkBytes = mlp::kH * kChunkN * 2;
constexpr int kHTileBytes = kRows * mlp::kH * 2;       // 128 rows of a saved hidden layer, laid out as the MMA operand tile
constexpr int kSmemMin = 52 * 1024;                    // caps residency at four CTAs per SM (TMEM: 4 x 128 columns)
constexpr int kWeightImgBytes = (mlp::kH * mlp::kIn + 2 * mlp::kH * mlp::kH) * 2;

enum { kLse = 0, kSample = 1 };

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

constexpr float kLog2e = 1.44269504088896341f;
// 2^x by the MUFU instruction (results below 2^-126 flush to zero)
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// A 32-column piece of one row is held as 16 float2 pairs (columns 2k, 2k+1),
// so that adds and FMAs run as packed FP32x2 operations (each lane of a
// packed op rounds exactly like the scalar op).
__device__ __forceinline__ float col(const float2 (&v)[16], int i) { return (i & 1) ? v[i >> 1].y : v[i >> 1].x; }
// max of three (IEEE maxNum, like fmaxf)
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float y;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}
// The piece's maximum; a: the maxima of columns 3 k .. 3 k + 2.
__device__ __forceinline__ float max32(const float2 (&v)[16], float (&a)[11]) {
#pragma unroll
    for (int k = 0; k < 10; ++k) a[k] = max3f(col(v, 3 * k), col(v, 3 * k + 1), col(v, 3 * k + 2));
    a[10] = fmaxf(col(v, 30), col(v, 31));
    const float b0 = max3f(a[0], a[1], a[2]), b1 = max3f(a[3], a[4], a[5]), b2 = max3f(a[6], a[7], a[8]);
    return fmaxf(max3f(b0, b1, b2), fmaxf(a[9], a[10]));
}
// The first column whose value is the maximum mp, by its triple (44
// instructions; one test per column takes 64).
__device__ __forceinline__ int first_max(const float2 (&v)[16], const float (&a)[11], float mp) {
    int t = 10;
    float e0 = col(v, 30), e1 = col(v, 31);
#pragma unroll
    for (int k = 9; k >= 0; --k)
        if (a[k] == mp) {
            t = k;
            e0 = col(v, 3 * k);
            e1 = col(v, 3 * k + 1);
        }
    return 3 * t + (e0 == mp ? 0 : e1 == mp ? 1 : 2);
}
__device__ __forceinline__ float sum32(const float2 (&v)[16]) {
    float2 t[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) t[k] = __fadd2_rn(v[k], v[k + 8]);
#pragma unroll
    for (int k = 0; k < 4; ++k) t[k] = __fadd2_rn(t[k], t[k + 4]);
    t[0] = __fadd2_rn(t[0], t[2]);
    t[1] = __fadd2_rn(t[1], t[3]);
    t[0] = __fadd2_rn(t[0], t[1]);
    return t[0].x + t[0].y;
}
// v[k] = 2^(v[k] * log2(e) + off), both columns of every pair
__device__ __forceinline__ void exp_piece(float2 (&v)[16], float off) {
    const float2 l2 = make_float2(kLog2e, kLog2e), o2 = make_float2(off, off);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const float2 t = __ffma2_rn(v[k], l2, o2);
        v[k] = make_float2(ex2(t.x), ex2(t.y));
    }
}
__device__ __forceinline__ float lg2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Next of n ascending order statistics of U(0,1) given the previous one:
// 1 - (1 - prev) * V^(1/remaining), V uniform; the power as 2^(log2(V) / n)
// on the MUFU unit (V = 0 gives 1: beyond every CDF total).
__device__ __forceinline__ float next_order_stat(Pcg &rng, float prev, int remaining) {
    const float v = rand_float(rng);
    return 1.0f - (1.0f - prev) * ex2(lg2(v) * rcp((float)remaining));
}
// z of cluster cl for the row whose h3 is h: FP32 dot (even and odd terms
// in two packed FMA chains) with the bf16 W4^T image (chunk tiles in the MMA
// operand layout) plus b4.
__device__ __forceinline__ float logit_of(const mlp::ProposalDev &pd, const float (&h)[64], int cl) {
    const unsigned char *tile = reinterpret_cast<const unsigned char *>(pd.w4t) + (size_t)(cl / kChunkN) * kChunkBytes;
    float2 z = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const uint4 w = __ldg(reinterpret_cast<const uint4 *>(tile + umma::kmajor_offset(cl % kChunkN, 8 * j, mlp::kH)));
        const __nv_bfloat162 *b = reinterpret_cast<const __nv_bfloat162 *>(&w);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            z = __ffma2_rn(make_float2(h[8 * j + 2 * i], h[8 * j + 2 * i + 1]), __bfloat1622float2(b[i]), z);
    }
    return (z.x + z.y) + __ldg(pd.b4e + cl);
}

__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(umma::smem_addr(smem_dst)), "l"(gsrc)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
// kBytes (a multiple of 16) by the block's 128 threads.  Both known when
// compiled, so a tile is a run of copies at fixed offsets: as a loop over
// blockDim, its address arithmetic was a tenth of inference (2,073,600 rows, 4096
// clusters: 6.28 against 5.78 ms) and 4 % of the gradients.
template <int kBytes>
__device__ __forceinline__ void copy_tile(unsigned char *dst, const unsigned char *src) {
    constexpr int kStep = kRows * 16;
    const int o = threadIdx.x * 16;
#pragma unroll
    for (int i = 0; i < kBytes / kStep; ++i) cp_async16(dst + o + i * kStep, src + o + i * kStep);
    if (kBytes % kStep != 0 && o < kBytes % kStep)
        cp_async16(dst + o + kBytes / kStep * kStep, src + o + kBytes / kStep * kStep);
}

struct FusedParams {
    mlp::ProposalDev pd;
    GBufView g;
    float cam[3];
    const int32_t *rows;       // pixel of each row; nullptr: row = pixel
    int n;
    float4 *stat;              // per row: lse, arg-max cluster (int bits), its probability, 0
    // training (kLse with save != 0)
    int save;
    __nv_bfloat16 *x, *h1, *h2, *h3;  // [n x 16]; the hidden layers by tiles of 128 rows (zeros from row n on)
    // sampling
    mlp::Candidate *cand;      // [n x kCand]
    uint32_t frame;
    int n_cand;
    int *err;
    // batched views (kViews): row -> view by binary search over first_row
    const mlp::ViewRows *views;
    int n_views;
    const uint32_t *frames;    // per view
};

// Features of one pixel (mlp.cuh), each rounded to bf16; non-finite values
// (a pixel at the camera position) become 0.
__device__ __forceinline__ void features(const mlp::ProposalDev &pd, const float4 *wpos_plane, const uint2 *normal_plane,
                                         float cx, float cy, float cz, size_t px, float x[mlp::kIn]) {
    const float4 wp = __ldg(wpos_plane + px);
    const uint2 nb = __ldg(normal_plane + px);
    const f3 wpos = mk(wp.x, wp.y, wp.z);
    const f3 n = mk(half_bits_to_float((uint16_t)(nb.x & 0xffffu)), half_bits_to_float((uint16_t)(nb.x >> 16)),
                    half_bits_to_float((uint16_t)(nb.y & 0xffffu)));
    const f3 v = normalize(mk(cx, cy, cz) - wpos);
    x[0] = (wpos.x - pd.box_center.x) * pd.box_inv_half.x;
    x[1] = (wpos.y - pd.box_center.y) * pd.box_inv_half.y;
    x[2] = (wpos.z - pd.box_center.z) * pd.box_inv_half.z;
    x[3] = n.x; x[4] = n.y; x[5] = n.z;
    x[6] = v.x; x[7] = v.y; x[8] = v.z;
#pragma unroll
    for (int i = 0; i < mlp::kIn; ++i) {
        const float t = i < mlp::kInUsed ? x[i] : 0.0f;
        x[i] = isfinite(t) ? bf16r(t) : 0.0f;
    }
}

// Writes 8 consecutive bf16 values (k = k0..k0+7) of row r into a K-major tile.
__device__ __forceinline__ void put8(unsigned char *tile, int r, int k0, int K, const float *v) {
    __align__(16) __nv_bfloat162 b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = __float22bfloat162_rn(make_float2(v[2 * i], v[2 * i + 1]));
    *reinterpret_cast<uint4 *>(tile + umma::kmajor_offset(r, k0, K)) = *reinterpret_cast<const uint4 *>(b);
}
__device__ __forceinline__ void store8(__nv_bfloat16 *dst, const float *v) {
    __align__(16) __nv_bfloat162 b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = __float22bfloat162_rn(make_float2(v[2 * i], v[2 * i + 1]));
    *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(b);
}

// One 32-column piece of a row's logit gradient, (softmax - onehot) / n as
// bf16 into the K-major dz tile: v holds the logits, nl2 = -lse * log2(e),
// hit = target - first column or kNoTarget (the row's gradient is 0).  Only the
// piece that holds a row's target pays for the one-hot: testing every column
// took 445 instructions a piece instead of about 150.  Returns the target's logit where the piece holds it, else 0.
constexpr int kNoTarget = INT32_MIN;
__device__ __forceinline__ float grad_piece(unsigned char *dztile, int row, int col0, const float2 (&v)[16], float nl2,
                                            float inv_n, int hit) {
    float2 d[16];
    const float2 l2 = make_float2(kLog2e, kLog2e), o2 = make_float2(nl2, nl2), s2 = make_float2(inv_n, inv_n);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const float2 t = __ffma2_rn(v[k], l2, o2);
        d[k] = __fmul2_rn(make_float2(ex2(t.x), ex2(t.y)), s2);
    }
    if (hit == kNoTarget) {
#pragma unroll
        for (int k = 0; k < 16; ++k) d[k] = make_float2(0.0f, 0.0f);
    }
#pragma unroll
    for (int q = 0; q < 32; q += 8) {
        uint4 w;
        uint32_t *b = reinterpret_cast<uint32_t *>(&w);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const __nv_bfloat162 h = __float22bfloat162_rn(d[q / 2 + k]);
            b[k] = *reinterpret_cast<const uint32_t *>(&h);
        }
        *reinterpret_cast<uint4 *>(dztile + umma::kmajor_offset(row, col0 + q, kChunkN)) = w;
    }
    float zt = 0.0f;
    if ((unsigned)hit < 32u) {  // the one-hot column: its logit by five rounds of selects, its gradient over the one stored
        float2 t[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) t[k] = (hit & 16) ? v[k + 8] : v[k];
#pragma unroll
        for (int k = 0; k < 4; ++k) t[k] = (hit & 8) ? t[k + 4] : t[k];
#pragma unroll
        for (int k = 0; k < 2; ++k) t[k] = (hit & 4) ? t[k + 2] : t[k];
        t[0] = (hit & 2) ? t[1] : t[0];
        zt = (hit & 1) ? t[0].y : t[0].x;
        *reinterpret_cast<__nv_bfloat16 *>(dztile + umma::kmajor_offset(row, col0 + hit, kChunkN)) =
            __float2bfloat16_rn((ex2(__fmaf_rn(zt, kLog2e, nl2)) - 1.0f) * inv_n);
    }
    return zt;
}

// Bounded wait for an MMA commit; warp-uniform result.
__device__ __forceinline__ bool mma_wait(uint64_t *mbar, uint32_t parity) {
    bool w = umma::mbar_wait(mbar, parity, kMaxPolls);
    umma::fence_after_sync();
    return __all_sync(0xffffffffu, w);
}

template <int kMode, bool kViews>
__global__ void __launch_bounds__(128, 4) k_mlp_fused(const FusedParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t mbar_layer, mbar_chunk[2];
    __shared__ uint32_t tmem_base;
    constexpr int kCols = kTmemCols;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int row = blockIdx.x * kRows + tid;
    const bool valid = row < p.n;
    size_t px;
    uint32_t frame = p.frame;
    int n_cand = p.n_cand;
    const float4 *wpos_plane = p.g.wpos;
    const uint2 *normal_plane = p.g.normal;
    float cx = p.cam[0], cy = p.cam[1], cz = p.cam[2];
    if constexpr (kViews) {
        // the view holding this row: the last one whose first row is <= row
        const uint32_t r = valid ? (uint32_t)row : 0u;
        int lo = 0, hi = p.n_views - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(&p.views[mid].first_row) <= r) lo = mid;
            else hi = mid - 1;
        }
        const mlp::ViewRows &vr = p.views[lo];
        px = (size_t)(r - vr.first_row);
        frame = __ldg(p.frames + lo);
        n_cand = vr.n_cand;
        wpos_plane = vr.g.wpos;
        normal_plane = vr.g.normal;
        cx = vr.cam[0];
        cy = vr.cam[1];
        cz = vr.cam[2];
    } else {
        px = valid ? (p.rows ? (size_t)p.rows[row] : (size_t)row) : 0;
    }
    const int nch = p.pd.c / kChunkN;
    const mlp::Layout L(p.pd.c);
    unsigned char *xtile = smem + kOffX, *htile = smem + kOffH;
    // by arithmetic: an array of pointers indexed at run time would live in local memory
    auto btile = [&](int i) { return smem + kOffB + i * kChunkBytes; };
    float *bias = reinterpret_cast<float *>(smem + kOffBias);
    const unsigned char *w4img = reinterpret_cast<const unsigned char *>(p.pd.w4t);

    // weights and the first two logit chunks start moving
    copy_tile<kWeightImgBytes>(smem + kOffW1, reinterpret_cast<const unsigned char *>(p.pd.w123img));
    copy_tile<kChunkBytes>(btile(0), w4img);
    unsigned char *b4s = smem + kOffB4;
    const float b4_first = tid < min(nch, 2) * kChunkN ? __ldg(p.pd.b4e + tid) : 0.0f;  // placed once the x tile is free
    const unsigned char *b4img = reinterpret_cast<const unsigned char *>(p.pd.b4e);
    cp_async_commit();
    if (nch > 1) copy_tile<kChunkBytes>(btile(1), w4img + kChunkBytes);
    cp_async_commit();
    for (int i = tid; i < 3 * mlp::kH; i += blockDim.x) {
        const size_t b = i < mlp::kH ? L.b1 : i < 2 * mlp::kH ? L.b2 : L.b3;
        bias[i] = p.pd.params[b + (size_t)(i % mlp::kH)];
    }
    if (warp == 0) umma::tmem_alloc(&tmem_base, kCols);
    if (tid == 0) {
        umma::mbar_init(&mbar_layer, 1);
        umma::mbar_init(&mbar_chunk[0], 1);
        umma::mbar_init(&mbar_chunk[1], 1);
    }
    {
        float x[mlp::kIn];
        if (valid) {
            features(p.pd, wpos_plane, normal_plane, cx, cy, cz, px, x);
        } else {
#pragma unroll
            for (int i = 0; i < mlp::kIn; ++i) x[i] = 0.0f;
        }
        put8(xtile, tid, 0, mlp::kIn, x);
        put8(xtile, tid, 8, mlp::kIn, x + 8);
        if (kMode == kLse && p.save && valid) {
            store8(p.x + (size_t)row * mlp::kIn, x);
            store8(p.x + (size_t)row * mlp::kIn + 8, x + 8);
        }
    }

    // kSample: which candidate slots take the learned branch, and the learned
    // slots' uniforms as ascending order statistics, from the pixel's own PCG
    // stream (two draws per slot: branch, uniform light; then one per
    // learned slot).  The k-th smallest uniform goes to the k-th learned slot.
    uint32_t lmask = 0;  // learned slots not yet assigned
    Pcg rng{};
    if (kMode == kSample && valid) {
        rng = pcg_seed((uint64_t)frame * mlp::kSeedMul + mlp::kSeedAdd, (uint64_t)px);
        for (int j = 0; j < n_cand; ++j) {
            const float u0 = rand_float(rng);
            rand_float(rng);
            if (u0 < p.pd.mix) lmask |= 1u << j;
        }
    }

    cp_async_wait_one();
    umma::fence_proxy_async();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tmem_base;
    bool ok = true;
    // thread 0's most recent MMA commit (the barrier and the parity of that
    // phase): on a timeout it waits, bounded, for that commit, which covers
    // every MMA issued before it
    uint64_t *last_mbar = nullptr;
    uint32_t last_parity = 0;

    // ---- hidden layers: MMA into columns 64*l, epilogue into the h tile
    for (int l = 0; l < 3 && ok; ++l) {
        // layer l accumulates in columns 64*(l&1): layer 3 reuses layer 1's,
        // whose loads completed before the barrier that preceded layer 2
        const uint32_t lcol = tmem + (uint32_t)(64 * (l & 1));
        if (tid == 0) {
            umma::mma_chunk(lcol, l == 0 ? xtile : htile, smem + (l == 0 ? kOffW1 : l == 1 ? kOffW2 : kOffW3), l == 0 ? mlp::kIn : mlp::kH, kRows, mlp::kH, false);
            umma::mma_commit(&mbar_layer);
            last_mbar = &mbar_layer;
            last_parity = (uint32_t)(l & 1);
        }
        const bool w = mma_wait(&mbar_layer, (uint32_t)(l & 1));
        if (w) {
            // the first two chunks' biases; the barriers of this loop come before their use
            if (l == 1 && tid < min(nch, 2) * kChunkN) reinterpret_cast<float *>(b4s)[tid] = b4_first;
            float v[64];
            umma::tmem_ld32(lcol, warp, 0, *reinterpret_cast<float(*)[32]>(v));
            umma::tmem_ld32(lcol, warp, 32, *reinterpret_cast<float(*)[32]>(v + 32));
#pragma unroll
            for (int j = 0; j < 64; j += 4) {  // put8 rounds to bf16
                const float4 b = *reinterpret_cast<const float4 *>(bias + 64 * l + j);
                const float2 lo = __fadd2_rn(make_float2(v[j], v[j + 1]), make_float2(b.x, b.y)),
                             hi = __fadd2_rn(make_float2(v[j + 2], v[j + 3]), make_float2(b.z, b.w));
                v[j] = fmaxf(lo.x, 0.0f);
                v[j + 1] = fmaxf(lo.y, 0.0f);
                v[j + 2] = fmaxf(hi.x, 0.0f);
                v[j + 3] = fmaxf(hi.y, 0.0f);
            }
#pragma unroll
            for (int j = 0; j < 64; j += 8) put8(htile, tid, j, mlp::kH, v + j);
            if (kMode == kLse && p.save) {  // as the tile itself: eight rows' 16 bytes are one 128-byte line
                unsigned char *dst = reinterpret_cast<unsigned char *>(l == 0 ? p.h1 : l == 1 ? p.h2 : p.h3) + (size_t)blockIdx.x * kHTileBytes;
#pragma unroll
                for (int j = 0; j < 64; ++j) v[j] = valid ? v[j] : 0.0f;
#pragma unroll
                for (int j = 0; j < 64; j += 8) put8(dst, tid, j, mlp::kH, v + j);
            }
        }
        umma::fence_proxy_async();
        umma::fence_before_sync();
        ok = __syncthreads_and(w) != 0;
        umma::fence_after_sync();
    }

    // ---- logit chunks
    float m = -INFINITY, s = 0.0f;  // kLse: running max and sum
    int amax = 0;
    float lse = 0.0f, cum = 0.0f;   // kSample
    float next_u = INFINITY;  // the row's next uniform; INFINITY: none left (cum never exceeds it, even when it overflows)
    int amax_row = 0;
    float qmax_row = 0.0f;
    if (kMode == kSample && valid) {
        const float4 st = p.stat[row];
        lse = st.x;
        amax_row = __float_as_int(st.y);
        qmax_row = st.z;
    }
    const float nl2 = -lse * kLog2e;
    const float *uni = reinterpret_cast<const float *>(smem + kOffW1) + tid;  // kSample: the row's uniforms
    // kSample: the learned slot of the current uniform gets cluster col with q
    auto take = [&](int col, float q) {
        if (!(q > 0.0f)) {  // rounding put the uniform on an empty column: the most probable cluster
            col = amax_row;
            q = qmax_row;
        }
        const int slot = __ffs(lmask) - 1;
        lmask &= lmask - 1;
        p.cand[(size_t)row * mlp::kCand + slot] = mlp::Candidate{-1 - col, q};
        uni += kRows;
        next_u = *uni;
    };
    if (ok && tid == 0) {
        umma::mma_chunk(tmem, htile, btile(0), mlp::kH, kRows, kChunkN, false);
        umma::mma_commit(&mbar_chunk[0]);
        last_mbar = &mbar_chunk[0];
        last_parity = 0;
    }
    // all of a row's uniforms at once (inside the search only the rows with a
    // uniform in the piece would draw: ten times as many warp executions),
    // over the hidden layers' weights, whose last product has completed
    if (kMode == kSample && ok) {
        float *us = reinterpret_cast<float *>(smem + kOffW1) + tid;
        const int n_u = __popc(lmask);
        float u = 0.0f;
        for (int k = 0; k < n_u; ++k) us[k * kRows] = u = next_order_stat(rng, u, n_u - k);
        us[n_u * kRows] = INFINITY;
        next_u = us[0];
    }
    // Every warp passes the same barriers whatever fails: a warp whose wait ran
    // out (ok_warp) does no more work and no more waits, thread 0 then issues no
    // more products, and `ok` is settled after the chunks.
    bool ok_warp = ok;
    int slot = 0;  // c % 3
    for (int c = 0; ok && c < nch; ++c, slot = slot == 2 ? 0 : slot + 1) {
        if (c + 1 < nch) {
            cp_async_wait_all();
            umma::fence_proxy_async();
            umma::fence_before_sync();
            __syncthreads();
            umma::fence_after_sync();
            if (tid == 0 && ok_warp) {
                umma::mma_chunk(tmem + (uint32_t)(((c + 1) & 1) * kChunkN), htile, btile((c + 1) & 1), mlp::kH, kRows,
                                kChunkN, false);
                umma::mma_commit(&mbar_chunk[(c + 1) & 1]);
                last_mbar = &mbar_chunk[(c + 1) & 1];
                last_parity = (uint32_t)(((c + 1) >> 1) & 1);
            }
        }
        ok_warp = ok_warp && mma_wait(&mbar_chunk[c & 1], (uint32_t)((c >> 1) & 1));
        if (ok_warp) {
        if (c + 2 < nch) {
            copy_tile<kChunkBytes>(btile(c & 1), w4img + (size_t)(c + 2) * kChunkBytes);
            // chunk c - 1's biases, the third place, were last read before this chunk's barrier
            copy_tile<kB4Bytes>(b4s + (slot == 0 ? 2 : slot - 1) * kB4Bytes, b4img + (size_t)(c + 2) * kB4Bytes);
            cp_async_commit();
        }
        const uint32_t half = tmem + (uint32_t)((c & 1) * kChunkN);
        uint32_t raw[2][32];
        umma::tmem_ld32_issue(half, warp, 0, raw[0]);
#pragma unroll
        for (int piece = 0; piece < kChunkN / 32; ++piece) {
            umma::tmem_ld32_wait(raw[piece & 1]);
            // the next piece's load runs under this piece's arithmetic
            if (piece + 1 < kChunkN / 32) umma::tmem_ld32_issue(half, warp, (piece + 1) * 32, raw[(piece + 1) & 1]);
            const uint32_t(&rw)[32] = raw[piece & 1];
            const int col0 = c * kChunkN + piece * 32;
            const float4 *be = reinterpret_cast<const float4 *>(b4s + slot * kB4Bytes) + piece * 8;
            float2 v[16];  // logits z = MMA result + b4
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float4 b = be[q];
                v[2 * q] = __fadd2_rn(make_float2(__uint_as_float(rw[4 * q]), __uint_as_float(rw[4 * q + 1])),
                                      make_float2(b.x, b.y));
                v[2 * q + 1] = __fadd2_rn(make_float2(__uint_as_float(rw[4 * q + 2]), __uint_as_float(rw[4 * q + 3])),
                                          make_float2(b.z, b.w));
            }
            if (kMode == kLse) {
                float triple[11];
                const float mp = max32(v, triple);
                if (mp == -INFINITY) continue;
                if (mp > m) amax = col0 + first_max(v, triple, mp);
                exp_piece(v, -mp * kLog2e);
                const float sp = sum32(v);
                if (mp > m) {
                    s = (m == -INFINITY) ? sp : __fmaf_rn(s, ex2((m - mp) * kLog2e), sp);
                    m = mp;
                } else {
                    s = __fmaf_rn(sp, ex2((mp - m) * kLog2e), s);
                }
            } else {
                exp_piece(v, nl2);
                const float end = cum + sum32(v);
                // the uniforms below `end` belong to this piece
                if (valid && next_u < end) {
                    // running sums within the piece, left to right
                    float r[32];
                    r[0] = v[0].x;
#pragma unroll
                    for (int i = 1; i < 32; ++i) r[i] = r[i - 1] + col(v, i);
                    do {
                        // the column is the first whose running sum exceeds the
                        // uniform (at most the last), by binary search; its
                        // probability is the width of its interval
                        const float ul = next_u - cum;
                        float a[16];
                        int idx = 0;
                        float lo = 0.0f;
                        {
                            const bool b = r[15] <= ul;
                            lo = b ? r[15] : lo;
                            idx += b ? 16 : 0;
#pragma unroll
                            for (int j = 0; j < 16; ++j) a[j] = b ? r[16 + j] : r[j];
                        }
#pragma unroll
                        for (int h = 8; h >= 1; h >>= 1) {
                            const bool b = a[h - 1] <= ul;
                            lo = b ? a[h - 1] : lo;
                            idx += b ? h : 0;
#pragma unroll
                            for (int j = 0; j < h; ++j) a[j] = b ? a[h + j] : a[j];
                        }
                        take(col0 + idx, a[0] - lo);
                    } while (next_u < end);
                }
                cum = end;
            }
        }
        }  // ok_warp
        umma::fence_before_sync();
    }
    ok = __syncthreads_and(ok && ok_warp) != 0;
    if (!ok) {
        if (tid == 0) {
            atomicAdd(p.err, 1);
            if (last_mbar) umma::mbar_wait(last_mbar, last_parity, kMaxPolls);
        }
        cp_async_wait_all();
    } else if (valid) {
        if (kMode == kLse) {
            const float lse_row = m + __logf(s);
            p.stat[row] = make_float4(lse_row, __int_as_float(amax), ex2((m - lse_row) * kLog2e), 0.0f);
            if (p.cand) {
                // uniform-branch candidates: the light and q of its cluster (the
                // same PCG stream as the learned branch's draws in kSample)
                float h[64];
#pragma unroll
                for (int j = 0; j < 64; j += 8) {
                    const uint4 w = *reinterpret_cast<const uint4 *>(htile + umma::kmajor_offset(tid, j, mlp::kH));
                    const __nv_bfloat162 *b = reinterpret_cast<const __nv_bfloat162 *>(&w);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __bfloat1622float2(b[i]);
                        h[j + 2 * i] = f.x;
                        h[j + 2 * i + 1] = f.y;
                    }
                }
                rng = pcg_seed((uint64_t)frame * mlp::kSeedMul + mlp::kSeedAdd, (uint64_t)px);
                const float nl = -lse_row * kLog2e;
                // first the slots that take the uniform branch (about 1 in 10),
                // then one loop iteration per such slot of this row: the warp
                // runs as many dot products as its busiest row has slots, not
                // one per slot index that any row uses
                uint32_t umask = 0;
                float *us = reinterpret_cast<float *>(smem + kOffW1) + tid;  // their draws, over the hidden weights
                for (int j = 0; j < n_cand; ++j) {
                    const float u0 = rand_float(rng), u1 = rand_float(rng);
                    if (!(u0 < p.pd.mix)) {
                        *us = u1;
                        us += kRows;
                        umask |= 1u << j;
                    }
                }
                us = reinterpret_cast<float *>(smem + kOffW1) + tid;
                while (umask) {
                    const int j = __ffs(umask) - 1;
                    umask &= umask - 1;
                    const float u1 = *us;
                    us += kRows;
                    const int l = imin((int)((float)p.pd.n_lights * u1), p.pd.n_lights - 1);
                    const float z = logit_of(p.pd, h, __ldg(p.pd.cluster_of + l));
                    p.cand[(size_t)row * mlp::kCand + j] = mlp::Candidate{l, ex2(__fmaf_rn(z, kLog2e, nl))};
                }
            }
        } else {
            // uniforms beyond the rounded CDF total: the most probable cluster
            while (next_u < INFINITY) take(amax_row, qmax_row);
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, kCols);
}

// ---------------------------------------------------------------- training: dh3 and the loss
// One CTA per 128 rows: the forward pass from the saved h3, then per chunk of
// 64 clusters z = h3 . W4[:, chunk] on the tensor cores, dz = (softmax -
// onehot) / n as bf16 into a tile, and dh3 += dz W4[:, chunk]^T, accumulated
// in tensor memory.  Bound by the latency of that chain, so four CTAs share an
// SM (128 tensor-memory columns and 49 KB each): the weight tiles are single,
// each refilled under the epilogue that follows its product, and a chunk has
// one barrier, after which both products are issued (its dh3 and the next z).
// 65,536 rows and 4096 clusters are 512 CTAs: with two an SM (88 KB, two
// barriers a chunk, the hidden layers run again, the one-hot tested at every
// column) they took 0.315 ms in two rounds; now 0.149 ms in one.
constexpr int kGOffH = 0;                                  // h3 tile, 128 x 64 bf16
constexpr int kGOffDz = kGOffH + kRows * mlp::kH * 2;      // dz tile, 128 x 64 (K-major over clusters)
constexpr int kGOffB = kGOffDz + kRows * kChunkN * 2;      // W4^T chunk (cluster x hidden)
constexpr int kGOffWk = kGOffB + kChunkBytes;              // W4 chunk (hidden x cluster)
constexpr int kGradSmem = kGOffWk + kWkBytes;
constexpr int kGradTmem = 2 * kChunkN;                     // z, dh3

struct GradParams {
    mlp::ProposalDev pd;
    const __nv_bfloat16 *h3;   // by tiles of 128 rows
    const float4 *stat;        // per row: lse first
    const int32_t *target;     // cluster per row, -1: no target
    int n;
    float inv_n;
    float *dh3;                // [n x 64] FP32: d(loss)/d(h3)
    float *loss_sum;
    int *err;
};

__global__ void __launch_bounds__(128, 4) k_mlp_grad(const GradParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t mbar_z, mbar_dh;
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int row = blockIdx.x * kRows + tid;
    const bool valid = row < p.n;
    const int nch = p.pd.c / kChunkN;
    unsigned char *htile = smem + kGOffH, *dztile = smem + kGOffDz, *btile = smem + kGOffB, *wk = smem + kGOffWk;
    const unsigned char *w4img = reinterpret_cast<const unsigned char *>(p.pd.w4t);
    const unsigned char *w4kimg = reinterpret_cast<const unsigned char *>(p.pd.w4k);
    copy_tile<kChunkBytes>(btile, w4img);
    copy_tile<kWkBytes>(wk, w4kimg);
    copy_tile<kHTileBytes>(htile, reinterpret_cast<const unsigned char *>(p.h3) + (size_t)blockIdx.x * kHTileBytes);
    cp_async_commit();
    if (warp == 0) umma::tmem_alloc(&tmem_base, kGradTmem);
    if (tid == 0) {
        umma::mbar_init(&mbar_z, 1);
        umma::mbar_init(&mbar_dh, 1);
    }
    float lse = 0.0f, zt = 0.0f;
    int target = -1;
    if (valid) {
        lse = p.stat[row].x;
        target = p.target[row];
    }
    const float nl2 = -lse * kLog2e;
    cp_async_wait_all();
    umma::fence_proxy_async();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tmem_base;
    bool ok = true, ok_warp = true;
    uint64_t *last_mbar = nullptr;  // thread 0's most recent commit
    uint32_t last_parity = 0;
    if (tid == 0) {
        umma::mma_chunk(tmem, htile, btile, mlp::kH, kRows, kChunkN, false);
        umma::mma_commit(&mbar_z);
        last_mbar = &mbar_z;
    }
    for (int c = 0; c < nch; ++c) {
        const bool w = mma_wait(&mbar_z, (uint32_t)(c & 1));
        ok_warp = ok_warp && w;
        if (w) {
            if (c + 1 < nch) {  // the product has read its weights
                copy_tile<kChunkBytes>(btile, w4img + (size_t)(c + 1) * kChunkBytes);
                cp_async_commit();
            }
            const float4 *be = reinterpret_cast<const float4 *>(p.pd.b4e + c * kChunkN);
            uint32_t raw[2][32];
            umma::tmem_ld32_issue(tmem, warp, 0, raw[0]);
#pragma unroll
            for (int piece = 0; piece < kChunkN / 32; ++piece) {
                umma::tmem_ld32_wait(raw[piece & 1]);
                if (piece + 1 < kChunkN / 32) umma::tmem_ld32_issue(tmem, warp, (piece + 1) * 32, raw[(piece + 1) & 1]);
                const uint32_t(&rw)[32] = raw[piece & 1];
                float2 v[16];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float4 b = __ldg(be + piece * 8 + q);
                    v[2 * q] = __fadd2_rn(make_float2(__uint_as_float(rw[4 * q]), __uint_as_float(rw[4 * q + 1])),
                                          make_float2(b.x, b.y));
                    v[2 * q + 1] = __fadd2_rn(
                        make_float2(__uint_as_float(rw[4 * q + 2]), __uint_as_float(rw[4 * q + 3])), make_float2(b.z, b.w));
                }
                if (piece == 0 && c > 0) {  // the previous chunk's product has read the dz tile and its weights
                    const bool w2 = mma_wait(&mbar_dh, (uint32_t)((c - 1) & 1));
                    ok_warp = ok_warp && w2;
                    if (w2) {
                        copy_tile<kWkBytes>(wk, w4kimg + (size_t)c * kWkBytes);
                        cp_async_commit();
                    }
                }
                zt += grad_piece(dztile, tid, piece * 32, v, nl2, p.inv_n,
                                 target < 0 ? kNoTarget : target - (c * kChunkN + piece * 32));
            }
        }
        cp_async_wait_all();
        umma::fence_proxy_async();
        umma::fence_before_sync();
        ok = __syncthreads_and(ok_warp) != 0;
        umma::fence_after_sync();
        if (!ok) break;
        if (tid == 0) {
            umma::mma_chunk(tmem + (uint32_t)kChunkN, dztile, wk, kChunkN, kRows, mlp::kH, c > 0);
            umma::mma_commit(&mbar_dh);
            last_mbar = &mbar_dh;
            last_parity = (uint32_t)(c & 1);
            if (c + 1 < nch) {
                umma::mma_chunk(tmem, htile, btile, mlp::kH, kRows, kChunkN, false);
                umma::mma_commit(&mbar_z);
                last_mbar = &mbar_z;
                last_parity = (uint32_t)((c + 1) & 1);
            }
        }
    }
    if (ok) ok_warp = mma_wait(&mbar_dh, (uint32_t)((nch - 1) & 1)) && ok_warp;
    ok = __syncthreads_and(ok && ok_warp) != 0;
    if (!ok) {
        if (tid == 0) {
            atomicAdd(p.err, 1);
            if (last_mbar) umma::mbar_wait(last_mbar, last_parity, kMaxPolls);
        }
        cp_async_wait_all();
    } else {
        float d[64];
        umma::tmem_ld32(tmem + (uint32_t)kChunkN, warp, 0, *reinterpret_cast<float(*)[32]>(d));
        umma::tmem_ld32(tmem + (uint32_t)kChunkN, warp, 32, *reinterpret_cast<float(*)[32]>(d + 32));
        if (valid) {
            float4 *dst = reinterpret_cast<float4 *>(p.dh3 + (size_t)row * mlp::kH);
#pragma unroll
            for (int j = 0; j < 16; ++j) dst[j] = make_float4(d[4 * j], d[4 * j + 1], d[4 * j + 2], d[4 * j + 3]);
        }
        float l = (valid && target >= 0) ? lse - zt : 0.0f;
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if ((tid & 31) == 0 && l != 0.0f) atomicAdd(p.loss_sum, l);
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, kGradTmem);
}

// ---------------------------------------------------------------- dW4, db4
// One CTA per (chunk of 64 clusters, slice of row tiles).  Per 128-row tile:
// the chunk's logits z = h3 . W4[:, chunk] on the tensor cores, the bf16
// gradient dz = (softmax - onehot) / n as in k_mlp_grad (same formula, so the same
// values), then dW[0..63] += h3^T dz and dW[64] += 1^T dz (db4) as one MMA
// with M = 128 and K = the tile's 128 rows, accumulated in tensor memory; the
// CTA adds its 65 x 64 result to the gradient with atomics at the end.
//
// No operand is transposed element by element: the h tile (rows x [h3 | 1 |
// 0], K-major over its 72 columns) and the dz tile (rows x clusters, K-major
// over clusters) are read a second time through MN-major descriptors, as
// [h3 | 1 | 0]^T (M, K = rows) and dz^T (N = clusters, K = rows): in the
// canonical no-swizzle layouts a core matrix is 8 rows of 16 bytes either way,
// with SBO the step between core matrices along M/N and LBO the step along K.
// M is 128, so columns 72..127 of that operand are the next row groups' (past
// the last one, the bytes behind the tile): they only reach product rows 72 to
// 127, which nothing reads.
//
// Bound by the latency of a tile's chain (products, logits out, dz in) at
// three CTAs an SM, so the next tile's logits are issued behind this tile's
// product after the one barrier, from a second h tile, and that tile travels
// in registers meanwhile.  h3 comes in the tile's own layout: rows of a plain
// matrix cost 33 cycles of the load pipe per instruction, and their transposed
// stores conflict.  65,536 rows x 4096 clusters: 0.152 ms; 0.289 with one h tile,
// two barriers and plain rows, 0.20 with 256 threads and two CTAs an SM.

// dst[0..3] += v[0..3], dst on a 16-byte boundary
__device__ __forceinline__ void red_add4(float *dst, const float *v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
                 : "memory");
}

struct Dw4Params {
    mlp::ProposalDev pd;
    const __nv_bfloat16 *h3;   // by tiles of 128 rows
    const float4 *stat;        // lse per row
    const int32_t *target;
    int n, tiles_per_slice;
    float inv_n;
    float *gw4, *gb4;          // gradient blocks of W4 (64 x C) and b4
    int *err;
};

constexpr int kDwHCols = 72;                                 // h tile columns: h3 (64) | 1 | 0 ... 0
constexpr int kDwHBytes = kRows * kDwHCols * 2;
constexpr int kDwOffH = 0;                                   // two h tiles, 128 rows x 72 (K-major, 18 KB each)
constexpr int kDwOffDz = kDwOffH + 2 * kDwHBytes;            // dz tile, 128 rows x 64 (K-major, 16 KB)
constexpr int kDwOffBz = kDwOffDz + kRows * kChunkN * 2;     // W4^T chunk, 64 x 64 (K-major, 8 KB)
constexpr int kDwSmem = kDwOffBz + kChunkBytes;
constexpr int kDwCtas = 3;                                   // resident per SM (shared memory, registers)

// kind::f16 instruction descriptor with both operands MN-major (bits 15, 16)
__device__ __forceinline__ uint32_t idesc_mn_major(int m, int n) {
    return umma::idesc_bf16_f32(m, n) | (1u << 15) | (1u << 16);
}

__global__ void __launch_bounds__(kRows, kDwCtas) k_mlp_dw4(const Dw4Params p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t mbar_z, mbar_w;
    __shared__ uint32_t tmem_base;
    __shared__ __align__(16) float bias[kChunkN];
    const int tid = threadIdx.x, warp = tid >> 5;
    const int chunk = blockIdx.x;
    const int t0 = blockIdx.y * p.tiles_per_slice;
    const int t1 = min((p.n + kRows - 1) / kRows, t0 + p.tiles_per_slice);
    unsigned char *ht = smem + kDwOffH, *dzt = smem + kDwOffDz, *bz = smem + kDwOffBz;
    copy_tile<kChunkBytes>(bz, reinterpret_cast<const unsigned char *>(p.pd.w4t) + (size_t)chunk * kChunkBytes);
    cp_async_commit();
    for (int r = tid; r < 2 * kRows; r += kRows) {  // columns 64..71 of both tiles: 1 (the db4 row of the product), zeros
        __align__(16) __nv_bfloat16 one[8];
        one[0] = __float2bfloat16_rn(1.0f);
#pragma unroll
        for (int i = 1; i < 8; ++i) one[i] = __float2bfloat16_rn(0.0f);
        *reinterpret_cast<uint4 *>(ht + (r / kRows) * kDwHBytes + umma::kmajor_offset(r % kRows, 64, kDwHCols)) =
            *reinterpret_cast<const uint4 *>(one);
    }
    if (tid < kChunkN) bias[tid] = __ldg(p.pd.b4e + chunk * kChunkN + tid);
    if (warp == 0) umma::tmem_alloc(&tmem_base, 128);
    if (tid == 0) {
        umma::mbar_init(&mbar_z, 1);
        umma::mbar_init(&mbar_w, 1);
    }
    // a saved tile travels in registers under the work on the tile before it
    constexpr int kPer = kHTileBytes / 16 / kRows;
    uint4 hrow[kPer];
    auto fetch_tile = [&](int t) {
        if (t >= t1) return;
        const uint4 *src = reinterpret_cast<const uint4 *>(p.h3) + (size_t)t * (kHTileBytes / 16);
#pragma unroll
        for (int i = 0; i < kPer; ++i) hrow[i] = __ldg(src + i * kRows + tid);
    };
    auto put_tile = [&](int buf) {  // 64 pieces of 16 bytes a row group, then the group's columns 64..71
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int q = i * kRows + tid;
            *reinterpret_cast<uint4 *>(ht + buf * kDwHBytes + (q >> 6) * (8 * kDwHCols * 2) + (q & 63) * 16) = hrow[i];
        }
    };
    float lse = 0.0f;   // of this thread's row of the next tile
    int target = -1;
    auto fetch_stat = [&](int t) {
        const int row = t * kRows + tid;
        const bool valid = t < t1 && row < p.n;
        target = valid ? __ldg(p.target + row) : -1;
        lse = valid ? __ldg(reinterpret_cast<const float *>(p.stat + row)) : 0.0f;
    };
#pragma unroll
    for (int i = 0; i < kPer; ++i) hrow[i] = make_uint4(0, 0, 0, 0);
    fetch_tile(t0);
    fetch_stat(t0);
    put_tile(0);
    fetch_tile(t0 + 1);
    cp_async_wait_all();
    umma::fence_proxy_async();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tmem_base;
    bool ok = t0 < t1, ok_warp = true;
    uint64_t *last_mbar = nullptr;
    uint32_t last_parity = 0;
    const float4 *be = reinterpret_cast<const float4 *>(bias);
    const uint32_t ht_a = umma::smem_addr(ht), dz_a = umma::smem_addr(dzt), bz_a = umma::smem_addr(bz);
    // z = h3 . W4[:, chunk]: A = h tile (K-major, first 64 columns), B = W4^T chunk
    auto issue_z = [&](int k) {
        const uint32_t idesc = umma::idesc_bf16_f32(kRows, kChunkN), a = ht_a + (uint32_t)((k & 1) * kDwHBytes);
#pragma unroll
        for (int ks = 0; ks < mlp::kH / 16; ++ks)
            umma::mma_bf16(tmem, umma::smem_desc(a + (uint32_t)ks * 256u, 128u, (kDwHCols / 8) * 128u),
                           umma::smem_desc(bz_a + (uint32_t)ks * 256u, 128u, (mlp::kH / 8) * 128u), idesc, ks > 0);
        umma::mma_commit(&mbar_z);
        last_mbar = &mbar_z;
        last_parity = (uint32_t)(k & 1);
    };
    if (ok && tid == 0) issue_z(0);
    for (int t = t0; t < t1 && ok; ++t) {
        const int k = t - t0;
        const float nl2 = -lse * kLog2e;
        const int hit = target < 0 ? kNoTarget : target - chunk * kChunkN;
        fetch_stat(t + 1);
        const bool w = mma_wait(&mbar_z, (uint32_t)(k & 1));
        ok_warp = ok_warp && w;
        if (w) {
#pragma unroll
            for (int piece = 0; piece < kChunkN / 32; ++piece) {
                uint32_t raw[32];
                umma::tmem_ld32_issue(tmem, warp, piece * 32, raw);
                umma::tmem_ld32_wait(raw);
                float2 v[16];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float4 b = be[piece * 8 + q];
                    v[2 * q] = __fadd2_rn(make_float2(__uint_as_float(raw[4 * q]), __uint_as_float(raw[4 * q + 1])),
                                          make_float2(b.x, b.y));
                    v[2 * q + 1] = __fadd2_rn(
                        make_float2(__uint_as_float(raw[4 * q + 2]), __uint_as_float(raw[4 * q + 3])), make_float2(b.z, b.w));
                }
                if (piece == 0) {  // the previous product has read the dz tile and the other h tile
                    if (k > 0) ok_warp = mma_wait(&mbar_w, (uint32_t)((k - 1) & 1)) && ok_warp;
                    put_tile((k + 1) & 1);
                    fetch_tile(t + 2);
                }
                grad_piece(dzt, tid, piece * 32, v, nl2, p.inv_n,
                           hit == kNoTarget ? kNoTarget : hit - piece * 32);
            }
        }
        umma::fence_proxy_async();
        umma::fence_before_sync();
        ok = __syncthreads_and(ok_warp) != 0;
        umma::fence_after_sync();
        if (!ok) break;
        if (tid == 0) {
            // dW += [h3 | 1 | 0]^T dz: both tiles through MN-major descriptors,
            // K = the tile's rows in steps of 16 (two core matrices along K)
            const uint32_t idesc = idesc_mn_major(128, kChunkN), a = ht_a + (uint32_t)((k & 1) * kDwHBytes);
            constexpr uint32_t lbo_h = 8 * kDwHCols * 2, lbo_dz = 8 * kChunkN * 2;  // K step: 8 rows of a tile
#pragma unroll
            for (int ks = 0; ks < kRows / 16; ++ks)
                umma::mma_bf16(tmem + 64, umma::smem_desc(a + (uint32_t)ks * 2u * lbo_h, lbo_h, 128u),
                               umma::smem_desc(dz_a + (uint32_t)ks * 2u * lbo_dz, lbo_dz, 128u), idesc,
                               k > 0 || ks > 0);
            umma::mma_commit(&mbar_w);
            last_mbar = &mbar_w;
            last_parity = (uint32_t)(k & 1);
            if (t + 1 < t1) issue_z(k + 1);
        }
    }
    if (ok && t1 > t0) ok_warp = mma_wait(&mbar_w, (uint32_t)((t1 - t0 - 1) & 1)) && ok_warp;
    ok = __syncthreads_and(ok && ok_warp) != 0;
    if (!ok && t1 > t0) {
        if (tid == 0) {
            atomicAdd(p.err, 1);
            if (last_mbar) umma::mbar_wait(last_mbar, last_parity, kMaxPolls);
        }
    } else if (ok && warp < 3) {
        // lanes 0..63: dW4 rows (hidden unit), lane 64: db4
        const int m = tid;
#pragma unroll
        for (int piece = 0; piece < kChunkN / 32; ++piece) {
            float v[32];
            umma::tmem_ld32(tmem + 64, warp, piece * 32, v);
            if (m <= 64) {
                float *dst = m < 64 ? p.gw4 + (size_t)m * p.pd.c + chunk * kChunkN + piece * 32
                                    : p.gb4 + chunk * kChunkN + piece * 32;
#pragma unroll
                for (int i = 0; i < 32; i += 4) red_add4(dst + i, v + i);
            }
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, 128);
}

// ---------------------------------------------------------------- training helpers
struct BackParams {
    const __nv_bfloat16 *w123;        // bf16 W1 | W2 | W3, row-major (row = input)
    const __nv_bfloat16 *x, *h1, *h2, *h3;
    const float *dh3;
    float *gw1, *gw2, *gw3;           // weight gradients (16 x 64, 64 x 64, 64 x 64), added
    float *gb1, *gb2, *gb3;           // bias gradients, added
    int n;
};

constexpr int kTileStride = 68;  // floats per row of the row tiles (16-byte rows, conflict-free)
constexpr int kBackThreads = 256;
// W2^T, W3^T, the da tile and the layer-input tile (128 rows each)
constexpr int kBackSmem = (2 * mlp::kH * mlp::kH + 2 * 128 * kTileStride) * 4;

// Two columns of FP32 FMAs: acc[j] += a * b[j].
__device__ __forceinline__ void fma4(float2 (&acc)[2], float a, const float4 &b) {
    const float2 a2 = make_float2(a, a);
    acc[0] = __ffma2_rn(a2, make_float2(b.x, b.y), acc[0]);
    acc[1] = __ffma2_rn(a2, make_float2(b.z, b.w), acc[1]);
}

// The rows of a bf16 matrix with W columns into the tile's first W columns.
template <int W>
__device__ __forceinline__ void load_tile(float *tile, const __nv_bfloat16 *src, int row0, int n) {
    for (int e = threadIdx.x; e < 128 * (W / 8); e += kBackThreads) {
        const int r = e / (W / 8), c = (e % (W / 8)) * 8;
        uint4 w = make_uint4(0, 0, 0, 0);
        if (row0 + r < n) w = *reinterpret_cast<const uint4 *>(src + (size_t)(row0 + r) * W + c);
        const __nv_bfloat162 *b = reinterpret_cast<const __nv_bfloat162 *>(&w);
        float4 *d = reinterpret_cast<float4 *>(tile + r * kTileStride + c);
        const float2 f0 = __bfloat1622float2(b[0]), f1 = __bfloat1622float2(b[1]), f2 = __bfloat1622float2(b[2]),
                     f3 = __bfloat1622float2(b[3]);
        d[0] = make_float4(f0.x, f0.y, f1.x, f1.y);
        d[1] = make_float4(f2.x, f2.y, f3.x, f3.y);
    }
}

// The same for a saved hidden layer (128 rows laid out as the MMA operand tile).
__device__ __forceinline__ void load_h_tile(float *tile, const __nv_bfloat16 *src) {
    const uint4 *img = reinterpret_cast<const uint4 *>(src) + (size_t)blockIdx.x * (kHTileBytes / 16);
    for (int e = threadIdx.x; e < kHTileBytes / 16; e += kBackThreads) {
        const uint4 w = __ldg(img + e);
        const __nv_bfloat162 *b = reinterpret_cast<const __nv_bfloat162 *>(&w);
        float4 *d = reinterpret_cast<float4 *>(tile + ((e >> 6) * 8 + (e & 7)) * kTileStride + ((e >> 3) & 7) * 8);
        const float2 f0 = __bfloat1622float2(b[0]), f1 = __bfloat1622float2(b[1]), f2 = __bfloat1622float2(b[2]),
                     f3 = __bfloat1622float2(b[3]);
        d[0] = make_float4(f0.x, f0.y, f1.x, f1.y);
        d[1] = make_float4(f2.x, f2.y, f3.x, f3.y);
    }
}

// The hidden layers' backward pass for 128 rows per block: da3 = dh3
// relu'(h3); for l = 3, 2, 1: db_l += column sums of da_l, dW_l += in_l^T da_l
// (in_3 = h2, in_2 = h1, in_1 = x), and da_{l-1} = (W_l da_l) relu'(h_{l-1}),
// FP32 with the bf16 weights of the forward pass.  The weight and bias
// gradients are added to the output with atomics, once per block.
//
// Bound by shared-memory reads, so a thread owns a register tile of each
// product: 4 x 4 of dW (two 16-byte reads for 16 FMAs a row) and 8 rows x 4
// columns of da (12 reads for 128 FMAs every four terms).  One row per thread
// read nine and four values for 32 and 16 FMAs: 65,536 rows took 0.241 ms, now
// 0.107.
__global__ void __launch_bounds__(kBackThreads, 2) k_mlp_backward_rows(const BackParams p) {
    extern __shared__ __align__(16) float bsm[];
    float *wt2 = bsm, *wt3 = bsm + mlp::kH * mlp::kH;
    float *dt = bsm + 2 * mlp::kH * mlp::kH, *it = dt + 128 * kTileStride;  // da tile, layer-input tile
    const int t = threadIdx.x, row0 = blockIdx.x * 128;
    for (int e = t; e < 2 * mlp::kH * mlp::kH; e += kBackThreads) {
        const int layer = e / (mlp::kH * mlp::kH), f = e % (mlp::kH * mlp::kH);
        const int i = f / mlp::kH, k = f % mlp::kH;  // W[i][k]
        (layer ? wt3 : wt2)[k * mlp::kH + i] = __bfloat162float(p.w123[mlp::kIn * mlp::kH + e]);
    }
    load_h_tile(it, p.h3);
    __syncthreads();
    for (int e = t; e < 128 * 16; e += kBackThreads) {  // da3
        const int r = e >> 4, c = (e & 15) * 4;
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row0 + r < p.n) {
            g = *reinterpret_cast<const float4 *>(p.dh3 + (size_t)(row0 + r) * mlp::kH + c);
            const float4 h = *reinterpret_cast<const float4 *>(it + r * kTileStride + c);
            g = make_float4(h.x > 0.0f ? g.x : 0.0f, h.y > 0.0f ? g.y : 0.0f, h.z > 0.0f ? g.z : 0.0f,
                            h.w > 0.0f ? g.w : 0.0f);
        }
        *reinterpret_cast<float4 *>(dt + r * kTileStride + c) = g;
    }
    const int c0 = (t & 15) * 4, g0 = t >> 4;  // this thread's 4 columns, its group of 16 threads
#pragma unroll 1
    for (int layer = 3; layer >= 1; --layer) {
        __syncthreads();  // da is complete and the input tile no longer read
        if (layer == 3) load_h_tile(it, p.h2);
        else if (layer == 2) load_h_tile(it, p.h1);
        else load_tile<mlp::kIn>(it, p.x, row0, p.n);
        __syncthreads();
        if (t < 128) {  // db_l: thread t sums half the rows of column t % 64
            const int c = t & 63, half = t >> 6;
            float sum = 0.0f;
#pragma unroll 8
            for (int q = 0; q < 64; ++q) sum += dt[(half * 64 + q) * kTileStride + c];
            atomicAdd((layer == 3 ? p.gb3 : layer == 2 ? p.gb2 : p.gb1) + c, sum);
        }
        if (layer == 1) {  // dW1, 16 x 64: one row of four columns a thread
            float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll 4
            for (int r = 0; r < 128; ++r)
                fma4(acc, it[r * kTileStride + g0], *reinterpret_cast<const float4 *>(dt + r * kTileStride + c0));
            float *dst = p.gw1 + g0 * mlp::kH + c0;
            atomicAdd(dst, acc[0].x);
            atomicAdd(dst + 1, acc[0].y);
            atomicAdd(dst + 2, acc[1].x);
            atomicAdd(dst + 3, acc[1].y);
            break;
        }
        {  // dW_l, 64 x 64: rows 4 g0 .. 4 g0 + 3, columns c0 .. c0 + 3
            float2 acc[4][2];
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);
#pragma unroll 4
            for (int r = 0; r < 128; ++r) {
                const float4 a = *reinterpret_cast<const float4 *>(it + r * kTileStride + 4 * g0);
                const float4 d = *reinterpret_cast<const float4 *>(dt + r * kTileStride + c0);
                fma4(acc[0], a.x, d);
                fma4(acc[1], a.y, d);
                fma4(acc[2], a.z, d);
                fma4(acc[3], a.w, d);
            }
            float *gw = (layer == 3 ? p.gw3 : p.gw2) + 4 * g0 * mlp::kH + c0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                atomicAdd(gw + i * mlp::kH, acc[i][0].x);
                atomicAdd(gw + i * mlp::kH + 1, acc[i][0].y);
                atomicAdd(gw + i * mlp::kH + 2, acc[i][1].x);
                atomicAdd(gw + i * mlp::kH + 3, acc[i][1].y);
            }
        }
        // da_{l-1}: rows 8 g0 .. 8 g0 + 7, columns c0 .. c0 + 3
        const float *wt = layer == 3 ? wt3 : wt2;
        float2 acc[8][2];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j][0] = acc[j][1] = make_float2(0.f, 0.f);
#pragma unroll 2
        for (int k = 0; k < mlp::kH; k += 4) {
            float4 w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) w[q] = *reinterpret_cast<const float4 *>(wt + (k + q) * mlp::kH + c0);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 d = *reinterpret_cast<const float4 *>(dt + (8 * g0 + j) * kTileStride + k);
                fma4(acc[j], d.x, w[0]);
                fma4(acc[j], d.y, w[1]);
                fma4(acc[j], d.z, w[2]);
                fma4(acc[j], d.w, w[3]);
            }
        }
        __syncthreads();  // every thread has read da
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int r = 8 * g0 + j;
            const float4 h = *reinterpret_cast<const float4 *>(it + r * kTileStride + c0);
            *reinterpret_cast<float4 *>(dt + r * kTileStride + c0) =
                make_float4(h.x > 0.0f ? acc[j][0].x : 0.0f, h.y > 0.0f ? acc[j][0].y : 0.0f,
                            h.z > 0.0f ? acc[j][1].x : 0.0f, h.w > 0.0f ? acc[j][1].y : 0.0f);
        }
    }
}

__global__ void k_adam(float *w, const float *g, float *m, float *v, size_t n, float lr, float b1, float b2,
                       float eps, float c1, float c2, size_t w1_pad_begin, size_t w1_pad_end) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || (i >= w1_pad_begin && i < w1_pad_end)) return;  // padded inputs stay zero
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * (gi * gi);
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// bf16 images of the weights: W1^T | W2^T | W3^T in the MMA operand layout
// (w123img), W4^T in chunk tiles (w4t: cluster x hidden, K-major over
// hidden), W4 in chunk tiles (w4k: hidden x cluster, K-major over clusters),
// W1 | W2 | W3 row-major (w123), W4 row-major (w4), and b4 with -inf for
// clusters without lights.
__global__ void k_refresh(const float *params, int c, const uint8_t *valid, __nv_bfloat16 *w123img,
                          __nv_bfloat16 *w4t, __nv_bfloat16 *w4k, __nv_bfloat16 *w123, __nv_bfloat16 *w4,
                          float *b4e) {
    const mlp::Layout L(c);
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t n1 = (size_t)mlp::kIn * mlp::kH, n2 = (size_t)mlp::kH * mlp::kH;
    unsigned char *img = reinterpret_cast<unsigned char *>(w123img);
    if (i < n1) {  // W1[k][n]
        const int k = (int)(i / mlp::kH), nn = (int)(i % mlp::kH);
        const __nv_bfloat16 b = __float2bfloat16_rn(params[L.w1 + i]);
        w123[i] = b;
        *reinterpret_cast<__nv_bfloat16 *>(img + umma::kmajor_offset(nn, k, mlp::kIn)) = b;
    } else if (i < n1 + 2 * n2) {
        const size_t j = i - n1;
        const int layer = (int)(j / n2);
        const size_t e = j % n2;
        const int k = (int)(e / mlp::kH), nn = (int)(e % mlp::kH);
        const __nv_bfloat16 b = __float2bfloat16_rn(params[(layer == 0 ? L.w2 : L.w3) + e]);
        w123[i] = b;
        *reinterpret_cast<__nv_bfloat16 *>(img + n1 * 2 + (size_t)layer * n2 * 2 +
                                           umma::kmajor_offset(nn, k, mlp::kH)) = b;
    } else if (i < n1 + 2 * n2 + (size_t)mlp::kH * c) {
        const size_t e = i - n1 - 2 * n2;  // W4[k][cl]
        const int k = (int)(e / (size_t)c), cl = (int)(e % (size_t)c);
        const __nv_bfloat16 b = __float2bfloat16_rn(params[L.w4 + e]);
        w4[e] = b;
        unsigned char *tile = reinterpret_cast<unsigned char *>(w4t) + (size_t)(cl / kChunkN) * kChunkBytes;
        *reinterpret_cast<__nv_bfloat16 *>(tile + umma::kmajor_offset(cl % kChunkN, k, mlp::kH)) = b;
        unsigned char *ktile = reinterpret_cast<unsigned char *>(w4k) + (size_t)(cl / kChunkN) * kWkBytes;
        *reinterpret_cast<__nv_bfloat16 *>(ktile + umma::kmajor_offset(k, cl % kChunkN, kChunkN)) = b;
    } else if (i < n1 + 2 * n2 + (size_t)(mlp::kH + 1) * c) {
        const size_t cl = i - n1 - 2 * n2 - (size_t)mlp::kH * c;
        b4e[cl] = valid[cl] ? params[L.b4 + cl] : -INFINITY;
    }
}

// Training target of each row: the cluster of its final reservoir's light,
// or -1 (no light kept).
__global__ void k_targets(const rg_reservoir *res, const int32_t *rows, int n, const int32_t *cluster_of,
                          int n_lights, int32_t *target, int *count) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const float4 c = __ldg(reinterpret_cast<const float4 *>(res + rows[r]) + 2);
    const int idx = __float_as_int(c.x);
    int t = -1;
    if (c.w > 0.0f && idx >= 0 && idx < n_lights) t = cluster_of[idx];
    target[r] = t;
    if (t >= 0) atomicAdd(count, 1);
}

// Training rows of one frame: a strided sweep over the pixels.
__global__ void k_batch_rows(int32_t *rows, int n, uint32_t pixels, uint32_t offset, uint32_t stride) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    rows[r] = (int32_t)(((uint64_t)r * stride + offset) % pixels);
}

__global__ void k_check_rows(const int32_t *rows, const int32_t *targets, int n, int64_t pixels, int c, uint32_t *bad) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    if (rows[r] < 0 || rows[r] >= pixels) atomicMin(bad, (uint32_t)r);
    if (targets[r] < -1 || targets[r] >= c) atomicMin(bad + 1, (uint32_t)r);
}

constexpr int kFusedSmem = kSmemUsed < kSmemMin ? kSmemMin : kSmemUsed;

// set_attr: set the shared-memory attribute first (the batched launches set it
// once, before any stream capture, in prepare_views)
template <int kMode, bool kViews = false>
cudaError_t launch_fused(const FusedParams &p, cudaStream_t st, bool set_attr = true) {
    if (p.pd.c % kChunkN != 0 || p.pd.c < kChunkN) return cudaErrorInvalidValue;
    constexpr int smem = kFusedSmem;
    if (set_attr) {
        cudaError_t e =
            cudaFuncSetAttribute(k_mlp_fused<kMode, kViews>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
    }
    if (p.n > 0) k_mlp_fused<kMode, kViews><<<(p.n + kRows - 1) / kRows, kRows, smem, st>>>(p);
    return cudaGetLastError();
}

}  // namespace

// ---------------------------------------------------------------- launchers (mlp.cuh)
namespace mlp {

size_t weight_image_bytes() { return (size_t)kWeightImgBytes; }

cudaError_t forward_lse(const ProposalDev &pd, const GBufView &g, const float cam[3], const int32_t *rows, int n,
                        float4 *stat, const TrainBuffers *save, uint32_t frame, int n_cand, Candidate *cand, int *err,
                        cudaStream_t st) {
    if (cand && (n_cand < 1 || n_cand > kCand)) return cudaErrorInvalidValue;
    FusedParams p{};
    p.pd = pd; p.g = g; p.cam[0] = cam[0]; p.cam[1] = cam[1]; p.cam[2] = cam[2];
    p.rows = rows; p.n = n; p.stat = stat; p.err = err;
    p.frame = frame; p.n_cand = n_cand; p.cand = cand;
    if (save) { p.save = 1; p.x = save->x; p.h1 = save->h1; p.h2 = save->h2; p.h3 = save->h3; }
    return launch_fused<kLse>(p, st);
}

cudaError_t forward_sample(const ProposalDev &pd, const GBufView &g, const float cam[3], int n, const float4 *stat,
                           uint32_t frame, int n_cand, Candidate *cand, int *err, cudaStream_t st) {
    if (n_cand < 1 || n_cand > kCand) return cudaErrorInvalidValue;
    FusedParams p{};
    p.pd = pd; p.g = g; p.cam[0] = cam[0]; p.cam[1] = cam[1]; p.cam[2] = cam[2];
    p.n = n; p.stat = const_cast<float4 *>(stat); p.frame = frame; p.n_cand = n_cand; p.cand = cand; p.err = err;
    return launch_fused<kSample>(p, st);
}

cudaError_t prepare_views() {
    cudaError_t e = cudaFuncSetAttribute(k_mlp_fused<kLse, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kFusedSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_mlp_fused<kSample, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kFusedSmem);
    return e;
}

cudaError_t forward_lse_views(const ProposalDev &pd, const ViewRows *views, int n_views, const uint32_t *frames,
                              int total, float4 *stat, Candidate *cand, int *err, cudaStream_t st) {
    if (!views || n_views < 1 || !frames || !cand) return cudaErrorInvalidValue;
    FusedParams p{};
    p.pd = pd; p.n = total; p.stat = stat; p.err = err; p.cand = cand;
    p.views = views; p.n_views = n_views; p.frames = frames;
    return launch_fused<kLse, true>(p, st, false);
}

cudaError_t forward_sample_views(const ProposalDev &pd, const ViewRows *views, int n_views, const uint32_t *frames,
                                 int total, const float4 *stat, Candidate *cand, int *err, cudaStream_t st) {
    if (!views || n_views < 1 || !frames || !cand) return cudaErrorInvalidValue;
    FusedParams p{};
    p.pd = pd; p.n = total; p.stat = const_cast<float4 *>(stat); p.err = err; p.cand = cand;
    p.views = views; p.n_views = n_views; p.frames = frames;
    return launch_fused<kSample, true>(p, st, false);
}

cudaError_t forward_grad(const ProposalDev &pd, const __nv_bfloat16 *h3, int n, const float4 *stat,
                         const int32_t *target, float inv_n, float *dh3, float *loss_sum, int *err, cudaStream_t st) {
    const GradParams p{pd, h3, stat, target, n, inv_n, dh3, loss_sum, err};
    if (pd.c % kChunkN != 0 || pd.c < kChunkN) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, kGradSmem);
    if (e != cudaSuccess) return e;
    if (n > 0) k_mlp_grad<<<(n + kRows - 1) / kRows, kRows, kGradSmem, st>>>(p);
    return cudaGetLastError();
}

cudaError_t dw4(const ProposalDev &pd, const __nv_bfloat16 *h3, const float4 *stat, const int32_t *target, int n,
                float inv_n, float *gw4, float *gb4, int *err, cudaStream_t st) {
    if (pd.c % kChunkN != 0 || n <= 0) return cudaErrorInvalidValue;
    Dw4Params p{pd, h3, stat, target, n, 0, inv_n, gw4, gb4, err};
    const int tiles = (n + kRows - 1) / kRows;
    const int chunks = pd.c / kChunkN;
    // as many slices as keep every CTA resident at once: a second round of a few
    // CTAs costs as much as a full one
    int slices = kDwCtas * 152 / chunks;
    if (slices < 1) slices = 1;
    if (slices > tiles) slices = tiles;
    p.tiles_per_slice = (tiles + slices - 1) / slices;
    slices = (tiles + p.tiles_per_slice - 1) / p.tiles_per_slice;
    cudaError_t e = cudaFuncSetAttribute(k_mlp_dw4, cudaFuncAttributeMaxDynamicSharedMemorySize, kDwSmem);
    if (e != cudaSuccess) return e;
    k_mlp_dw4<<<dim3(chunks, slices), kRows, kDwSmem, st>>>(p);
    return cudaGetLastError();
}

cudaError_t backward_rows(const __nv_bfloat16 *w123, const TrainBuffers &t, const float *dh3, float *gw1, float *gw2,
                          float *gw3, float *gb1, float *gb2, float *gb3, int n, cudaStream_t st) {
    BackParams p{w123, t.x, t.h1, t.h2, t.h3, dh3, gw1, gw2, gw3, gb1, gb2, gb3, n};
    cudaError_t e = cudaFuncSetAttribute(k_mlp_backward_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, kBackSmem);
    if (e != cudaSuccess) return e;
    if (n > 0) k_mlp_backward_rows<<<(n + 127) / 128, kBackThreads, kBackSmem, st>>>(p);
    return cudaGetLastError();
}

cudaError_t adam(float *w, const float *g, float *m, float *v, size_t n, float lr, int step, int c, cudaStream_t st) {
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
    const Layout L(c);
    k_adam<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(w, g, m, v, n, lr, b1, b2, 1e-8f, c1, c2,
                                                         L.w1 + (size_t)kInUsed * kH, L.w1 + (size_t)kIn * kH);
    return cudaGetLastError();
}

cudaError_t refresh(const float *params, int c, const uint8_t *valid, __nv_bfloat16 *w123img, __nv_bfloat16 *w4t,
                    __nv_bfloat16 *w4k, __nv_bfloat16 *w123, __nv_bfloat16 *w4, float *b4e, cudaStream_t st) {
    const size_t n = (size_t)kIn * kH + 2 * (size_t)kH * kH + (size_t)(kH + 1) * c;
    k_refresh<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(params, c, valid, w123img, w4t, w4k, w123, w4, b4e);
    return cudaGetLastError();
}

cudaError_t targets(const rg_reservoir *res, const int32_t *rows, int n, const int32_t *cluster_of, int n_lights,
                    int32_t *target, int *count, cudaStream_t st) {
    if (n > 0) k_targets<<<(n + 127) / 128, 128, 0, st>>>(res, rows, n, cluster_of, n_lights, target, count);
    return cudaGetLastError();
}

cudaError_t check_rows(const int32_t *rows, const int32_t *targets, int n, int64_t pixels, int c, uint32_t *bad,
                       cudaStream_t st) {
    if (n > 0) k_check_rows<<<(n + 127) / 128, 128, 0, st>>>(rows, targets, n, pixels, c, bad);
    return cudaGetLastError();
}

cudaError_t batch_rows(int32_t *rows, int n, uint32_t pixels, uint32_t offset, uint32_t stride, cudaStream_t st) {
    if (n > 0) k_batch_rows<<<(n + 127) / 128, 128, 0, st>>>(rows, n, pixels, offset, stride);
    return cudaGetLastError();
}

}  // namespace mlp
