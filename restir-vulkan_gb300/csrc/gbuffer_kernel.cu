// gbuffer_kernel.cu -- primary-ray G-buffer on the GPU (one thread per pixel,
// closest hit on the uploaded tree).  Rays, triangle tests and shading are the
// host tracer's (rg_gbuffer.cuh); the walk is a second version of
// rgm::closest_hit with the same tests in the same order, so both write
// identical planes (tests/test_gpu_launch_sizes.py, test_gpu_parity.py).
//
// Bound by instruction issue and the L1's data pipe (both 75 % busy; 18 of 32
// lanes a warp at work).  1920x1080, 1.05M triangles: 0.82 ms, against 1.02 ms
// with scalar slab tests and 1.28 ms with the node read as single words too; 16 x
// 2 or 4 x 8 pixels a warp are 1 to 3 % slower than 8 x 4.
#include <cuda_runtime.h>

#include "rg_gbuffer.cuh"
#include "rg_internal.h"

namespace {

struct GbufParams {
    rgm::TraceScene s;
    int box_nan;
    const rg_material *mats;
    int n_mats;
    rg_camera cam;
    int w, h;
    uint32_t *albedo;
    uint2 *normal;
    uint32_t *material;
    float4 *wpos;
    float *depth;
};

__device__ __forceinline__ void ldg256(const float *p, float (&v)[8]) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(p));
}
__device__ __forceinline__ void test_tri(const rgm::TraceScene &s, int tri, rgm::f3 o, rgm::f3 d, rgm::Hit &h) {
    const float4 *tp = reinterpret_cast<const float4 *>(s.tris + 12 * (size_t)tri);
    const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
    float t;
    if (rgm::tri_t(rgm::mk(a.x, a.y, a.z), rgm::mk(a.w, b.x, b.y), rgm::mk(b.z, b.w, c.x), o, d, t))
        if (t < h.t || (t == h.t && tri < h.tri)) { h.t = t; h.tri = tri; }
}

// Both children's slab tests (rgm::slab) as packed pairs with IEEE min / max:
// the same values where no slab distance is NaN (the caller checks the ray and
// the scene), apart from the sign of a zero, which no comparison sees.
__device__ __forceinline__ void slab_pair(const float (&p)[8], const float (&q)[8], rgm::f3 o, rgm::f3 inv, float best,
                                          bool &hl, float &tl, bool &hr, float &tr) {
    const float2 ox = make_float2(-o.x, -o.x), oy = make_float2(-o.y, -o.y), oz = make_float2(-o.z, -o.z);
    const float2 ix = make_float2(inv.x, inv.x), iy = make_float2(inv.y, inv.y), iz = make_float2(inv.z, inv.z);
    const float2 ax = __fmul2_rn(__fadd2_rn(make_float2(p[0], p[1]), ox), ix);
    const float2 bx = __fmul2_rn(__fadd2_rn(make_float2(p[2], p[3]), ox), ix);
    const float2 ay = __fmul2_rn(__fadd2_rn(make_float2(p[4], p[5]), oy), iy);
    const float2 by = __fmul2_rn(__fadd2_rn(make_float2(p[6], p[7]), oy), iy);
    const float2 az = __fmul2_rn(__fadd2_rn(make_float2(q[0], q[1]), oz), iz);
    const float2 bz = __fmul2_rn(__fadd2_rn(make_float2(q[2], q[3]), oz), iz);
    tl = fmaxf(fminf(ax.x, bx.x), fmaxf(fminf(ay.x, by.x), fminf(az.x, bz.x)));
    tr = fmaxf(fminf(ax.y, bx.y), fmaxf(fminf(ay.y, by.y), fminf(az.y, bz.y)));
    const float xl = fminf(fmaxf(ax.x, bx.x), fminf(fmaxf(ay.x, by.x), fmaxf(az.x, bz.x)));
    const float xr = fminf(fmaxf(ax.y, bx.y), fminf(fmaxf(ay.y, by.y), fmaxf(az.y, bz.y)));
    hl = xl >= tl && xl > 0.0f && tl < best;
    hr = xr >= tr && xr > 0.0f && tr < best;
}

// rgm::closest_hit with the node as two 256-bit loads, the triangle as three
// 128-bit ones and packed slab tests: the same tests in the same order.
__device__ __forceinline__ rgm::Hit closest_hit_wide(const rgm::TraceScene &s, bool box_nan, rgm::f3 o, rgm::f3 d) {
    using rgm::mk;
    rgm::Hit h;
    h.t = 3.402823466e38f;
    h.tri = -1;
    if (s.n_nodes <= 0) return h;
    const rgm::f3 inv = mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
    // no zero times infinity and no difference of infinities: 1/d finite and
    // nonzero, o finite, no NaN box
    constexpr float kLo = 7.8886090522101181e-31f, kHi = 1.2676506002282294e30f;  // 2^-100, 2^100
    const float dmin = fminf(fminf(fabsf(d.x), fabsf(d.y)), fabsf(d.z));
    const float dmax = fmaxf(fmaxf(fabsf(d.x), fabsf(d.y)), fabsf(d.z));
    const bool packed = !box_nan && dmin >= kLo && dmax <= kHi && fabsf(o.x) <= kHi && fabsf(o.y) <= kHi &&
                        fabsf(o.z) <= kHi && !(isnan(d.x) || isnan(d.y) || isnan(d.z));
    int stack[RG_MAX_TREE_DEPTH + 1];
    int top = 0, node = 0, visits = 0;
    while (true) {
        if (++visits > s.n_nodes) { h.tri = -1; return h; }
        float p[8], q[8];  // per axis lmin rmin lmax rmax: x, y; z, links
        ldg256(s.nodes + 16 * (size_t)node, p);
        ldg256(s.nodes + 16 * (size_t)node + 8, q);
        const int left = __float_as_int(q[4]), right = __float_as_int(q[5]);
        float tl, tr;
        bool hl, hr;
        if (packed) {
            slab_pair(p, q, o, inv, h.t, hl, tl, hr, tr);
        } else {
            hl = rgm::slab(o, inv, mk(p[0], p[4], q[0]), mk(p[2], p[6], q[2]), h.t, tl);
            hr = rgm::slab(o, inv, mk(p[1], p[5], q[1]), mk(p[3], p[7], q[3]), h.t, tr);
        }
        int first = -1, second = -1;
        if (hl) {
            if (left < 0) test_tri(s, ~left, o, d, h);
            else first = left;
        }
        if (hr) {
            if (right < 0) {
                test_tri(s, ~right, o, d, h);
            } else if (first < 0) {
                first = right;
            } else if (tr < tl) {
                second = first;
                first = right;
            } else {
                second = right;
            }
        }
        if (second >= 0) {
            if (top > RG_MAX_TREE_DEPTH) { h.tri = -1; return h; }
            stack[top++] = second;
        }
        if (first < 0) {
            if (top == 0) return h;
            first = stack[--top];
        }
        node = first;
    }
}

// A block of 128 threads covers 16 x 8 pixels, a warp 8 x 4 of them.
__global__ void __launch_bounds__(128) k_trace_gbuffer(const GbufParams p) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int tw = 8, th = 4;
    const int x = blockIdx.x * 16 + (warp % (16 / tw)) * tw + lane % tw;
    const int y = blockIdx.y * 8 + (warp / (16 / tw)) * th + lane / tw;
    if (x >= p.w || y >= p.h) return;
    rgm::f3 o, d;
    rgm::primary_ray(p.cam, x, y, p.w, p.h, o, d);
    const rgm::Hit hit = closest_hit_wide(p.s, p.box_nan != 0, o, d);
    rgm::GTexel g;
    rgm::shade_texel(p.s, p.mats, p.n_mats, p.cam, o, d, hit, g);
    const size_t i = (size_t)y * (size_t)p.w + (size_t)x;
    p.albedo[i] = g.albedo;
    p.normal[i] = make_uint2((uint32_t)g.normal[0] | ((uint32_t)g.normal[1] << 16),
                             (uint32_t)g.normal[2] | ((uint32_t)g.normal[3] << 16));
    p.material[i] = g.material;
    p.wpos[i] = make_float4(g.wpos[0], g.wpos[1], g.wpos[2], g.wpos[3]);
    p.depth[i] = g.depth;
}

}  // namespace

cudaError_t launch_trace_gbuffer(const DevScene &s, const rg_camera &cam, const rg_gbuffer_out &out, cudaStream_t st) {
    GbufParams p;
    p.s.nodes = reinterpret_cast<const float *>(s.nodes);
    p.s.n_nodes = s.n_nodes;
    p.s.tris = reinterpret_cast<const float *>(s.tris);
    p.s.n_tris = s.n_tris;
    p.box_nan = s.box_nan;
    p.mats = s.materials;
    p.n_mats = s.n_materials;
    p.cam = cam;
    p.w = out.width;
    p.h = out.height;
    p.albedo = static_cast<uint32_t *>(out.albedo);
    p.normal = static_cast<uint2 *>(out.normal);
    p.material = static_cast<uint32_t *>(out.material);
    p.wpos = static_cast<float4 *>(out.world_pos);
    p.depth = static_cast<float *>(out.depth);
    const dim3 grid((unsigned)((out.width + 15) / 16), (unsigned)((out.height + 7) / 8));
    k_trace_gbuffer<<<grid, 128, 0, st>>>(p);
    return cudaGetLastError();
}
