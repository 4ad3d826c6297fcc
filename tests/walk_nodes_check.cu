// Host-side check of the nodes that the device's quantized walk reads
// (host_walk_nodes), built by tests/test_walk_nodes.py and run on the CPU.
//
// For seeded scenes it builds the reference's tree, packs the quantized copy
// and its walk form, and checks:
//  - every plane lies outside the child's exact box (in real arithmetic, by at
//    least 1/16 of a code), for every child of every node;
//  - the nodes are a tree over every leaf record: inner children consecutive
//    in the first slots, leaf records consecutive, each reached once;
//  - for segments aimed at triangle edges, nearly axis-aligned segments, tiny
//    and huge direction components and random ones, the triangles that the
//    walk tests (the arithmetic of trace_pool.cuh's qlive, then the exact
//    leaf gate) are those whose whole box path passes the reference's slab
//    test (softwareRaytracing.glsl:9-14), and the any-hit answers agree.
// Prints one line of counts; exit status 0 when every check holds.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <set>
#include <vector>

#include "host_internal.h"
#include "rg_math.cuh"

using rgm::f3;
using rgm::mk;

namespace {

float f_of(uint32_t u) {
    float f;
    memcpy(&f, &u, 4);
    return f;
}
float sat(float x) { return x > 0.0f ? (x < 1.0f ? x : 1.0f) : 0.0f; }

struct Scene {
    std::vector<rg_aabb_tree_node> nodes;
    std::vector<rg_triangle> tris;
    std::vector<float> t12;
    std::vector<uint32_t> q;
    std::vector<float> ql;
};

// Triangles tested by the reference's walk (every box on the path passes).
void binary_set(const Scene &s, f3 o, f3 d, std::set<int> &tested, bool &any) {
    std::vector<int> st{0};
    while (!st.empty()) {
        const int x = st.back();
        st.pop_back();
        const rg_aabb_tree_node &nd = s.nodes[(size_t)x];
        for (int side = 0; side < 2; ++side) {
            const float *lo = side ? nd.right_aabb_min : nd.left_aabb_min;
            const float *hi = side ? nd.right_aabb_max : nd.left_aabb_max;
            if (!rgm::ray_aabb(o, d, mk(lo[0], lo[1], lo[2]), mk(hi[0], hi[1], hi[2]))) continue;
            const int c = side ? nd.right_child : nd.left_child;
            if (c >= 0) {
                st.push_back(c);
            } else {
                tested.insert(~c);
                const float *p = &s.t12[12 * (size_t)(~c)];
                any = any || rgm::ray_tri(mk(p[0], p[1], p[2]), mk(p[3], p[4], p[5]), mk(p[6], p[7], p[8]), o, d);
            }
        }
    }
}

// The axes' planes and distances of child k of a walk node.
struct Node {
    const uint32_t *w;
    float base(int a) const { return f_of(w[a]); }
    float scale(int a) const { return a == 2 ? f_of(w[3] & 0x7f800000u) : f_of(w[10 + a]); }
    unsigned code(int a, int side, int k) const { return (w[4 + 2 * a + side] >> (8 * k)) & 255u; }
    double plane(int a, int side, int k) const { return (double)base(a) + (32768.0 + code(a, side, k)) * (double)scale(a); }
    unsigned leaves() const { return w[3] & 15u; }
    unsigned inner() const { return (w[3] >> 4) & 15u; }
};

bool live(const Node &n, int k, f3 o, f3 inv) {
    const float K = 3.814697265625e-6f, oo[3] = {o.x, o.y, o.z}, iv[3] = {inv.x, inv.y, inv.z};
    float tn[3], tf[3];
    for (int a = 0; a < 3; ++a) {
        const bool neg = iv[a] < 0.0f;
        const float A = n.scale(a) * iv[a], c = n.base(a) - oo[a];
        const float fn = f_of(0x47000000u | n.code(a, neg ? 1 : 0, k) << 8);
        const float ff = f_of(0x47000000u | n.code(a, neg ? 0 : 1, k) << 8);
        tn[a] = fmaf(fn, A, fmaf(c, iv[a], -K));
        tf[a] = fmaf(ff, A, fmaf(c, iv[a], K));
    }
    tn[0] = sat(tn[0]);
    tf[0] = sat(tf[0]);
    return fmaxf(fmaxf(tn[0], tn[1]), tn[2]) < fminf(fminf(tf[0], tf[1]), tf[2]);
}

bool leaf_box(const float *r, f3 o, f3 d) { return rgm::ray_aabb(o, d, mk(r[0], r[1], r[2]), mk(r[3], r[4], r[5])); }

void walk_set(const Scene &s, f3 o, f3 d, f3 inv, std::set<int> &gated, bool &any, long &visits) {
    std::vector<uint32_t> st{0};
    while (!st.empty()) {
        const Node n{&s.q[16 * (size_t)st.back()]};
        st.pop_back();
        ++visits;
        for (int k = 0; k < 4; ++k) {
            if (!((n.leaves() | n.inner()) >> k & 1u) || !live(n, k, o, inv)) continue;
            if (n.inner() >> k & 1u) {
                st.push_back(n.w[12] + (uint32_t)k);
                continue;
            }
            const uint32_t rec = (n.w[13] + (uint32_t)k) & 0x7ffffffu;
            const float *r = &s.ql[16 * (size_t)rec];
            if (!leaf_box(r, o, d)) continue;
            gated.insert((int)rec);
            any = any || rgm::ray_tri(mk(r[6], r[7], r[8]), mk(r[9], r[10], r[11]), mk(r[12], r[13], r[14]), o, d);
        }
    }
}

// Structure and containment below node x; adds its leaf-box union to lo/hi.
long check_node(const Scene &s, uint32_t x, float lo[3], float hi[3], std::vector<int> &leaf_seen,
                std::vector<int> &node_seen) {
    long bad = 0;
    if (x >= node_seen.size() || node_seen[x]++) return 1;
    const Node n{&s.q[16 * (size_t)x]};
    const int ni = __builtin_popcount(n.inner()), nl = __builtin_popcount(n.leaves());
    if (n.inner() != (1u << ni) - 1u || n.leaves() != ((1u << nl) - 1u) << ni || ni + nl < 2) ++bad;
    for (int a = 0; a < 3; ++a) { lo[a] = INFINITY; hi[a] = -INFINITY; }
    for (int k = 0; k < ni + nl; ++k) {
        float clo[3], chi[3];
        if (k < ni) {
            bad += check_node(s, n.w[12] + (uint32_t)k, clo, chi, leaf_seen, node_seen);
        } else {
            const uint32_t rec = (n.w[13] + (uint32_t)k) & 0x7ffffffu;
            if (rec >= leaf_seen.size() || leaf_seen[rec]++) return bad + 1;
            for (int a = 0; a < 3; ++a) { clo[a] = s.ql[16 * (size_t)rec + a]; chi[a] = s.ql[16 * (size_t)rec + 3 + a]; }
        }
        for (int a = 0; a < 3; ++a) {
            const double pad = 0.0625 * (double)n.scale(a);
            if (!(n.plane(a, 0, k) <= (double)clo[a] - pad) || !(n.plane(a, 1, k) >= (double)chi[a] + pad)) ++bad;
            lo[a] = fminf(lo[a], clo[a]);
            hi[a] = fmaxf(hi[a], chi[a]);
        }
    }
    return bad;
}

}  // namespace

int main(int argc, char **argv) {
    const int ntri = argc > 1 ? atoi(argv[1]) : 20000;
    const int nrays = argc > 2 ? atoi(argv[2]) : 10000;
    const float off = argc > 3 ? (float)atof(argv[3]) : 0.0f;
    const unsigned seed = argc > 4 ? (unsigned)atoi(argv[4]) : 7u;
    std::mt19937 rng(seed);
    std::uniform_real_distribution<float> U(-10.f, 10.f), S(0.f, 1.f);
    std::vector<float> xyz;
    const int g = 40;  // floor grid: flat boxes
    for (int i = 0; i < g; ++i)
        for (int j = 0; j < g; ++j) {
            const float x0 = -10 + 20.f * i / g, x1 = -10 + 20.f * (i + 1) / g;
            const float z0 = -10 + 20.f * j / g, z1 = -10 + 20.f * (j + 1) / g;
            const float a[18] = {x0, 0, z0, x1, 0, z0, x1, 0, z1, x0, 0, z0, x1, 0, z1, x0, 0, z1};
            xyz.insert(xyz.end(), a, a + 18);
        }
    while ((int)xyz.size() / 9 < ntri) {
        const float cx = U(rng), cy = 5 + 0.5f * U(rng), cz = U(rng), sz = 0.05f + 0.5f * S(rng);
        if (S(rng) < 0.2f) {  // axis-aligned quad
            float a[9] = {cx, cy, cz, cx + sz, cy, cz, cx, cy, cz + sz};
            if (S(rng) < 0.5f) { a[3] = cx; a[4] = cy + sz; a[6] = cx; a[7] = cy; a[8] = cz + sz; }
            xyz.insert(xyz.end(), a, a + 9);
        } else {
            for (int k = 0; k < 3; ++k) {
                xyz.push_back(cx + sz * (S(rng) - 0.5f));
                xyz.push_back(cy + sz * (S(rng) - 0.5f));
                xyz.push_back(cz + sz * (S(rng) - 0.5f));
            }
        }
    }
    for (size_t i = 0; i < xyz.size(); i += 3) xyz[i] += off;
    const int n = (int)xyz.size() / 9;
    Scene s;
    s.nodes.resize((size_t)n - 1);
    s.tris.resize((size_t)n);
    int undefined = 0;
    if (host_build_bvh(xyz.data(), n, s.nodes.data(), s.tris.data(), &undefined) < 0) {
        printf("tree build failed\n");
        return 1;
    }
    s.t12.resize(12 * (size_t)n);
    host_pack_tris(s.tris.data(), n, s.t12.data());
    int depth = 0;
    const int nq = host_pack_quant(s.nodes.data(), n - 1, s.t12.data(), s.q, s.ql, &depth);
    if (nq <= 0 || (int)(s.ql.size() / 16) != n) {
        printf("quantized copy not built (%d)\n", nq);
        return 1;
    }
    s.q = host_walk_nodes(s.q);
    if ((int)(s.q.size() / 16) != nq) {
        printf("walk nodes not built\n");
        return 1;
    }
    float rlo[3], rhi[3];
    std::vector<int> leaf_seen((size_t)n, 0), node_seen((size_t)nq, 0);
    long contain = check_node(s, 0, rlo, rhi, leaf_seen, node_seen);
    for (int v : leaf_seen) contain += v != 1;
    for (int v : node_seen) contain += v != 1;
    long fast = 0, set_mismatch = 0, any_mismatch = 0, visits = 0;
    std::uniform_int_distribution<int> T(0, n - 1);
    for (int i = 0; i < nrays; ++i) {
        f3 p1, p2;
        const int kind = i % 5;
        if (kind == 0) {
            p1 = mk(U(rng), 0.0f, U(rng));
            p2 = mk(U(rng), 8 + U(rng) * 0.3f, U(rng));
        } else if (kind == 1) {  // through a point of a triangle edge
            const rg_triangle &t = s.tris[(size_t)T(rng)];
            const float u = S(rng);
            const f3 m = mk(t.p1[0] + u * (t.p2[0] - t.p1[0]), t.p1[1] + u * (t.p2[1] - t.p1[1]),
                            t.p1[2] + u * (t.p2[2] - t.p1[2]));
            p1 = mk(U(rng) + off, 0.0f, U(rng));
            p2 = mk(m.x + (m.x - p1.x), m.y + (m.y - p1.y), m.z + (m.z - p1.z));
            p1.x -= off;
            p2.x -= off;
        } else if (kind == 2) {  // nearly axis-aligned
            p1 = mk(U(rng), 0.0f, U(rng));
            p2 = mk(p1.x + 1e-4f * U(rng), 9.0f, p1.z + 1e-4f * U(rng));
        } else if (kind == 3) {
            p1 = mk(U(rng), 5 + U(rng) * 0.3f, U(rng));
            p2 = mk(U(rng), 5 + U(rng) * 0.3f, U(rng));
        } else {  // one component down to 2^-60 of the others
            p1 = mk(0.0f, 5 + U(rng) * 0.3f, U(rng));
            p2 = mk(ldexpf(U(rng), -(i / 5) % 58), 5 + U(rng) * 0.3f, U(rng));
        }
        p1.x += off;
        p2.x += off;
        f3 o, d;
        rgm::shadow_segment(p1, p2, o, d);
        const float lo = 8.67361737988403547e-19f, hi = 1.152921504606846976e18f;  // 2^-60, 2^60
        if (!(fabsf(d.x) >= lo && fabsf(d.x) <= hi && fabsf(d.y) >= lo && fabsf(d.y) <= hi && fabsf(d.z) >= lo &&
              fabsf(d.z) <= hi))
            continue;  // off the fast path: those rays walk the reference's tree
        ++fast;
        const f3 inv = mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
        std::set<int> bt, qg;
        bool ba = false, qa = false;
        binary_set(s, o, d, bt, ba);
        walk_set(s, o, d, inv, qg, qa, visits);
        // leaf records hold the triangles' own fields: compare the sets by them
        std::set<int> qg_tri;
        for (int r : qg) {
            const float *rp = &s.ql[16 * (size_t)r];
            int found = -1;
            for (int t : bt)
                if (!memcmp(&s.t12[12 * (size_t)t], rp + 6, 36)) { found = t; break; }
            qg_tri.insert(found);
        }
        if (qg_tri != bt || qg.size() != bt.size()) ++set_mismatch;
        if (ba != qa) ++any_mismatch;
    }
    printf("triangles %d quantized_nodes %d containment_failures %ld fast_rays %ld set_mismatches %ld "
           "answer_mismatches %ld visits_per_ray %.2f\n",
           n, nq, contain, fast, set_mismatch, any_mismatch, fast ? (double)visits / fast : 0.0);
    return (contain || set_mismatch || any_mismatch || fast < nrays / 2) ? 2 : 0;
}
