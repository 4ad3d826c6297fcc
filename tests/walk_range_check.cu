// The quantized walk over scenes and segments of every magnitude, built by
// tests/test_walk_ranges.py and run on the CPU with the node check and the two
// walks of walk_nodes_check.cu.
//
// A scene of about unit size is scaled by 2^e (exact, so the tree keeps its
// shape) and packed; its nodes are checked, and each segment that the device
// sends down the quantized walk (components within 2^+-100, rgm::walk_fits)
// has to test the reference's triangles: random segments, segments with one
// component down to 2^-99 of the scene or none that small, with one up to 2^60
// of it, and from starts up to 2^40 scene sizes away.
// Prints one line of counts: `fast` of `usable` segments took the walk;
// `infinite` node visits met a plane that was not finite.
#define main walk_nodes_main
#include "walk_nodes_check.cu"
#undef main

namespace {

// Distances of node x's planes that are not finite.
bool finite_planes(const Scene &s, uint32_t x, f3 o, f3 inv) {
    const Node n{&s.q[16 * (size_t)x]};
    const float oo[3] = {o.x, o.y, o.z}, iv[3] = {inv.x, inv.y, inv.z};
    for (int a = 0; a < 3; ++a) {
        const float A = n.scale(a) * iv[a], B = fmaf(n.base(a) - oo[a], iv[a], 0.0f);
        if (!std::isfinite(A) || !std::isfinite(B) || !std::isfinite(65536.0f * A) || !std::isfinite(fmaf(65536.0f, A, B)))
            return false;
    }
    return true;
}

}  // namespace

int main(int argc, char **argv) {
    const int e = argc > 1 ? atoi(argv[1]) : 0;
    const int nrays = argc > 2 ? atoi(argv[2]) : 4000;
    const int n = 3000;
    std::mt19937 rng(17);
    std::uniform_real_distribution<float> U(-1.f, 1.f);
    std::vector<float> xyz;
    for (int i = 0; i < n; ++i) {
        const float c[3] = {U(rng), U(rng), U(rng)};
        for (int k = 0; k < 9; ++k) xyz.push_back(ldexpf(c[k % 3] + 0.1f * U(rng), e));
    }
    Scene s;
    s.nodes.resize((size_t)n - 1);
    s.tris.resize((size_t)n);
    int undefined = 0, depth = 0;
    if (host_build_bvh(xyz.data(), n, s.nodes.data(), s.tris.data(), &undefined) < 0) return 1;
    s.t12.resize(12 * (size_t)n);
    host_pack_tris(s.tris.data(), n, s.t12.data());
    const int nq = host_pack_quant(s.nodes.data(), n - 1, s.t12.data(), s.q, s.ql, &depth);
    float reach = 0.0f;
    s.q = host_walk_nodes(s.q, &reach);
    if (nq <= 0 || (int)(s.q.size() / 16) != nq) {
        printf("walk nodes not built: %d packed, %zu\n", nq, s.q.size() / 16);
        return 1;
    }
    float rlo[3], rhi[3];
    std::vector<int> leaf_seen((size_t)n, 0), node_seen((size_t)nq, 0);
    const long contain = check_node(s, 0, rlo, rhi, leaf_seen, node_seen);
    long usable = 0, fast = 0, set_mismatch = 0, any_mismatch = 0, visits = 0, infinite = 0, hits = 0;
    for (int i = 0; i < nrays; ++i) {
        float a[3], b[3];
        for (int k = 0; k < 3; ++k) {
            a[k] = U(rng);
            b[k] = U(rng);
        }
        const int kind = i % 4, axis = (i / 4) % 3, p = i / 12;
        if (kind == 1) {  // one tiny component: both ends near the plane through the centre
            a[axis] = 0.0f;
            b[axis] = ldexpf(U(rng), -(p % 99));
        } else if (kind == 2) {  // one huge component
            b[axis] = ldexpf(U(rng), p % 60);
        } else if (kind == 3) {  // a far start, the other end beyond the scene's middle
            for (int k = 0; k < 3; ++k) {
                const float m = 0.2f * U(rng);
                a[k] = ldexpf(U(rng), p % 40);
                b[k] = m + (m - a[k]) * ldexpf(1.0f, -(p % 40));
            }
        }
        const f3 p1 = mk(ldexpf(a[0], e), ldexpf(a[1], e), ldexpf(a[2], e));
        const f3 p2 = mk(ldexpf(b[0], e), ldexpf(b[1], e), ldexpf(b[2], e));
        f3 o, d;
        rgm::shadow_segment(p1, p2, o, d);
        const float lo = ldexpf(1.0f, -100), hi = ldexpf(1.0f, 100);
        const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
        if (!(ax >= lo && ax <= hi && ay >= lo && ay <= hi && az >= lo && az <= hi)) continue;
        ++usable;
        if (!rgm::walk_fits(reach, o, d)) continue;
        ++fast;
        const f3 inv = mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
        for (int x = 0; x < nq; ++x) infinite += !finite_planes(s, (uint32_t)x, o, inv);
        std::set<int> bt, qg;
        bool ba = false, qa = false;
        binary_set(s, o, d, bt, ba);
        walk_set(s, o, d, inv, qg, qa, visits);
        if (qg.size() != bt.size()) ++set_mismatch;
        if (ba != qa) ++any_mismatch;
        hits += ba;
    }
    printf("scale %d reach %g containment_failures %ld usable %ld fast %ld infinite %ld set_mismatches %ld "
           "answer_mismatches %ld hits %ld visits_per_ray %.2f\n",
           e, reach, contain, usable, fast, infinite, set_mismatch, any_mismatch, hits, fast ? (double)visits / fast : 0.0);
    return 0;
}
