// The byte boxes of the device nodes and what the traversal makes of them, on
// the CPU in the kernels' float expressions:
//   planes    a node's bytes enclose its children's float boxes and the margin
//   slabs     a ray that a child's float box admits is admitted by its bytes
//   traversal the closest hit through byte boxes, of instances under transforms
//             too, is that through float boxes unless found ambiguous
#include "fake_cuda.h"

#include "../../psycles_b200/csrc/psy_host.cpp"

#include <cstdio>
#include <random>

namespace {

std::mt19937 rng(7);
double uniform(double lo, double hi) { return std::uniform_real_distribution<double>(lo, hi)(rng); }

#define CHECK(x)                                              \
    do {                                                      \
        if (!(x)) {                                           \
            std::printf("line %d: %s\n", __LINE__, #x);       \
            std::exit(1);                                     \
        }                                                     \
    } while (0)

double factor(uint32_t byte) { return byte < 128u ? 0.5 + byte / 256.0 : 1.0 + (byte - 128u) / 128.0; }
float plane_factor(uint32_t word, int k) {
    const uint32_t bits = 0x3f000000u | ((word >> (8 * k)) & 0xffu) << 16;
    float f;
    std::memcpy(&f, &bits, 4);
    CHECK(double(f) == factor((word >> (8 * k)) & 0xffu));
    return f;
}

WideNode random_node(double scale, double offset, int children, int flat_axis) {
    WideNode w;
    for (int k = 0; k < children; ++k) {
        Box b;
        for (int c = 0; c < 2; ++c) {
            double p[3];
            for (int a = 0; a < 3; ++a)
                p[a] = float(offset + scale * (a == flat_axis ? 0.25 : uniform(-1.0, 1.0) * (k == 1 ? 1e-3 : 1.0)));
            b.grow(p[0], p[1], p[2]);
        }
        float lo[3], hi[3];
        padded(b, lo, hi);
        for (int a = 0; a < 3; ++a) {
            w.lo[a][k] = lo[a];
            w.hi[a][k] = hi[a];
        }
        w.link[k] = psy::kLinkLeaf | uint32_t(k);
    }
    return w;
}

void planes() {
    for (const double scale : {1e-30, 1e-12, 1e-4, 1.0, 37.0, 1e4, 1e12, 1e30, 3e37})
        for (const double offset : {0.0, 1.0, -50.0, 2e3, -1e30})
            for (int children = 0; children <= 4; ++children)
                for (int flat = -1; flat < 3; ++flat) {
                    if (std::fabs(offset) + 2.0 * scale > 3e38) continue;
                    const WideNode w = random_node(scale, offset, children, flat);
                    const psy::NodeGpu g = quantise(w, 10u, 20u);
                    const uint32_t lo[3] = {g.lox, g.loy, g.loz}, hi[3] = {g.hix, g.hiy, g.hiz};
                    for (int a = 0; a < 3; ++a) {
                        CHECK(std::isfinite(g.base[a]) == std::isfinite(g.span[a]));
                        if (!std::isfinite(g.base[a])) {
                            CHECK(scale > 1e37);
                            continue;
                        }
                        double l = 1e300, h = -1e300;
                        for (int k = 0; k < children; ++k) {
                            l = std::min(l, double(w.lo[a][k]));
                            h = std::max(h, double(w.hi[a][k]));
                        }
                        const double margin = 3.99e-6 * ((h - l) + std::max(std::fabs(l), std::fabs(h)));
                        for (int k = 0; k < children; ++k) {
                            const double low = g.base[a] + double(g.span[a]) * factor((lo[a] >> (8 * k)) & 0xffu);
                            const double high = g.base[a] + double(g.span[a]) * factor((hi[a] >> (8 * k)) & 0xffu);
                            CHECK(low <= w.lo[a][k] - margin && high >= w.hi[a][k] + margin);
                            // and by no more than two planes' distance
                            CHECK(low >= w.lo[a][k] - 3.0 * margin - g.span[a] / 60.0 - 1e-29);
                        }
                    }
                    for (int k = 0; k < 4; ++k)
                        CHECK(g.link[k] == (k < children ? psy::kLinkLeaf | uint32_t(20 + k) : psy::kInvalidId));
                }
    // what float cannot hold constrains nothing
    WideNode w = random_node(1.0, 0.0, 2, -1);
    w.hi[1][0] = INFINITY;
    CHECK(std::isnan(quantise(w, 0u, 0u).base[1]) && !std::isnan(quantise(w, 0u, 0u).base[0]));
}

struct Slabs {
    V3 o, d, inv, oinv;
};
Slabs slabs(V3 o, V3 d) {
    // the hardware's reciprocal may be a unit in the last place off
    auto rcp = [](float x) {
        const float r = 1.0f / x;
        const int off = int(rng() % 3u) - 1;
        return off < 0 ? std::nextafter(r, -INFINITY) : off > 0 ? std::nextafter(r, INFINITY) : r;
    };
    Slabs s{o, d, {rcp(d.x), rcp(d.y), rcp(d.z)}, {}};
    s.oinv = {o.x * s.inv.x, o.y * s.inv.y, o.z * s.inv.z};
    return s;
}
// box_admits
bool admits(const Slabs &r, const float lo[3], const float hi[3], float tmin, float tmax, float &near) {
    const float d[3] = {r.d.x, r.d.y, r.d.z}, inv[3] = {r.inv.x, r.inv.y, r.inv.z}, oinv[3] = {r.oinv.x, r.oinv.y, r.oinv.z};
    float far = tmax;
    near = tmin;
    for (int a = 0; a < 3; ++a) {
        near = std::fmax(near, std::fma(d[a] < 0.0f ? hi[a] : lo[a], inv[a], -oinv[a]));
        far = std::fmin(far, std::fma(d[a] < 0.0f ? lo[a] : hi[a], inv[a], -oinv[a]));
    }
    return near <= std::fmax(std::fma(far, 1.00000095367431640625f, 1.0e-30f), far);
}
// the slab test of visit_node
void node_hits(const psy::NodeGpu &g, const Slabs &r, float tmin, float tmax, float near[4], bool hit[4]) {
    const float inv[3] = {r.inv.x, r.inv.y, r.inv.z}, oinv[3] = {r.oinv.x, r.oinv.y, r.oinv.z};
    const uint32_t lo[3] = {g.lox, g.loy, g.loz}, hi[3] = {g.hix, g.hiy, g.hiz};
    for (int k = 0; k < 4; ++k) {
        float far = tmax;
        near[k] = tmin;
        for (int a = 0; a < 3; ++a) {
            const float b = std::fma(g.base[a], inv[a], -oinv[a]), s = g.span[a] * inv[a];
            near[k] = std::fmax(near[k], std::fma(plane_factor(inv[a] < 0.0f ? hi[a] : lo[a], k), s, b));
            far = std::fmin(far, std::fma(plane_factor(inv[a] < 0.0f ? lo[a] : hi[a], k), s, b));
        }
        hit[k] = near[k] <= std::fma(far, 1.0000038146972656f, 1.0e-30f) && g.link[k] != psy::kInvalidId;
    }
}

V3 direction() {
    for (;;) {
        V3 d{float(uniform(-1, 1)), float(uniform(-1, 1)), float(uniform(-1, 1))};
        if (rng() % 6u == 0u) (&d.x)[rng() % 3u] *= 1e-5f;
        const float l = std::sqrt(dt(d, d));
        if (l > 0.1f && l < 1.0f && d.x != 0.0f && d.y != 0.0f && d.z != 0.0f) return {d.x / l, d.y / l, d.z / l};
    }
}
// A ray from `distance` away towards `target`, rounded.
bool aim(V3 target, double distance, V3 &o, V3 &d) {
    const V3 back = direction();
    o = {float(target.x - distance * back.x), float(target.y - distance * back.y), float(target.z - distance * back.z)};
    const V3 v = sub(target, o);
    const float l = std::sqrt(dt(v, v));
    if (!(l > 0.0f)) return false;
    d = {v.x / l, v.y / l, v.z / l};
    return d.x != 0.0f && d.y != 0.0f && d.z != 0.0f;
}

void slab_tests() {
    int admitted = 0;
    for (int n = 0; n < 300000; ++n) {
        const double scale = std::pow(10.0, uniform(-5, 5)), offset = rng() % 2u ? uniform(-1e3, 1e3) * scale : 0.0;
        const int children = 1 + int(rng() % 4u);
        const WideNode w = random_node(scale, offset, children, int(rng() % 4u) - 1);
        const psy::NodeGpu g = quantise(w, 0u, 0u);
        // towards a point of an edge of a child's box
        const int k = int(rng()) & 3;
        if (k >= children) continue;
        float p[3];
        const int along = int(rng() % 3u);
        for (int a = 0; a < 3; ++a)
            p[a] = a == along ? float(uniform(w.lo[a][k], w.hi[a][k])) : rng() % 2u ? w.lo[a][k] : w.hi[a][k];
        V3 o, d;
        if (!aim({p[0], p[1], p[2]}, scale * std::pow(10.0, uniform(-2, 5)), o, d)) continue;
        const Slabs r = slabs(o, d);
        float near[4];
        bool hit[4];
        const float tmax = rng() % 2u ? 1e30f : float(uniform(0.5, 1.5) * std::sqrt(dt(sub({p[0], p[1], p[2]}, o), sub({p[0], p[1], p[2]}, o))));
        node_hits(g, r, 0.0f, tmax, near, hit);
        for (int c = 0; c < children; ++c) {
            const float lo[3] = {w.lo[0][c], w.lo[1][c], w.lo[2][c]}, hi[3] = {w.hi[0][c], w.hi[1][c], w.hi[2][c]};
            float t;
            if (!admits(r, lo, hi, 0.0f, tmax, t)) continue;
            CHECK(hit[c]);
            ++admitted;
        }
    }
    CHECK(admitted > 100000);
}

// intersect_triangle's distance
V3 cr(V3 a, V3 b) {
    return {std::fma(a.y, b.z, -(a.z * b.y)), std::fma(a.z, b.x, -(a.x * b.z)), std::fma(a.x, b.y, -(a.y * b.x))};
}
float ip(V3 a, V3 b) { return std::fma(a.x, b.x, std::fma(a.y, b.y, a.z * b.z)); }
V3 ad(V3 a, V3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
bool hits(V3 o, V3 d, float tmin, float tmax, V3 p0, V3 p1, V3 p2, float &t) {
    const V3 v0 = sub(p0, o), v1 = sub(p1, o), v2 = sub(p2, o), e0 = sub(v2, v0), e1 = sub(v0, v1), e2 = sub(v1, v2);
    const float u = ip(cr(e0, ad(v2, v0)), d), v = ip(cr(e1, ad(v0, v1)), d), w = ip(cr(e2, ad(v1, v2)), d);
    const float sum = u + v + w, tol = 1.1920928955078125e-07f * std::fabs(sum);
    if (!(std::fmin(u, std::fmin(v, w)) >= -tol || std::fmax(u, std::fmax(v, w)) <= tol)) return false;
    V3 n = cr(e1, e0);
    n = {n.x * 2.0f, n.y * 2.0f, n.z * 2.0f};
    const float den = ip(n, d);
    if (den == 0.0f) return false;
    t = ip(v0, n) / den;
    return t >= tmin && t <= tmax;
}

struct Mesh {
    std::vector<V3> p;
    std::vector<uint32_t> idx;
    std::vector<WideNode> wide;
    std::vector<psy::NodeGpu> nodes;
    std::vector<uint32_t> leaf;  // triangle of each leaf slot
    std::vector<std::array<float, 6>> box;
    bool hit(uint32_t t, const Slabs &r, float tmin, float tmax, float &th) const {
        return hits(r.o, r.d, tmin, tmax, p[idx[3 * t]], p[idx[3 * t + 1]], p[idx[3 * t + 2]], th);
    }
    void build() {
        Builder b;
        b.prims.resize(idx.size() / 3u);
        box.resize(b.prims.size());
        for (uint32_t k = 0; k < b.prims.size(); ++k) {
            Prim &q = b.prims[k];
            for (int c = 0; c < 3; ++c) q.box.grow(p[idx[3 * k + c]].x, p[idx[3 * k + c]].y, p[idx[3 * k + c]].z);
            for (int a = 0; a < 3; ++a) q.c[a] = 0.5 * (q.box.lo[a] + q.box.hi[a]);
            q.id = k;
            padded(q.box, &box[k][0], &box[k][3]);
        }
        b.build_root();
        std::vector<uint32_t> order;
        wide = b.widen(order);
        for (const uint32_t o : order) leaf.push_back(b.prims[o].id);
        for (const WideNode &w : wide) nodes.push_back(quantise(w, 0u, 0u));
    }
};
// Instances of meshes under the instance tree, as scene compile lays them out.
struct Scene {
    std::vector<const Mesh *> mesh;  // of each instance
    std::vector<M34> o2w, w2o;
    std::vector<std::array<float, 6>> box;
    std::vector<WideNode> wide;
    std::vector<psy::NodeGpu> nodes;
    void add(const Mesh &m, const M34 &t) {
        mesh.push_back(&m);
        o2w.push_back(t);
        w2o.push_back(inverse34(t));
    }
    void build() {
        Builder b;
        b.leaf_is_id = true;
        box.resize(mesh.size());
        for (uint32_t i = 0; i < mesh.size(); ++i) {
            Prim q;
            const M34 &t = o2w[i];
            for (const V3 &v : mesh[i]->p) {
                const double x = v.x, y = v.y, z = v.z;
                q.box.grow(x * t.c0.x + y * t.c1.x + z * t.c2.x + t.c3.x, x * t.c0.y + y * t.c1.y + z * t.c2.y + t.c3.y,
                           x * t.c0.z + y * t.c1.z + z * t.c2.z + t.c3.z);
            }
            for (int a = 0; a < 3; ++a) {
                const double pad = 1e-4 * (q.box.hi[a] - q.box.lo[a]) +
                                   1e-5 * std::max(std::fabs(q.box.lo[a]), std::fabs(q.box.hi[a]));
                q.box.lo[a] -= pad;
                q.box.hi[a] += pad;
                q.c[a] = 0.5 * (q.box.lo[a] + q.box.hi[a]);
            }
            padded(q.box, &box[i][0], &box[i][3]);
            q.id = i;
            b.prims.push_back(q);
        }
        b.build_root();
        std::vector<uint32_t> order;
        wide = b.widen(order);
        for (const WideNode &w : wide) nodes.push_back(quantise(w, 0u, 0u));
    }
};
// A ray in the world and in every instance's object space.
struct SceneRay {
    Slabs world;
    std::vector<Slabs> object;
    SceneRay(const Scene &s, V3 o, V3 d) : world(slabs(o, d)) {
        for (const M34 &t : s.w2o) {
            V3 od = xaff(t, d, false);
            for (int a = 0; a < 3; ++a)
                if (std::fabs((&od.x)[a]) <= 8.271806e-25f) (&od.x)[a] = std::copysign(8.271806e-25f, (&od.x)[a]);
            object.push_back(slabs(xaff(t, o, true), od));
        }
    }
};
struct Found {
    float t;
    uint32_t instance, prim;
    bool operator==(const Found &o) const { return t == o.t && instance == o.instance && prim == o.prim; }
};
bool better(const Found &best, float t, uint32_t instance, uint32_t prim) {
    return best.instance == psy::kInvalidId || t < best.t ||
           (t == best.t && (instance > best.instance || (instance == best.instance && prim > best.prim)));
}
using Children = std::vector<std::pair<float, uint32_t>>;
void push(std::vector<uint32_t> &stack, Children &c) {
    std::stable_sort(c.begin(), c.end(), [](const auto &a, const auto &b) { return a.first > b.first; });
    for (const auto &i : c) stack.push_back(i.second);
}

// closest_exact: one tree, the instance tree's entries handed to `enter`
template <typename Enter, typename Leaf>
void walk_floats(const std::vector<WideNode> &wide, const Slabs &r, float tmin, const Found &best, Enter enter, Leaf leaf) {
    std::vector<uint32_t> stack{0u};
    while (!stack.empty()) {
        const uint32_t e = stack.back();
        stack.pop_back();
        if (e >= psy::kLinkInstance) {
            enter(e - psy::kLinkInstance);
            continue;
        }
        const WideNode &w = wide[e];
        float near[4];
        bool hit[4];
        for (int k = 0; k < 4; ++k) {
            const float lo[3] = {w.lo[0][k], w.lo[1][k], w.lo[2][k]}, hi[3] = {w.hi[0][k], w.hi[1][k], w.hi[2][k]};
            hit[k] = w.link[k] != psy::kInvalidId && admits(r, lo, hi, tmin, best.t, near[k]);
        }
        Children inner;
        for (int k = 0; k < 4; ++k)
            if (hit[k] && (w.link[k] & psy::kLinkLeaf) != 0u) leaf(w.link[k] & ~psy::kLinkLeaf);
        for (int k = 0; k < 4; ++k)
            if (hit[k] && (w.link[k] & psy::kLinkLeaf) == 0u && near[k] <= best.t) inner.push_back({near[k], w.link[k]});
        push(stack, inner);
    }
}
Found through_floats(const Scene &s, const SceneRay &ray, float tmin) {
    Found best{1e30f, psy::kInvalidId, psy::kInvalidId};
    walk_floats(s.wide, ray.world, tmin, best, [&](uint32_t i) {
        const Mesh &m = *s.mesh[i];
        walk_floats(m.wide, ray.object[i], tmin, best, [](uint32_t) {}, [&](uint32_t slot) {
            float t;
            if (m.hit(m.leaf[slot], ray.object[i], tmin, best.t, t) && better(best, t, i, m.leaf[slot]))
                best = {t, i, m.leaf[slot]};
        });
    }, [](uint32_t) {});
    return best;
}

// k_intersect's traversal, closest_hit and closest_ambiguous
template <typename Enter, typename Leaf>
void walk_bytes(const std::vector<psy::NodeGpu> &nodes, const Slabs &r, float tmin, const float &tmax, Enter enter, Leaf leaf) {
    std::vector<uint32_t> stack{0u};
    while (!stack.empty()) {
        const uint32_t e = stack.back();
        stack.pop_back();
        if (e >= psy::kLinkInstance) {
            enter(e - psy::kLinkInstance);
            continue;
        }
        float near[4];
        bool hit[4];
        node_hits(nodes[e], r, tmin, tmax, near, hit);
        Children inner;
        for (int k = 0; k < 4; ++k) {
            const uint32_t link = nodes[e].link[k];
            if (hit[k] && (link & psy::kLinkLeaf) != 0u) leaf(link & ~psy::kLinkLeaf);
            else if (hit[k]) inner.push_back({near[k], link});
        }
        push(stack, inner);
    }
}
Found through_bytes(const Scene &s, const SceneRay &ray, float tmin, bool &ambiguous) {
    Found best{1e30f, psy::kInvalidId, psy::kInvalidId};
    float tmax = 1e30f, second = 1e30f;
    walk_bytes(s.nodes, ray.world, tmin, tmax, [&](uint32_t i) {
        const Mesh &m = *s.mesh[i];
        walk_bytes(m.nodes, ray.object[i], tmin, tmax, [](uint32_t) {}, [&](uint32_t slot) {
            float t;
            if (!m.hit(m.leaf[slot], ray.object[i], tmin, tmax, t)) return;
            if (!better(best, t, i, m.leaf[slot])) {
                second = std::fmin(second, t);
                return;
            }
            second = best.t;
            best = {t, i, m.leaf[slot]};
            tmax = std::fma(t, 1.00000095367431640625f, 1.0e-30f);
        });
    }, [](uint32_t) {});
    ambiguous = false;
    if (best.instance != psy::kInvalidId) {
        float near, entry;
        const float *b = s.mesh[best.instance]->box[best.prim].data(), *w = s.box[best.instance].data();
        ambiguous = !admits(ray.object[best.instance], b, b + 3, tmin, INFINITY, near) ||
                    !admits(ray.world, w, w + 3, tmin, INFINITY, entry) || second < std::fmax(near, entry) ||
                    tmax < std::fmax(near, entry);
    }
    return best;
}

Mesh sphere(int n, float radius, V3 centre) {
    Mesh m;
    for (int i = 0; i <= n; ++i)
        for (int j = 0; j < 2 * n; ++j) {
            const double a = M_PI * i / n, b = M_PI * j / n;
            m.p.push_back({float(centre.x + radius * std::sin(a) * std::cos(b)), float(centre.y + radius * std::cos(a)),
                           float(centre.z + radius * std::sin(a) * std::sin(b))});
        }
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < 2 * n; ++j) {
            const uint32_t a = uint32_t(2 * n * i + j), b = uint32_t(2 * n * i + (j + 1) % (2 * n));
            for (const uint32_t k : {a, b, a + 2u * n, b, b + 2u * n, a + 2u * n}) m.idx.push_back(k);
        }
    return m;
}
Mesh room(float x, float y0, float y1) {
    Mesh m;
    for (int k = 0; k < 8; ++k) m.p.push_back({k & 1 ? x : -x, k & 2 ? y1 : y0, k & 4 ? x : -x});
    const uint32_t quads[6][4] = {{0, 1, 3, 2}, {4, 6, 7, 5}, {0, 4, 5, 1}, {2, 3, 7, 6}, {0, 2, 6, 4}, {1, 5, 7, 3}};
    for (const auto &q : quads)
        for (const int k : {0, 1, 2, 0, 2, 3}) m.idx.push_back(q[k]);
    return m;
}

// A mirrored or even scale, a rotation and a translation; `plain`: none.
M34 placed(bool plain, double spread) {
    M34 t{{1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {0, 0, 0}};
    if (plain) return t;
    const V3 u = direction();
    V3 v = crs(u, direction());
    const float length = std::sqrt(dt(v, v));
    if (length > 1e-2f) {
        v = {v.x / length, v.y / length, v.z / length};
        t = {u, v, crs(u, v), {}};
    }
    const float k = float(std::pow(10.0, uniform(-0.5, 0.5)) * (rng() % 4u ? 1.0 : -1.0));
    for (V3 *c : {&t.c0, &t.c1, &t.c2}) *c = {c->x * k, c->y * k, c->z * k};
    t.c3 = {float(uniform(-spread, spread)), float(uniform(-spread, spread)), float(uniform(-spread, spread))};
    return t;
}

void traversal() {
    Mesh meshes[] = {sphere(24, 1.0f, {0, 0, 0}), sphere(6, 0.3f, {0, 0, 0}), sphere(40, 2.3f, {4, 1, -7}),
                     room(1.0f, 0.0f, 2.0f), room(0.5f, -0.5f, 0.5f)};
    std::vector<Scene> scenes;
    for (Mesh &m : meshes) {
        m.build();
        scenes.emplace_back();
        scenes.back().add(m, placed(true, 0.0));
    }
    for (const double spread : {0.5, 3.0})
        for (int copies : {1, 6}) {
            scenes.emplace_back();
            for (int k = 0; k < copies; ++k)
                for (const int m : {0, 1, 3, 4}) scenes.back().add(meshes[m], placed(k == 0 && m == 3, spread));
        }
    long rays = 0, ambiguous_rays = 0, changed = 0;
    for (Scene &s : scenes) {
        s.build();
        for (const double distance : {3.0, 30.0, 3000.0})
            for (int n = 0; n < 12000; ++n) {
                // towards an edge or a corner, then on behind each hit
                const uint32_t i = uint32_t(rng() % s.mesh.size());
                const Mesh &m = *s.mesh[i];
                const uint32_t tri = uint32_t(rng() % (m.idx.size() / 3u)), e = uint32_t(rng() % 3u);
                const V3 a = m.p[m.idx[3 * tri + e]], b = m.p[m.idx[3 * tri + (e + 1u) % 3u]];
                const float u = rng() % 8u ? float(uniform(0, 1)) : 0.0f;
                V3 o, d;
                if (!aim(xaff(s.o2w[i], {a.x + u * (b.x - a.x), a.y + u * (b.y - a.y), a.z + u * (b.z - a.z)}, true),
                         distance * uniform(0.01, 1.0), o, d))
                    continue;
                const SceneRay ray(s, o, d);
                float tmin = 0.0f;
                for (int k = 0; k < 3; ++k) {
                    bool ambiguous;
                    const Found bytes = through_bytes(s, ray, tmin, ambiguous), floats = through_floats(s, ray, tmin);
                    ++rays;
                    ambiguous_rays += ambiguous;
                    changed += !(bytes == floats);
                    CHECK(ambiguous || bytes == floats);
                    if (floats.instance == psy::kInvalidId) break;
                    tmin = std::nextafter(floats.t, INFINITY);
                }
            }
    }
    // ambiguity is rare even among such rays, and needed
    std::printf("%ld rays, %ld ambiguous, %ld of these change\n", rays, ambiguous_rays, changed);
    CHECK(rays > 500000 && ambiguous_rays < rays / 50 && changed > 0);
}

}  // namespace

int main() {
    planes();
    slab_tests();
    traversal();
    return 0;
}
