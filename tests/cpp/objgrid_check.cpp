// CPU check of the object grid's rules (interflect_b200/csrc/objgrid.h, the
// header the kernels use) against the reference's traversal: the cells'
// lists are formed over the oracle's objects, and at points inside the scene,
// near its surfaces and along marches every answer that og_exact or
// og_exact_box accepts must be what the oracle's Scene::dist_mat (bvh.rs:100-150, pruned near-first)
// returns, distance bits and material; a dist-only answer may differ where
// both are at or below zero. Along marches of 0.12 steps, og_open_first and
// og_open_next must bound the distances that follow. Prints the counts; exits
// 1 on a disagreement.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <random>
#include <sstream>
#include <unordered_map>

#include "../../interflect_b200/csrc/objgrid.h"
#include "../../oracle/oracle.h"

using namespace orc;

int main(int argc, char** argv) {
    std::ifstream f(argv[1]);
    const int cells = std::atoi(argv[2]);
    std::stringstream ss;
    ss << f.rdbuf();
    Scene sc;
    std::string err;
    if (!parse_scene(ss.str(), sc, err)) {
        std::printf("parse: %s\n", err.c_str());
        return 1;
    }
    std::vector<const Object*> objs;
    for (auto& o : sc.planes) objs.push_back(&o);
    for (uint32_t i : sc.bvh.order) objs.push_back(&sc.objects[i]);
    std::vector<int> leaf(objs.size(), -1);
    for (size_t n = 0; n < sc.bvh.nodes.size(); ++n)
        for (uint32_t k = 0; k < sc.bvh.nodes[n].count; ++k)
            leaf[sc.planes.size() + sc.bvh.nodes[n].start + k] = (int)n;
    const float lo[3] = {sc.lo.x, sc.lo.y, sc.lo.z}, hi[3] = {sc.hi.x, sc.hi.y, sc.hi.z};
    ifx::ObjGrid g{};
    float from[2][3];
    const double diag = sc.diag(), side[2] = {
        ifx::og_level(g.fine, lo, hi, cells, 1.0, 0.0, diag, 0, from[0]),
        ifx::og_level(g.coarse, lo, hi, ifx::kOgCoarseCells, ifx::kOgCoarseExtent, 0.0, diag,
                      g.fine.dim[0] * g.fine.dim[1] * g.fine.dim[2], from[1])};
    // Per cell: its objects and their keys, nearest first, and the nearest distance at the centre.
    struct Cell {
        std::vector<std::pair<uint32_t, uint32_t>> items;
        float base;
    };
    std::unordered_map<uint32_t, Cell> lists;
    auto list_of = [&](uint32_t c) -> const Cell& {
        auto it = lists.find(c);
        if (it != lists.end()) return it->second;
        const int k = c >= g.coarse.base;
        const ifx::OgLevel& l = k ? g.coarse : g.fine;
        const uint32_t i = c - l.base, x = i % l.dim[0], y = i / l.dim[0] % l.dim[1], z = i / (l.dim[0] * l.dim[1]);
        const float s = (float)side[k], *lo = from[k];
        const V3 p(lo[0] + ((float)x + 0.5f) * s, lo[1] + ((float)y + 0.5f) * s, lo[2] + ((float)z + 0.5f) * s);
        float m = 3.4028235e38f;
        std::vector<float> d;
        for (auto* o : objs) {
            d.push_back(o->dist(p));
            m = std::fmin(m, d.back());
        }
        Cell v;
        v.base = m - std::fabs(m) * 1e-3f;  // as much lower as half precision can round
        for (uint32_t i = 0; i < objs.size(); ++i)
            if (ifx::og_listed(d[i], m, ifx::og_margin(ifx::og_half(s, l.delta), l.delta)))
                v.items.push_back({i, ifx::og_key(d[i], v.base, l.key_step)});
        std::stable_sort(v.items.begin(), v.items.end(),
                         [&](auto& a, auto& b) { return d[a.first] < d[b.first]; });
        return lists.emplace(c, v).first->second;
    };
    std::mt19937 rng(7);
    std::uniform_real_distribution<float> U(0.0f, 1.0f);
    long q = 0, bad = 0, outside = 0, ties = 0, unsure = 0, unknown = 0, listed = 0, evaluated = 0, open = 0;
    auto check = [&](V3 p) {
        const DistHit ref = sc.dist_mat(p);
        ++q;
        uint32_t c;
        bool coarse;
        if (!ifx::og_cell(g, p.x, p.y, p.z, c, coarse)) {
            ++outside;
            return ref.d;
        }
        float d1 = 3.4028235e38f, d2 = d1;
        uint32_t o1 = 0;
        const ifx::OgLevel& l = coarse ? g.coarse : g.fine;
        const float delta = l.delta, off = ifx::og_from_centre(l, p.x, p.y, p.z);
        const Cell& cell = list_of(c);
        const bool capped = cell.items.size() > ifx::kOgListLen;
        bool known = true;
        for (size_t n = 0; n < cell.items.size(); ++n) {
            const auto [i, key] = cell.items[n];
            ++listed;
            if (ifx::og_beyond(key, l.key_step, cell.base, off, d1, delta)) break;
            if (capped && n == ifx::kOgListLen - 1) {
                known = false;
                break;
            }
            const float d = objs[i]->dist(p);
            ++evaluated;
            if (d < d1) {
                d2 = d1;
                d1 = d;
                o1 = i;
            } else if (d < d2) {
                d2 = d;
            }
        }
        if (!known) {
            ++unknown;
            return ref.d;
        }
        bool wrong = false;
        for (bool dist_only : {false, true}) {
            bool ok = ifx::og_exact(d1, d2, delta, dist_only);
            if (!ok) {
                if (dist_only) ++ties;
                if (leaf[o1] < 0) {
                    ok = dist_only || d2 > d1;
                } else {
                    const BvhNode& nd = sc.bvh.nodes[leaf[o1]];
                    const V3 b = vmax(vmax(nd.lo - p, p - nd.hi), V3(0.0f, 0.0f, 0.0f));
                    ok = ifx::og_exact_box(d1, d2, std::sqrt(dot(b, b)), dist_only);
                }
            }
            if (!ok) {
                if (dist_only) ++unsure;
            } else if (dist_only) {
                wrong |= !(d1 <= 0.0f && ref.d <= 0.0f) && std::memcmp(&d1, &ref.d, 4) != 0;
            } else {
                wrong |= std::memcmp(&d1, &ref.d, 4) != 0 || objs[o1]->mat != ref.mat;
            }
        }
        if (wrong) {
            if (bad < 5) std::printf("disagree at (%.9g %.9g %.9g): %.9g vs %.9g\n", p.x, p.y, p.z, d1, ref.d);
            ++bad;
        }
        return ref.d;
    };
    for (int i = 0; i < 40000; ++i) {
        V3 p(lo[0] + (hi[0] - lo[0]) * U(rng), lo[1] + (hi[1] - lo[1]) * U(rng), lo[2] + (hi[2] - lo[2]) * U(rng));
        check(p);
        // Toward a surface, then just inside and outside it.
        const V3 rd = normalize(V3(U(rng) - 0.5f, U(rng) - 0.5f, U(rng) - 0.5f));
        float t = 0.0f;
        for (int s = 0; s < 24; ++s) {
            const float d = check(p + rd * t);
            if (std::fabs(d) < 1e-4f) {
                for (float e : {-3e-3f, -5e-4f, -1e-6f, 1e-6f, 5e-4f, 3e-3f}) check(p + rd * (t + e));
                break;
            }
            t += d;
        }
        float h = sc.dist(p), lower = ifx::og_open_first(h, g.coarse.delta);
        t = 0.0f;
        for (int s = 0; s < 60; ++s) {
            t += ifx::kOpenStep;
            const float d = sc.dist(p + rd * t);
            if (lower >= ifx::kOpenStep) {
                ++open;
                if (!(d >= lower)) {
                    std::printf("bound %.9g above the distance %.9g\n", lower, d);
                    ++bad;
                }
                lower = ifx::og_open_next(lower);
            } else {
                lower = ifx::og_open_first(d, g.coarse.delta);
            }
        }
    }
    std::printf("objects %zu, queries %ld, mean listed %.2f evaluated %.2f, outside %ld, unknown %ld, near ties %ld (unsure %ld), open steps %ld, "
                "disagreements %ld\n",
                objs.size(), q, (double)listed / q, (double)evaluated / q, outside, unknown, ties, unsure, open, bad);
    if (bad) return 1;
    std::printf("every accepted answer equals the reference traversal\n");
    return 0;
}
