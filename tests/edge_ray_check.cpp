// Test helper (compiled by tests/test_edge_rays.py with the engine's host builder): rays that start on or just past a
// triangle's edge, in its plane or a little off it, and leave it almost along that plane, against a loop over every
// triangle, as box_test_check.cpp (whose host forms of the device intrinsics and scene pieces it shares). The distance
// that the triangle test computes for such a ray is the least certain one: it may lie ahead of an origin that is already
// past the triangle, however large the boxes are, so the walk has to find every hit whose triangle's own box, expanded by
// 2^-16 of the scene's largest coordinate, passes the slab test (the oracle's boxes), and nothing that is not a hit.
#include "box_test_check.cpp"

namespace {
bool kept(const Ray& r, F3 v0, F3 v1, F3 v2, float M) {
  const float eps = M * (1.f / 65536.f);
  float in = 1e-5f, out = INFINITY;
  for (int a = 0; a < 3; ++a) {
    const float x0 = comp(v0, a), x1 = comp(v1, a), x2 = comp(v2, a), inv = comp(r.inv, a), o = comp(r.oinv, a);
    const float lo = fmaf(std::min({x0, x1, x2}) - eps, inv, -o), hi = fmaf(std::max({x0, x1, x2}) + eps, inv, -o);
    in = std::max(in, std::min(lo, hi));
    out = std::min(out, std::max(lo, hi));
  }
  return in <= out;
}
}  // namespace

// out: rays, hits (every triangle's), rays whose any-hit set lacks a kept hit or holds something else, rays whose closest
// hit is none or comes after the closest kept one, hits that are not kept
extern "C" void edge_ray_check(uint64_t seed, int kind, int nRays, uint64_t out[5]) {
  Gen G;
  G.g.seed(seed * 100 + uint64_t(kind));
  const float scale[4] = {1.f, 40.f, 500.f, 20000.f}, M = scale[kind % 4];
  for (int b = 0; b < 12; ++b) {   // walls and floors of small quads, axis-aligned or turned
    const F3 o = f3(G.U(-M, M), G.U(-M, M), G.U(-M, M) * 0.3f);
    const float th = kind >= 4 ? G.U(0, 6.28) : 0.f, L = M * G.U(0.02, 0.3), H = M * G.U(0.02, 0.3);
    const F3 a = f3(L * cosf(th), L * sinf(th), 0);
    G.grid(o, a, f3(0, 0, H), 6, 6);
    G.grid(o, a, f3(-a.y, a.x, 0), 5, 5);
  }
  G.grid(f3(-M, -M, -M * .3f), f3(2 * M, 0, 0), f3(0, 2 * M, 0), 1, 1);
  for (int t = 0; t < 40; ++t) {   // triangles of any direction
    const float x = G.U(-M, M), y = G.U(-M, M), z = G.U(-M, M) * .3f, s = M * G.U(1e-3, 1e-1);
    const uint32_t i = G.V(x, y, z), j = G.V(x + G.U(-s, s), y + G.U(-s, s), z + G.U(-s, s));
    G.T(i, j, G.V(x + G.U(-s, s), y + G.U(-s, s), z + G.U(-s, s)));
  }
  const size_t nt = G.tri.size() / 3;
  BvhOut B;
  build_bvh8(G.v.data(), G.v.size() / 3, G.tri.data(), nt, nullptr, nullptr, B);
  std::vector<Node8> nodes(B.nNodes);
  std::vector<TriRec> recs(nt);
  std::memcpy(nodes.data(), B.nodes.data(), B.nodes.size() * 4);
  std::memcpy(recs.data(), B.tris.data(), B.tris.size() * 4);
  const Scene s{nodes.data(), recs.data(), B.nNodes};
  for (int q = 0; q < nRays; ++q) {
    const size_t t = G.g() % nt;
    const int k = int(G.g() % 3);
    const auto corner = [&](int c) { return ld3(&G.v[3 * G.tri[3 * t + (k + c) % 3]]); };
    const F3 a = corner(0), e = sub(corner(1), a), e2 = sub(corner(2), a);
    F3 n = f3(e.y * e2.z - e.z * e2.y, e.z * e2.x - e.x * e2.z, e.x * e2.y - e.y * e2.x);
    const float area2 = sqrtf(dot(n, n)), L2 = std::max(dot(e, e), dot(e2, e2)), L = sqrtf(L2);
    if (!(area2 > 0)) continue;
    n = mul(1 / area2, n);
    F3 m = f3(e.y * n.z - e.z * n.y, e.z * n.x - e.x * n.z, e.x * n.y - e.y * n.x);   // in the plane, across the edge, outwards
    m = mul(1 / sqrtf(dot(m, m)), m);
    const float sine = std::pow(10.f, G.U(-7, -1)) * (G.g() % 2 ? 1.f : -1.f);
    F3 d = add(add(m, mul(G.U(-3, 3) / sqrtf(dot(e, e)), e)), mul(sine, n));
    d = mul(1 / sqrtf(dot(d, d)), d);
    F3 o = add(add(a, mul(G.U(0, 1), e)), mul(L * std::pow(10.f, G.U(-8, -1)), G.g() % 2 ? m : d));
    if (G.g() % 4 == 0) o = add(o, mul(L * std::pow(10.f, G.U(-8, -4)), n));
    const Ray r = make_ray(o, d);
    std::vector<uint32_t> all, must, walk;
    uint32_t overflow = 0, first = ~0u;
    float best = INFINITY;
    for (uint32_t j = 0; j < nt; ++j) {
      F3 v0, v1, v2;
      uint32_t prim, flags, slot;
      Hit h;
      load_tri(recs.data(), j, v0, v1, v2, prim, flags, slot);
      if (!hit_vertices(r, v0, v1, v2, 1e-5f, INFINITY, false, h)) continue;
      all.push_back(prim);
      if (!kept(r, v0, v1, v2, M)) { out[4]++; continue; }
      must.push_back(prim);
      if (h.t < best || (h.t == best && prim < first)) { best = h.t; first = prim; }
    }
    for_hits<false, true>(s, r, 1e-5f, INFINITY, false, [&](const Hit& h, F3, F3, F3, uint32_t, uint32_t) { walk.push_back(h.prim); return false; }, overflow);
    for (auto* x : {&all, &must, &walk}) std::sort(x->begin(), x->end());
    const bool some = std::includes(walk.begin(), walk.end(), must.begin(), must.end()), only = std::includes(all.begin(), all.end(), walk.begin(), walk.end());
    ClosestOut c;
    const bool found = closest<true>(s, r, 1e-5f, FLT_MAX, false, c, overflow);
    out[0]++;
    out[1] += all.size();
    if (!some || !only || overflow) out[2]++;
    if (found ? !std::binary_search(all.begin(), all.end(), c.h.prim) || c.h.t > best || (c.h.t == best && c.h.prim > first) : !must.empty()) out[3]++;
  }
}
