// Test helper (compiled by tests/test_box_test.py with the engine's host builder): the device traversal of rt.cuh,
// compiled for the CPU, against a loop over every triangle. The rays are made where a box test that is not conservative
// drops hits: through edges and vertices, grazing, lifted off their own face, along an axis (or a tiny component away from
// it), from far outside; the scenes hold coplanar grids, a ground and a strip of two triangles each, needles and small
// triangles, at four scales.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

// the device intrinsics the header uses, on the CPU
#undef __device__
#undef __forceinline__
#define __device__
#define __forceinline__ inline
template <class T> inline T __ldg(const T* p) { return *p; }
inline uint32_t __float_as_uint(float f) { uint32_t r; std::memcpy(&r, &f, 4); return r; }
inline float __uint_as_float(uint32_t u) { float r; std::memcpy(&r, &u, 4); return r; }
inline int __float_as_int(float f) { int r; std::memcpy(&r, &f, 4); return r; }
inline float __int_as_float(int u) { float r; std::memcpy(&r, &u, 4); return r; }
inline int __ffs(int x) { return __builtin_ffs(x); }
inline int __popc(unsigned x) { return __builtin_popcount(x); }
inline double __hiloint2double(int h, int l) { const uint64_t v = (uint64_t(uint32_t(h)) << 32) | uint32_t(l); double d; std::memcpy(&d, &v, 8); return d; }
inline uint32_t min(uint32_t a, uint32_t b) { return a < b ? a : b; }
#include "../kit-sim_daylight_gb300/csrc/rt.cuh"

using namespace kgb;

namespace {
struct Gen {
  std::mt19937_64 g;
  std::vector<float> v;
  std::vector<uint32_t> tri;
  float U(double a, double b) { return float(a + (b - a) * (double(g() >> 11) * (1.0 / 9007199254740992.0))); }
  uint32_t V(float x, float y, float z) { v.push_back(x); v.push_back(y); v.push_back(z); return uint32_t(v.size() / 3 - 1); }
  void T(uint32_t a, uint32_t b, uint32_t c) { tri.push_back(a); tri.push_back(b); tri.push_back(c); }
  void grid(F3 o, F3 a, F3 b, int na, int nb) {
    const uint32_t base = uint32_t(v.size() / 3);
    for (int j = 0; j <= nb; ++j)
      for (int i = 0; i <= na; ++i) {
        const float s = float(i) / na, t = float(j) / nb;
        V(o.x + a.x * s + b.x * t, o.y + a.y * s + b.y * t, o.z + a.z * s + b.z * t);
      }
    for (int j = 0; j < nb; ++j)
      for (int i = 0; i < na; ++i) {
        const uint32_t q = base + uint32_t(j * (na + 1) + i), w = uint32_t(na) + 1;
        T(q, q + 1, q + w + 1);
        T(q, q + w + 1, q + w);
      }
  }
};
}  // namespace

// out: rays, hits (every triangle's), rays whose any-hit set differs, rays whose closest hit differs
extern "C" void box_test_check(uint64_t seed, int kind, int nRays, uint64_t out[4]) {
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
  G.grid(f3(-M, -M, -M * .29f), f3(2 * M, 0, 0), f3(0, M * 0.004f, 0), 1, 1);
  for (int t = 0; t < 40; ++t) {   // needles
    const uint32_t i = G.V(G.U(-M, M), G.U(-M, M), G.U(-M, M) * .3f), j = G.V(G.U(-M, M), G.U(-M, M), G.U(-M, M) * .3f);
    const F3 p = ld3(&G.v[3 * j]);
    G.T(i, j, G.V(p.x + M * G.U(-1e-3, 1e-3), p.y + M * G.U(-1e-3, 1e-3), p.z));
  }
  for (int t = 0; t < 60; ++t) {   // small triangles
    const float x = G.U(-M, M), y = G.U(-M, M), z = G.U(-M, M) * .3f, s = M * G.U(1e-4, 1e-1);
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
  const auto corner = [&](size_t t, int k) { return ld3(&G.v[3 * G.tri[3 * t + k]]); };
  const float tiny[7] = {0.f, 1e-30f, 1e-9f, 1e-6f, 1e-4f, 3e-3f, 5e-3f};
  for (int q = 0; q < nRays; ++q) {
    const size_t t = G.g() % nt;
    const F3 a = corner(t, 0), e1 = sub(corner(t, 1), a), e2 = sub(corner(t, 2), a);
    float u = G.U(0, 1), w = G.U(0, 1);
    if (u + w > 1) { u = 1 - u; w = 1 - w; }
    if (q % 3 == 0) u = 0;        // on an edge
    if (q % 7 == 0) w = 1 - u;
    const F3 p = add(add(a, mul(u, e1)), mul(w, e2));
    F3 n = f3(e1.y * e2.z - e1.z * e2.y, e1.z * e2.x - e1.x * e2.z, e1.x * e2.y - e1.y * e2.x);
    float l = sqrtf(dot(n, n));
    if (!(l > 0)) continue;
    n = mul(1 / l, n);
    const int axis = int(G.g() % 3);
    const auto at = [&](F3& x) -> float& { return axis == 0 ? x.x : axis == 1 ? x.y : x.z; };
    F3 o, d;
    switch (q % 6) {
      case 0: case 1:   // off its own face; grazing
        o = offset_ray(p, n);
        d = f3(G.U(-1, 1), G.U(-1, 1), G.U(-1, 1));
        if (q % 6 == 1) d = sub(d, mul(dot(d, n) * (1 - G.U(-1e-5, 1e-3)), n));
        break;
      case 2: {   // from anywhere, and from far outside
        const float far = q % 4 == 0 ? 1.f : 30.f;
        o = f3(G.U(-M, M) * far, G.U(-M, M) * far, G.U(-M, M) * far);
        d = sub(p, o);
        break;
      }
      case 3:   // along an axis' planes
        o = f3(G.U(-M, M), G.U(-M, M), G.U(-M, M));
        d = sub(p, o);
        at(o) = at(const_cast<F3&>(p));
        at(d) = tiny[G.g() % 7] * (G.g() % 2 ? 1.f : -1.f);
        break;
      case 4: {   // from just above or below a face
        o = p;
        float h = G.U(-1e-3, 1e-3) * M;
        if (G.g() % 2) h *= 1e-3f;
        at(o) += h;
        d = f3(G.U(-1, 1), G.U(-1, 1), G.U(-1, 1));
        if (G.g() % 2) at(d) *= 1e-4f;
        break;
      }
      default: {   // from a face to another triangle's edge
        const size_t t2 = G.g() % nt;
        o = offset_ray(p, n);
        d = sub(add(corner(t2, 0), mul(u, sub(corner(t2, 1), corner(t2, 0)))), o);
      }
    }
    l = sqrtf(dot(d, d));
    if (!(l > 0)) continue;
    d = mul((q % 11 ? 1.f : G.U(0.01, 50)) / l, d);
    const Ray r = make_ray(o, d);
    std::vector<uint32_t> all, walk;
    uint32_t overflow = 0, first = 0;
    float best = INFINITY;
    for (uint32_t k = 0; k < nt; ++k) {
      F3 v0, v1, v2;
      uint32_t prim, flags, slot;
      Hit h;
      load_tri(recs.data(), k, v0, v1, v2, prim, flags, slot);
      if (!hit_vertices(r, v0, v1, v2, 1e-5f, INFINITY, false, h)) continue;
      all.push_back(prim);
      if (h.t < best || (h.t == best && prim < first)) { best = h.t; first = prim; }
    }
    const auto note = [&](const Hit& h, F3, F3, F3, uint32_t, uint32_t) { walk.push_back(h.prim); return false; };
    if (q % 2) for_hits<false, false>(s, r, 1e-5f, INFINITY, false, note, overflow);   // both forms of the triangle test
    else for_hits<false, true>(s, r, 1e-5f, INFINITY, false, note, overflow);
    std::sort(all.begin(), all.end());
    std::sort(walk.begin(), walk.end());
    ClosestOut c;
    const bool found = closest<true>(s, r, 1e-5f, FLT_MAX, false, c, overflow);
    out[0]++;
    out[1] += all.size();
    if (all != walk || overflow) out[2]++;
    if (found == all.empty() || (found && (c.h.t != best || c.h.prim != first))) out[3]++;
  }
}
