// Test helper (compiled by tests/test_frontier_build.py with the engine's host builder): rt.cuh's frontier, built on the
// CPU by 32 threads that stand for a warp's lanes. Sound trees: the entries' subtrees hold every triangle exactly once,
// for origins in one place, spread over the scene, and with lanes that are not finite or have no sensor. Damaged trees (a
// node that is its own only child, inner nodes without children): the build ends, with entries within its arrays.
#include <cuda_runtime.h>
#include <pthread.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <random>
#include <thread>
#include <vector>

#include "../kit-sim_daylight_gb300/csrc/engine.h"

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
inline uint32_t max(uint32_t a, uint32_t b) { return a > b ? a : b; }
// the warp's collectives, by a barrier on each side of the exchange
static pthread_barrier_t gBar;
static uint32_t gWord[32];
static thread_local uint32_t tLane;
struct Lane3 { uint32_t x, y, z; };
#define threadIdx (Lane3{tLane, 0, 0})
inline void __syncwarp() { pthread_barrier_wait(&gBar); }
template <class F> inline uint32_t exchange(uint32_t v, F f) {
  gWord[tLane] = v;
  __syncwarp();
  const uint32_t r = f();
  __syncwarp();
  return r;
}
inline uint32_t __ballot_sync(unsigned, bool p) { return exchange(p, [] { uint32_t m = 0; for (int k = 0; k < 32; ++k) m |= gWord[k] << k; return m; }); }
inline bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
inline uint32_t __reduce_max_sync(unsigned, uint32_t v) { return exchange(v, [] { return *std::max_element(gWord, gWord + 32); }); }
inline uint32_t __reduce_min_sync(unsigned, uint32_t v) { return exchange(v, [] { return *std::min_element(gWord, gWord + 32); }); }
inline uint32_t __shfl_sync(unsigned, uint32_t v, int from) { return exchange(v, [&] { return gWord[from]; }); }
#define __CUDACC__ 1
#include "../kit-sim_daylight_gb300/csrc/rt.cuh"
#undef __CUDACC__

using namespace kgb;

static void warp(const std::function<void(uint32_t)>& f) {
  pthread_barrier_init(&gBar, nullptr, 32);
  std::vector<std::thread> t;
  for (uint32_t k = 0; k < 32; ++k) t.emplace_back([&, k] { tLane = k; f(k); });
  for (auto& x : t) x.join();
  pthread_barrier_destroy(&gBar);
}

// 0: right; else which check failed. damage: 0 none, 1 the first inner child of some nodes is the node itself and its only
// child, 2 some inner nodes have no children. out: entries.
extern "C" int frontier_check(uint64_t seed, int damage, int spread, uint32_t* out) {
  std::mt19937_64 g(seed);
  const auto U = [&](double a, double b) { return float(a + (b - a) * (double(g() >> 11) * (1.0 / 9007199254740992.0))); };
  const uint32_t nt = seed % 5 == 0 ? 1 : 3000;
  std::vector<float> v;
  std::vector<uint32_t> tri;
  for (uint32_t t = 0; t < nt; ++t) {
    const float c[3] = {U(-50, 50), U(-50, 50), U(0, 10)};
    for (int k = 0; k < 3; ++k) {
      for (int a = 0; a < 3; ++a) v.push_back(c[a] + U(-1, 1));
      tri.push_back(3 * t + uint32_t(k));
    }
  }
  BvhOut B;
  build_bvh8(v.data(), v.size() / 3, tri.data(), nt, nullptr, nullptr, B);
  std::vector<Node8> nodes(B.nNodes);
  std::memcpy(nodes.data(), B.nodes.data(), B.nodes.size() * 4);
  if (damage)
    for (uint32_t w = 0; w < B.nNodes; ++w) {
      uint32_t* r = reinterpret_cast<uint32_t*>(&nodes[w]);
      const uint32_t imask = r[0] >> 24;
      if (!imask || (damage == 2 && w == 0)) continue;
      const int k = __builtin_ctz(imask);
      r[0] = damage == 1 ? (1u << (24 + k)) | w : 0u;
      r[2] = r[3] = 0u;
      for (int f = 0; f < 6; ++f) reinterpret_cast<float*>(r)[4 + 8 * f + k] = f % 2 ? 1000.f : -1000.f;
    }
  const Scene s{nodes.data(), nullptr, B.nNodes};
  F3 at[32];
  bool valid[32];
  for (int k = 0; k < 32; ++k) {
    const float d = spread == 0 ? 1.f : spread == 1 ? 20.f : 0.01f;
    at[k] = f3(U(-d, d), U(-d, d), 5 + U(-d, d) * 0.1f);
    if (spread == 2 && k % 5 == 1) at[k].x = k % 2 ? NAN : -INFINITY;
    valid[k] = spread != 2 || k < 30;
  }
  Frontier f;
  uint32_t n = 0;
  warp([&](uint32_t lane) {
    const Bounds b = origin_bounds(at[lane], valid[lane]);
    const uint32_t m = build_frontier(s, b, f, lane);
    if (!lane) n = m;
  });
  *out = n;
  if (n > uint32_t(kEntries)) return 1;
  for (uint32_t e = 0; e < n; ++e) if (!f.ref[e].y && f.ref[e].x >= B.nNodes) return 2;
  if (damage) return 0;
  std::vector<uint32_t> seen(nt, 0), todo;
  const auto leaf = [&](uint32_t first, uint32_t cnt) { for (uint32_t j = first; j < first + cnt; ++j) if (j < nt) seen[j]++; };
  for (uint32_t e = 0; e < n; ++e) if (f.ref[e].y) leaf(f.ref[e].x, f.ref[e].y); else todo.push_back(f.ref[e].x);
  while (!todo.empty()) {
    const uint32_t* r = reinterpret_cast<const uint32_t*>(&nodes[todo.back()]);
    todo.pop_back();
    uint32_t rank = 0;
    for (int k = 0; k < 8; ++k) {
      const uint32_t meta = ((k < 4 ? r[2] : r[3]) >> (8 * (k & 3))) & 0x7fu;
      if (r[0] >> (24 + k) & 1u) todo.push_back((r[0] & 0xffffffu) + rank++);
      else if (meta) leaf(r[1] + (meta & 31u), meta >> 5);
    }
  }
  return std::all_of(seen.begin(), seen.end(), [](uint32_t x) { return x == 1; }) ? 0 : 3;
}
