// Test helper (compiled by tests/test_ordered_sum.py): the integer sums of ordered_sum.cuh against std::fma in double,
// term by term. out: terms, sums whose bits differ.
#include <cmath>
#include <cstring>
#include <random>
#define __host__
#define __device__
#define __forceinline__ inline
#include "../kit-sim_daylight_gb300/csrc/ordered_sum.cuh"

extern "C" void ordered_sum_check(int kind, uint64_t seed, int sums, uint64_t out[2]) {
  std::mt19937_64 g(seed * 16 + uint64_t(kind));
  const auto u = [&] { return double(g() >> 11) * (1.0 / 9007199254740992.0); };
  const auto pow2 = [&](int lo, int hi) { return std::ldexp(1.f, lo + int(g() % uint64_t(hi - lo + 1))); };
  for (int t = 0; t < sums; ++t) {
    kgb::OrderedSum s;
    double acc = 0;
    bool bad = false;
    const int n = kind == 0 ? 3000 : 60;
    for (int k = 0; k < n; ++k) {
      float x = 1.f, w = 0.f;
      switch (kind) {
        case 0: x = float(u()); w = float(u() * u() * 1000); break;                          // cosines and weights
        case 1: w = pow2(-30, 30); break;                                                     // ties, terms above the sum
        case 2: x = float(1 + g() % 16) * pow2(-20, 20); w = float(1 + g() % 16) * pow2(-50, 50); break;
        case 3: x = float(0.5 + u()) * pow2(-120, 120); w = float(0.5 + u()) * pow2(-120, 120); break;   // the whole range
        case 4: w = float(g() % 1000); break;                                                 // whole numbers and zeros
        case 5: x = float(u()); w = g() % 3 ? 0.f : float(0.5 + u()) * pow2(-60, 0); break;   // mostly zero weights
        default: x = (1.f + std::ldexp(float(g() % 8), -23)) * pow2(-30, 0); w = (1.f + std::ldexp(float(g() % 8), -23)) * pow2(-30, 0);   // near ties
      }
      uint32_t bx, bw;
      std::memcpy(&bx, &x, 4);
      std::memcpy(&bw, &w, 4);
      if ((x != 0 && kgb::os_odd(bx)) || (w != 0 && kgb::os_odd(bw))) continue;
      acc = std::fma(double(x), double(w), acc);
      kgb::os_add(s, x != 0 && w != 0 ? uint64_t(kgb::os_sig(bx)) * kgb::os_sig(bw) : 0ull, int32_t((bx >> 23) + (bw >> 23)));
      uint64_t b;
      std::memcpy(&b, &acc, 8);
      out[0]++;
      bad = bad || b != kgb::os_bits(s);
    }
    out[1] += bad ? 1 : 0;
  }
}
