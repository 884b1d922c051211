// A double sum of products of floats, term by term in order, in integer arithmetic: acc = fma(x, w, acc) with x >= 0 and
// w >= 0 floats widened to double, bit for bit, without the FP64 pipe.
//
// GB300's FP64 pipe takes 0.84 terms a clock per SM, and a chain of fmas waits over 250 cycles a term. The sums of the
// reduces are such chains, whose order decides their bits. But a sum's rounding is simple while its exponent stays: the
// product of two 24-bit significands is exact in 48 bits, and adding it to the accumulator's 53-bit significand is an
// integer addition of its whole part, rounded to nearest even by its remainder. So the terms of many directions can be
// rounded at once, and only the terms that take the sum into the next binade have to be added by themselves (k_sum_warp,
// reduce.cu: 16 sensors x 4746 directions 0.94 to 0.10 ms a call). One thread a sensor, term by term in this form, was
// no faster than the fmas: some 160 issue slots a term.
//
// The accumulator is a 2^(g - 300), a = 0 or 2^52 <= a < 2^53; a term is p 2^(e - 300), p = 0 or 2^46 <= p < 2^48 (the
// biased exponents of x and w add up to e, each significand counting 2^-150).
#pragma once
#include <cstdint>

namespace kgb {

struct OrderedSum {
  uint64_t a = 0;
  int32_t g = 0;
};

__host__ __device__ __forceinline__ int os_clz(uint64_t x) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)x);
#else
  return __builtin_clzll(x);
#endif
}

// The whole part q of a + p 2^-sh (0 <= sh <= 63) and its remainder in units of 2^-64, rounded to nearest even; a term
// of p = 0 changes nothing. p < 2^48, so the sum passes 2^53 by at most one bit.
__host__ __device__ __forceinline__ void os_round(OrderedSum& s, uint64_t p, uint32_t sh) {
  const uint64_t q = s.a + (p >> sh), rem = (p << (63u - sh)) << 1;
  const uint64_t up = rem + (0x7fffffffffffffffull + (q & 1u));   // carries when the remainder rounds up
  s.a = q + (up < rem ? 1u : 0u);
  if (s.a >> 53) {   // the next binade: rounded once, on its own grid
    if (q >> 53) {
      const uint64_t h = q >> 1;
      s.a = h + ((q & 1u) && (rem || (h & 1u)) ? 1u : 0u);
    } else {
      s.a = 1ull << 52;
    }
    s.g++;
  }
}

// The terms the fast path leaves out: the first one, and one whose lowest bit lies above the accumulator's.
__host__ __device__ inline void os_add_rare(OrderedSum& s, uint64_t p, int32_t e) {
  const int lead = os_clz(p) - 11;
  if (!s.a) { s.a = p << lead; s.g = e - lead; return; }
  const int up = e - s.g;
  if (up > 15) {   // the term is far larger: the accumulator is what is added
    OrderedSum t;
    t.a = p << lead;
    t.g = e - lead;
    const int sh = t.g - s.g;
    // the accumulator has 53 bits, so its part above 2^48 is none here: sh >= 10
    const uint64_t q = t.a + (sh > 63 ? 0ull : s.a >> sh);
    const uint64_t rem = sh > 63 ? (sh == 64 ? s.a : 1ull) : (s.a << (63 - sh)) << 1;
    const uint64_t c = rem + (0x7fffffffffffffffull + (q & 1u));
    t.a = q + (c < rem ? 1u : 0u);
    if (t.a >> 53) {
      if (q >> 53) { const uint64_t h = q >> 1; t.a = h + ((q & 1u) && (rem || (h & 1u)) ? 1u : 0u); }
      else t.a = 1ull << 52;
      t.g++;
    }
    s = t;
    return;
  }
  const uint64_t q = s.a + (p << up);   // exact: p < 2^48, up <= 15
  const int k = 11 - os_clz(q);         // bits past 53
  if (k <= 0) { s.a = q; return; }
  const uint64_t low = q & ((1ull << k) - 1ull), half = 1ull << (k - 1), h = q >> k;
  s.a = h + (low > half || (low == half && (h & 1u)) ? 1u : 0u);
  s.g += k;
  if (s.a >> 53) { s.a = 1ull << 52; s.g++; }
}

__host__ __device__ __forceinline__ void os_add(OrderedSum& s, uint64_t p, int32_t e) {
  const int32_t sh = s.g - e;
  if (p && (sh < 0 || !s.a)) { os_add_rare(s, p, e); return; }
  os_round(s, p, uint32_t(sh) < 63u ? uint32_t(sh) : 63u);
}

__host__ __device__ __forceinline__ uint64_t os_bits(const OrderedSum& s) {   // the sum as a double's bits
  return s.a ? (uint64_t(uint32_t(s.g + 775)) << 52) + (s.a - (1ull << 52)) : 0ull;
}

// The significand of a normal float (its biased exponent: bits >> 23); os_odd: not a positive normal float.
__host__ __device__ __forceinline__ uint32_t os_sig(uint32_t bits) { return (bits & 0x7fffffu) | 0x800000u; }
__host__ __device__ __forceinline__ bool os_odd(uint32_t bits) { return (bits >> 23) - 1u >= 254u; }

}  // namespace kgb
