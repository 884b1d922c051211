// Accumulation kernels over the visibility the ray-casting kernels leave on the device (compiled with -fmad=false):
//  k_reduce_bits / k_reduce_bytes / k_reduce_dc  out[i] = sum over d (or bins) in order of
//      double(float(max(0, N_i . D_d) x T) ) x W[d]   (replaces the reference's k_reduce, gpu.cu:99-114)
//  k_view_reduce  per sensor and class: weight, weight x ln d, min d; own weight; reach; glazing (replaces k_view,
//      gpu.cu:238-274), one warp per sensor, lane l summing d = l, l + 32, ..., then a fixed shuffle tree
//  k_iso          the isovist area / volume through the rays' end points (replaces k_iso + iso_lane, gpu.cu:187-236)
// The summation orders are fixed (direction order per thread; lane order + shuffle tree per warp), so a sensor's
// doubles do not depend on the chunk it is in, and equal the oracle's restatement bit for bit.
#include "engine.h"
#include "ordered_sum.cuh"
#include "rt.cuh"

namespace kgb {

__device__ __forceinline__ float dotf(F3 a, F3 b) { return (a.x * b.x + a.y * b.y) + a.z * b.z; }   // per-op rounding (gpu.cu:69-72)

// GB300's FP64 pipe is narrow (a few lanes per clock per SM), so each term of a sum costs one FP64 instruction:
//  - the float factor x > 0 becomes a double exactly by integer operations (widen, rt.cuh);
//  - the weights are read as doubles: converted once per call into a device array (or, where the caller has no room
//    for one, once per block into shared memory);
//  - the product of two floats is exact in double, so fma(x, w, acc) equals acc + x * w rounded once, as the
//    reference's separate multiply and add;
//  - a zero factor adds +0, which leaves the sum as it is: it is skipped.

constexpr uint32_t kReduceSmemDirs = 24576;   // weights held as doubles in shared memory (192 KB) up to this many

template <bool SMEM>
__device__ __forceinline__ const double* weights_to_smem(const float* W, uint32_t n, double* sW) {
  if constexpr (SMEM) {
    for (uint32_t d = threadIdx.x; d < n; d += blockDim.x) sW[d] = (double)__ldg(W + d);
    __syncthreads();
    return sW;
  } else {
    return nullptr;
  }
}
template <bool SMEM>
__device__ __forceinline__ double weight(const double* sW, const float* W, uint32_t d) { return SMEM ? sW[d] : (double)__ldg(W + d); }

template <bool SMEM>
__global__ void __launch_bounds__(256) k_reduce_bits(const uint32_t* __restrict__ bits, uint32_t nc, uint32_t nWords, uint32_t nDir,
                                                     const float* __restrict__ N, const float* __restrict__ D, const float* __restrict__ W,
                                                     int useCos, double* __restrict__ out) {
  extern __shared__ double sW[];
  const double* w64 = weights_to_smem<SMEM>(W, nDir, sW);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  const F3 n = ld3(N + 3 * size_t(i));
  double acc = 0;
  for (uint32_t w = 0; w < nWords; ++w) {
    uint32_t m = bits[size_t(w) * nc + i];
    while (m) {
      const uint32_t d = w * 32 + (__ffs(m) - 1);
      m &= m - 1;
      const float c = useCos ? fmaxf(dotf(n, ld3(D + 3 * d)), 0.f) : 1.f;
      if (c != 0.f) acc = __fma_rn(widen(c), weight<SMEM>(w64, W, d), acc);
    }
  }
  out[i] = acc;
}

template <bool SMEM>
__global__ void __launch_bounds__(256) k_reduce_bytes(const uint8_t* __restrict__ bytes, uint32_t nc, uint32_t nDir, const float* __restrict__ N,
                                                      const float* __restrict__ D, const float* __restrict__ W, int useCos, double* __restrict__ out) {
  extern __shared__ double sW[];
  const double* w64 = weights_to_smem<SMEM>(W, nDir, sW);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  const F3 n = ld3(N + 3 * size_t(i));
  double acc = 0;
  // 16 directions' bytes are loaded before any is used (16 loads in flight per thread: a chunk of the reference's
  // size leaves few threads per SM), then added in direction order
  constexpr uint32_t G = 16;
  for (uint32_t d0 = 0; d0 < nDir; d0 += G) {
    uint32_t bb[G];
#pragma unroll
    for (uint32_t k = 0; k < G; ++k) bb[k] = d0 + k < nDir ? uint32_t(__ldg(bytes + size_t(d0 + k) * nc + i)) : 0u;
#pragma unroll
    for (uint32_t k = 0; k < G; ++k) {
      if (!bb[k]) continue;
      const uint32_t d = d0 + k;
      const float at = float(bb[k]) / 255.f;
      const float c = useCos ? fmaxf(dotf(n, ld3(D + 3 * d)), 0.f) : 1.f;
      const float x = c * at;
      if (x != 0.f) acc = __fma_rn(widen(x), weight<SMEM>(w64, W, d), acc);
    }
  }
  out[i] = acc;
}

__global__ void __launch_bounds__(256) k_reduce_dc(const float* __restrict__ dc, uint32_t nc, uint32_t nBins, const float* __restrict__ W, double* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  double acc = 0;
  for (uint32_t b = 0; b < nBins; ++b) acc += (double)(1.f * dc[size_t(b) * nc + i]) * (double)__ldg(W + b);
  out[i] = acc;
}

// widen (rt.cuh) for either sign and for zero: a conversion instruction takes the FP64 pipe, which bounds k_view_reduce
// (12,000 sensors x 3600 cells 637 to 559 us, 25,000 x 16,200 with reach and isovist 5.92 to 5.68 ms)
__device__ __forceinline__ double widen_signed(float x) {
  const uint32_t b = __float_as_uint(x), m = b & 0x7fffffffu;
  return __hiloint2double(int((b & 0x80000000u) | (m ? (m >> 3) + (896u << 20) : 0u)), int(b << 29));
}
__device__ __forceinline__ double warp_sum(double v) {
  for (uint32_t s = 16; s; s >>= 1) v += __shfl_down_sync(~0u, v, s);
  return v;
}

// One warp per sensor. A lane's per-class sums sit in shared memory as [class][lane] (a warp's lanes touch 32
// different banks whatever their classes), so a ray costs its own class's three updates, not a select over every
// class: GB300's FP64 pipe is narrow, and predicated double operations still take its slots. Classes at or past nClass
// are never reported and are not kept; the reach sums likewise hold nReach slots.
constexpr uint32_t kViewWarps = 8;   // warps (sensors) per block
__global__ void __launch_bounds__(256) k_view_reduce(ViewReduceArgs a) {
  extern __shared__ double vsm[];
  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x & 31, i = blockIdx.x * kViewWarps + warp;
  const uint32_t C = a.nClass, R = a.nReach;
  double* sw = vsm + size_t(warp) * (2 * C + R) * 32;   // w [C][32], wl [C][32], reach [R][32]
  double* swl = sw + C * 32;
  double* src = swl + C * 32;
  float* smn = reinterpret_cast<float*>(vsm + size_t(kViewWarps) * (2 * C + R) * 32) + size_t(warp) * C * 32;   // mn [C][32]
  for (uint32_t c = 0; c < C; ++c) { sw[c * 32 + lane] = 0; swl[c * 32 + lane] = 0; smn[c * 32 + lane] = __int_as_float(0x7f800000); }
  for (uint32_t r = 0; r < R; ++r) src[r * 32 + lane] = 0;
  if (i >= a.nc) return;   // whole warps
  double own = 0, gz = 0;
  for (uint32_t d = lane; d < a.K; d += 32) {
    uint32_t c = a.cls[size_t(d) * a.nc + i];
    const float t = a.dist[size_t(d) * a.nc + i];
    const double wd = a.wRow[d / a.nAz];
    if (c == 254) { own += wd; continue; }
    if (c & KGB_VIEW_GLAZED) { gz += wd; c &= ~uint32_t(KGB_VIEW_GLAZED); }
    const float dd = fminf(fmaxf(t, 0.1f), a.farDist);
    const double ln = dd == a.farDist ? a.lnFar : dd == 0.1f ? -2.302585092994045684 : widen_signed(kgb_logf(dd));
    if (c < C) {
      const uint32_t at = c * 32 + lane;
      sw[at] += wd;
      swl[at] += wd * ln;
      smn[at] = fminf(smn[at], dd);
    }
    for (uint32_t r = 0; r < R; ++r) if (t >= a.reach[r]) src[r * 32 + lane] += wd;
  }
  double* o = a.out + size_t(i) * a.NA;
  for (uint32_t c = 0; c < C; ++c) {
    float m = smn[c * 32 + lane];
    for (uint32_t s = 16; s; s >>= 1) m = fminf(m, __shfl_down_sync(~0u, m, s));
    const double x = warp_sum(sw[c * 32 + lane]), y = warp_sum(swl[c * 32 + lane]);
    if (!lane) { o[3 * c] = x; o[3 * c + 1] = y; o[3 * c + 2] = m; }
  }
  const double ow = warp_sum(own);
  if (!lane) o[3 * C] = ow;
  for (uint32_t r = 0; r < R; ++r) {
    const double x = warp_sum(src[r * 32 + lane]);
    if (!lane) o[3 * C + 1 + r] = x;
  }
  if (a.glazing) {
    const double x = warp_sum(gz);
    if (!lane) o[3 * C + 1 + R] = x;
  }
}

// view cell of direction d (the reference's view_cell, params.h:77-89), sincospif as kgb_sincospi
__device__ __forceinline__ F3 iso_cell(uint32_t d, uint32_t col, float rsx, float rsy, float az0, float dAz, bool jitter, uint32_t element, uint32_t side) {
  float a = 0.5f, s = 0.5f * (rsx + rsy);
  if (jitter) { const U3 h = pcg3d(element, d, side); a = u01(h.x); s = rsx + u01(h.y) * (rsy - rsx); }
  float sa, ca;
  kgb_sincospi((az0 + (float(col) + a) * dAz) * (1.f / 180.f), &sa, &ca);
  const float c = sqrtf(fmaxf(0.f, 1.f - s * s));
  return f3(c * sa, c * ca, s);
}
__device__ __forceinline__ float det3(F3 a, F3 b, F3 c) {
  const F3 u = sub(b, a), w = sub(c, a);
  return a.x * (u.y * w.z - u.z * w.y) + a.y * (u.z * w.x - u.x * w.z) + a.z * (u.x * w.y - u.y * w.x);
}

// Isovist of a sensor, one warp per sensor. A ray's end point is its clipped length (0 on the sensor's own surface, at
// most farDist) along its cell's direction in the field's own frame. isoDim 2: the area of the polygon through row 0's
// end points, one triangle (eye, column c, column c + 1) per column. isoDim 3: the volume enclosed by the end points,
// as the signed volumes of two tetrahedra with the eye per cell quad between rows r - 1 and r and columns c and c + 1.
// Column c + 1 of the last column is column 0 for a full circle; a narrower fan has no piece after its last column.
// Lane l owns the columns l, l + 32, ... Each piece is evaluated in float and added to the lane's double sum in row
// order; the lanes' sums are then combined by warp_sum's fixed tree. Those two orders and the float expressions of the
// pieces decide the resulting double, so they are kept equal to the reference's k_iso (gpu.cu:197-236).
__device__ __forceinline__ float iso_len(const ViewReduceArgs& a, uint32_t i, uint32_t k) {
  const size_t at = size_t(k) * a.nc + i;
  return a.cls[at] == 254 ? 0.f : fminf(a.dist[at], a.farDist);
}
// The cells' directions (a hash, a sine and cosine, a square root) are most of the work. A lane takes the next column's
// direction and length from lane + 1, except where lane + 1 does not hold it (lane 31, or the wrap to column 0): that
// column, one to a group of 32, is computed by all lanes at once, a row each, every 32 rows. (With both columns' directions
// computed by each lane: the view reduces of 25,000 sensors x 16,200 cells 7.02 ms against 5.93, of 300 x 7200 315 us
// against 244.)
__global__ void __launch_bounds__(256) k_iso(ViewReduceArgs a) {
  const uint32_t i = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
  if (i >= a.nc) return;   // the whole warp leaves together
  const uint32_t gi = a.i0 + i, element = gi / a.nS, side = a.nS == 2 ? gi % 2 : a.back;
  const bool jit = a.jitter != 0;
  const uint32_t rows = a.isoDim == 2 ? 1 : a.nEl;
  double sum = 0;
  for (uint32_t base = 0; base < a.nAz; base += 32) {
    // lanes past the last column repeat it and add nothing, but still take part in the shuffles
    const uint32_t col = min(base + lane, a.nAz - 1), edge = base + 32 < a.nAz ? base + 32 : 0;
    const bool last = col + 1 == a.nAz, adds = base + lane < a.nAz && (a.world || !last), atEdge = lane == 31 || last;
    F3 up0{}, up1{}, edgeDir{};
    float topHere = 0.f, topNext = 0.f, edgeLen = 0.f;
    for (uint32_t r = 0; r < rows; ++r) {
      if (!(r & 31u)) {
        const uint32_t q = min(r + lane, rows - 1), k = q * a.nAz + edge;
        edgeDir = iso_cell(k, edge, a.rowSin[2 * q], a.rowSin[2 * q + 1], a.az0, a.dAz, jit, element, side);
        edgeLen = iso_len(a, i, k);
      }
      const uint32_t d = r * a.nAz + col;
      const float here = iso_len(a, i, d);
      const F3 lo0 = iso_cell(d, col, a.rowSin[2 * r], a.rowSin[2 * r + 1], a.az0, a.dAz, jit, element, side);
      const auto beside = [&](float own, float edges) {
        const float x = __shfl_down_sync(~0u, own, 1), y = __shfl_sync(~0u, edges, int(r & 31u));
        return atEdge ? y : x;
      };
      const F3 lo1 = f3(beside(lo0.x, edgeDir.x), beside(lo0.y, edgeDir.y), beside(lo0.z, edgeDir.z));
      const float next = beside(here, edgeLen);
      if (a.isoDim == 2) {   // the triangle's area: half the two lengths times the sine of the clockwise turn
        if (adds) sum += double(0.5f * here * next * (lo0.y * lo1.x - lo0.x * lo1.y));
      } else if (r && adds) {
        // six times the volumes of (eye, up0, up1, lo0) and (eye, up1, lo1, lo0), each determinant scaled by its lengths
        sum += double(topHere * topNext * here * det3(up0, up1, lo0) + topNext * next * here * det3(up1, lo1, lo0));
      }
      up0 = lo0; up1 = lo1; topHere = here; topNext = next;
    }
  }
  const double v = warp_sum(a.isoDim == 2 ? sum : sum / 6);
  if (!lane) a.out[size_t(i) * a.NA + a.NA - 1] = v;
}

// The weights go to shared memory as doubles when they fit (kReduceSmemDirs); the kernels' sums are the same either way.
static bool reduce_smem_ready() {
  static bool ok = [] {
    const int bytes = int(kReduceSmemDirs * sizeof(double));
    return cudaFuncSetAttribute(k_reduce_bits<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess &&
           cudaFuncSetAttribute(k_reduce_bytes<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
  }();
  return ok;
}
// The weights as doubles in global memory (read through L1), one thread per sensor in blocks of 128: no shared memory
// per block, so the SMs hold as many blocks as their registers allow and take new ones as blocks end. The shared-memory
// form below (a block's copy of every weight, 45 KB at 5610 directions) kept four or five 256-thread blocks an SM, about
// one wave for the urban block, and the blocks of heavy sensors (roofs see most directions) held their SMs while the
// others idled: the urban step's four reduces took 8.85 ms that way, 4.93 ms this way (sums bit-identical; blocks of
// 64 and 256 threads: 5.23 and 5.76 ms). Widening the float weights in the kernel instead of converting them once
// took 9.95 ms.
constexpr uint32_t kReduceBlock = 128;
__global__ void k_weights64(const float* __restrict__ W, uint32_t n, double* __restrict__ W64) {
  const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d < n) W64[d] = (double)W[d];
}
__global__ void __launch_bounds__(kReduceBlock) k_reduce_bits_w64(const uint32_t* __restrict__ bits, uint32_t nc, uint32_t nWords,
                                                                  const float* __restrict__ N, const float* __restrict__ D,
                                                                  const double* __restrict__ W64, int useCos, double* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  const F3 n = ld3(N + 3 * size_t(i));
  double acc = 0;
  for (uint32_t w = 0; w < nWords; ++w) {
    uint32_t m = bits[size_t(w) * nc + i];
    while (m) {
      const uint32_t d = w * 32 + (__ffs(m) - 1);
      m &= m - 1;
      const float c = useCos ? fmaxf(dotf(n, ld3(D + 3 * d)), 0.f) : 1.f;
      if (c != 0.f) acc = __fma_rn(widen(c), __ldg(W64 + d), acc);
    }
  }
  out[i] = acc;
}
__global__ void __launch_bounds__(kReduceBlock) k_reduce_bytes_w64(const uint8_t* __restrict__ bytes, uint32_t nc, uint32_t nDir,
                                                                   const float* __restrict__ N, const float* __restrict__ D,
                                                                   const double* __restrict__ W64, int useCos, double* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  const F3 n = ld3(N + 3 * size_t(i));
  double acc = 0;
  constexpr uint32_t G = 16;   // 16 directions' bytes in flight before any is used, then added in direction order
  for (uint32_t d0 = 0; d0 < nDir; d0 += G) {
    uint32_t bb[G];
#pragma unroll
    for (uint32_t k = 0; k < G; ++k) bb[k] = d0 + k < nDir ? uint32_t(__ldg(bytes + size_t(d0 + k) * nc + i)) : 0u;
#pragma unroll
    for (uint32_t k = 0; k < G; ++k) {
      if (!bb[k]) continue;
      const uint32_t d = d0 + k;
      const float at = float(bb[k]) / 255.f;
      const float c = useCos ? fmaxf(dotf(n, ld3(D + 3 * d)), 0.f) : 1.f;
      const float x = c * at;
      if (x != 0.f) acc = __fma_rn(widen(x), __ldg(W64 + d), acc);
    }
  }
  out[i] = acc;
}

// The sums in integer arithmetic (ordered_sum.cuh: the same bits), for weights that are zero or positive normal floats; a
// direction's weight is (significand, biased exponent). Terms gives what a sensor's term of a direction is made from
// (raw), read ahead of its use, and its factor; where a factor is not a normal float (a normal of almost no length), the
// sensor's sum is done again with FP64 fmas.
__global__ void k_weight_parts(const float* __restrict__ W, uint32_t n, uint2* __restrict__ out) {
  const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= n) return;
  const uint32_t b = __float_as_uint(W[d]);
  out[d] = (b & 0x7fffffffu) ? make_uint2(os_sig(b), b >> 23) : make_uint2(0u, 1u);
}
__device__ __forceinline__ double part_weight(uint2 w) { return w.x ? (double)__uint_as_float((w.y << 23) | (w.x & 0x7fffffu)) : 0.0; }

template <bool COS>
struct BitsTerms {   // a visibility bit: the cosine, or 1
  const uint32_t* bits;
  uint32_t nc;
  const float *N, *D;
  using Raw = uint32_t;   // the word that holds the direction's bit
  __device__ __forceinline__ F3 sensor(uint32_t i) const { return COS ? ld3(N + 3 * size_t(i)) : f3(0.f, 0.f, 0.f); }
  __device__ __forceinline__ Raw raw(uint32_t d, uint32_t i) const { return __ldg(bits + size_t(d / 32) * nc + i); }
  __device__ __forceinline__ float factor(Raw m, uint32_t d, float c) const { return (m >> (d & 31u)) & 1u ? c : 0.f; }
};
template <bool COS>
struct BytesTerms {   // a transmittance byte: the cosine or 1 times b / 255
  const uint8_t* bytes;
  uint32_t nc;
  const float *N, *D;
  using Raw = uint32_t;
  __device__ __forceinline__ F3 sensor(uint32_t i) const { return COS ? ld3(N + 3 * size_t(i)) : f3(0.f, 0.f, 0.f); }
  __device__ __forceinline__ Raw raw(uint32_t d, uint32_t i) const { return __ldg(bytes + size_t(d) * nc + i); }
  __device__ __forceinline__ float factor(Raw b, uint32_t, float c) const { return b ? c * (float(b) / 255.f) : 0.f; }
};
struct DcTerms {   // a sky bin's reflected light
  const float* dc;
  uint32_t nc;
  const float* D;   // none
  using Raw = float;
  __device__ __forceinline__ F3 sensor(uint32_t) const { return f3(0.f, 0.f, 0.f); }
  __device__ __forceinline__ Raw raw(uint32_t d, uint32_t i) const { return __ldg(dc + size_t(d) * nc + i); }
  __device__ __forceinline__ float factor(Raw x, uint32_t, float) const { return x; }
};
template <bool COS> __device__ __forceinline__ float cosine(F3 n, F3 d) { return COS ? fmaxf(dotf(n, d), 0.f) : 1.f; }

__device__ __forceinline__ void term(float x, uint2 w, uint64_t& p, int32_t& e, bool& odd) {
  const uint32_t b = __float_as_uint(x);
  odd = odd || (x != 0.f && os_odd(b));
  p = x != 0.f ? uint64_t(os_sig(b)) * w.x : 0ull;
  e = int32_t((b >> 23) + w.y);
}
template <bool COS, class S>
__device__ __noinline__ double fp64_sum(const S& s, uint32_t n, const uint2* W, uint32_t i) {
  const F3 v = s.sensor(i);
  double acc = 0;
  for (uint32_t d = 0; d < n; ++d) {
    const float x = s.factor(s.raw(d, i), d, cosine<COS>(v, COS ? ld3(s.D + 3 * d) : F3{}));
    if (x != 0.f) acc = __fma_rn((double)x, part_weight(W[d]), acc);
  }
  return acc;
}

// A warp for a sensor, a lane per direction. While a sum's exponent stays, every term can be rounded by itself and the
// rounded terms added in any order: each lane rounds its own, and the warp adds them up. A term halfway between two
// values goes to the even one, which depends on the parity of the sum before it: the parity of the rounded terms since
// the last such term (which left an even sum) or since the 32 began. The term that starts the sum, one that lies above
// the sum's grid and one that takes the sum into the next binade are added alone, between those before and after.
__device__ __forceinline__ void add_32(OrderedSum& s, uint64_t p, int32_t e, uint32_t lane) {
  uint32_t todo = __ballot_sync(~0u, p != 0);
  const auto alone = [&](int from) {
    const uint64_t q = uint64_t(__shfl_sync(~0u, uint32_t(p), from)) | uint64_t(__shfl_sync(~0u, uint32_t(p >> 32), from)) << 32;
    os_add(s, q, __shfl_sync(~0u, e, from));
    todo &= ~1u << from;
  };
  while (todo) {
    if (!s.a) { alone(__ffs(todo) - 1); continue; }
    const int32_t sh = s.g - e;
    const uint32_t by = uint32_t(sh) < 63u ? uint32_t(sh) : 63u, below = (1u << lane) - 1u, above = __ballot_sync(~0u, sh < 0) & todo;
    const uint32_t now = above ? todo & ((above & (0u - above)) - 1u) : todo;   // the terms before the first one above the grid
    const bool mine = now >> lane & 1u;
    const uint64_t rem = (p << (63u - by)) << 1, half = 1ull << 63;
    uint64_t r = mine ? (p >> by) + (rem > half ? 1u : 0u) : 0ull;   // at most 2^48
    const uint32_t ties = __ballot_sync(~0u, mine && rem == half);
    if (ties) {
      const uint32_t odd = __ballot_sync(~0u, uint32_t(r) & 1u), last = ties & below;
      const uint32_t since = last ? below & (~1u << (31 - __clz(last))) : below;
      const uint32_t before = (__popc(odd & since) & 1u) ^ (last ? 0u : uint32_t(s.a) & 1u);
      if (ties >> lane & 1u) r += before ^ (uint32_t(r) & 1u);
    }
    const uint64_t a = s.a + __reduce_add_sync(~0u, uint32_t(r) & 0xffffffu) + (uint64_t(__reduce_add_sync(~0u, uint32_t(r >> 24))) << 24);
    if (!(a >> 53)) {
      s.a = a;
      todo &= ~now;
      if (above) alone(__ffs(above) - 1);
      continue;
    }
    uint64_t upTo = r;   // the sum of the terms up to and with the lane's
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t x = uint64_t(__shfl_up_sync(~0u, uint32_t(upTo), o)) | uint64_t(__shfl_up_sync(~0u, uint32_t(upTo >> 32), o)) << 32;
      if (lane >= uint32_t(o)) upTo += x;
    }
    const int past = __ffs(__ballot_sync(~0u, (s.a + upTo) >> 53)) - 1;
    const uint64_t less = upTo - r;
    s.a += uint64_t(__shfl_sync(~0u, uint32_t(less), past)) | uint64_t(__shfl_sync(~0u, uint32_t(less >> 32), past)) << 32;
    alone(past);   // and the terms before it are done
  }
}
// Four warps a block, and four words of directions read before any is added: a warp alone on its SM quarter is bound by the
// latency of its reads, many of them by issue, some 150 slots a word.
constexpr uint32_t kSumWarps = 4;
constexpr int kAhead = 4;
template <bool COS, class S>
__global__ void __launch_bounds__(32 * kSumWarps) k_sum_warp(S t, uint32_t n, const uint2* __restrict__ W, double* __restrict__ out) {
  const uint32_t i = blockIdx.x * kSumWarps + threadIdx.x / 32, lane = threadIdx.x & 31;
  if (i >= t.nc) return;   // whole warps
  const F3 v = t.sensor(i);
  OrderedSum s;
  bool odd = false;
  typename S::Raw raw[kAhead];
  F3 dir[kAhead];
  uint2 w[kAhead];
  const auto read = [&](uint32_t d0) {
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const uint32_t d = min(d0 + 32 * k + lane, n - 1);
      raw[k] = t.raw(d, i);
      if (COS) dir[k] = ld3(t.D + 3 * d);
      w[k] = __ldg(W + d);
    }
  };
  read(0);
  for (uint32_t d0 = 0; d0 < n; d0 += 32 * kAhead) {
    uint64_t p[kAhead];
    int32_t e[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const uint32_t d = d0 + 32 * k + lane;
      term(d < n ? t.factor(raw[k], d, cosine<COS>(v, dir[k])) : 0.f, w[k], p[k], e[k], odd);
    }
    if (d0 + 32 * kAhead < n) read(d0 + 32 * kAhead);   // under way while these are added
#pragma unroll
    for (int k = 0; k < kAhead; ++k) add_32(s, p[k], e[k], lane);
  }
  odd = __any_sync(~0u, odd);
  if (lane) return;
  out[i] = odd ? fp64_sum<COS>(t, n, W, i) : __longlong_as_double((long long)os_bits(s));
}

// The same sum by a block, for few sensors, where a warp a sensor leaves the SMs idle and a word takes it 0.4 us of
// dependent instructions: a word to each of kBlockWords warps at a time. Each warp rounds its terms on the grid of the
// sum so far and publishes their total; where no term lies above the grid and the totals keep the sum in its binade, the
// sum is that much larger. A warp's first halfway term depends on the sum's parity before the warp: its total is given
// for an even sum, with the difference for an odd one. Otherwise the totals before the first word that leaves the binade
// are added, that word's warp adds its terms as above, and the words after it are rounded again on the new grid. That is
// 2.5 us a word that leaves the binade, so it takes sums long enough that most words do not, and no more sensors than
// three or so an SM (a warp a sensor / 4 / 8 / 16 / 32 warps, us a call with the cosine): 16 sensors x 4746 directions
// 82 / 65 / 60 / 60 / 63, 300 x 5610 87 / 73 / 69 / 73 / 107, 600 x 5610 89 / 83 / 84 / 109 / 174, 1000 x 5610
// 97 / 104 / 119 / 151 / 262; 100 x 9066 bytes 124 / 90 / 77 / 76 / 83; 100 x 1290 49 / 50 / 48 / 49 / 55.
constexpr uint32_t kBlockWords = 8;
struct WordTotal {
  uint64_t even;    // the total, given an even sum before it
  int32_t odd;      // what an odd sum before it adds: 0, 1 or -1
  uint32_t flags;   // 1: the sum's parity after it (after its last halfway term, if any); 2: halfway terms; 4: adds alone
};
__device__ __forceinline__ WordTotal word_total(const OrderedSum& s, uint64_t p, int32_t e, uint32_t lane) {
  const int32_t sh = s.g - e;
  const uint32_t by = uint32_t(sh) < 63u ? uint32_t(sh) : 63u;
  const uint64_t rem = (p << (63u - by)) << 1, half = 1ull << 63;
  uint64_t r = (p >> by) + (rem > half ? 1u : 0u);
  WordTotal t{0, 0, 0};
  t.flags = __any_sync(~0u, p != 0 && (sh < 0 || !s.a)) ? 4u : 0u;
  const uint32_t ties = __ballot_sync(~0u, rem == half), odd = __ballot_sync(~0u, uint32_t(r) & 1u);
  uint32_t after = odd;
  if (ties) {
    const uint32_t below = (1u << lane) - 1u, last = ties & below;
    const uint32_t since = last ? below & (~1u << (31 - __clz(last))) : below;
    const uint32_t bump = (__popc(odd & since) & 1u) ^ (uint32_t(r) & 1u);
    if (ties >> lane & 1u) r += bump;
    t.odd = __shfl_sync(~0u, bump, __ffs(ties) - 1) ? -1 : 1;
    after = odd & (~1u << (31 - __clz(ties)));
    t.flags |= 2u;
  }
  t.flags |= __popc(after) & 1u;
  t.even = __reduce_add_sync(~0u, uint32_t(r) & 0xffffffu) + (uint64_t(__reduce_add_sync(~0u, uint32_t(r >> 24))) << 24);
  return t;
}
template <bool COS, class S>
__global__ void __launch_bounds__(32 * kBlockWords) k_sum_block(S t, uint32_t n, const uint2* __restrict__ W, double* __restrict__ out) {
  __shared__ WordTotal tot[2][kBlockWords];
  __shared__ OrderedSum left;
  const uint32_t i = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x / 32;
  const F3 v = t.sensor(i);
  OrderedSum s;
  bool odd = false;
  typename S::Raw raw;
  F3 dir{};
  uint2 w;
  const auto read = [&](uint32_t d0) {
    const uint32_t d = min(d0 + threadIdx.x, n - 1);
    raw = t.raw(d, i);
    if (COS) dir = ld3(t.D + 3 * d);
    w = __ldg(W + d);
  };
  read(0);
  uint32_t turn = 0;
  for (uint32_t d0 = 0; d0 < n; d0 += 32 * kBlockWords) {
    uint64_t p;
    int32_t e;
    const uint32_t d = d0 + threadIdx.x;
    term(d < n ? t.factor(raw, d, cosine<COS>(v, dir)) : 0.f, w, p, e, odd);
    if (d0 + 32 * kBlockWords < n) read(d0 + 32 * kBlockWords);   // under way while these are added
    for (uint32_t from = 0; from < kBlockWords;) {   // the words before it are added
      const WordTotal mine = word_total(s, p, e, lane);
      WordTotal* all = tot[turn++ & 1u];
      if (!lane) all[warp] = warp < from ? WordTotal{0, 0, 0} : mine;
      __syncthreads();
      const WordTotal x = lane < kBlockWords ? all[lane] : WordTotal{0, 0, 0};
      uint64_t r = x.even;
      const uint32_t ties = __ballot_sync(~0u, x.flags & 2u);
      if (ties) {
        const uint32_t parity = __ballot_sync(~0u, x.flags & 1u), below = (1u << lane) - 1u, last = ties & below;
        const uint32_t since = last ? below & (~0u << (31 - __clz(last))) : below;
        if ((__popc(parity & since) & 1u) ^ (last ? 0u : uint32_t(s.a) & 1u)) r += int64_t(x.odd);
      }
      const uint32_t alone = __ballot_sync(~0u, x.flags & 4u);
      const uint64_t a = s.a + __reduce_add_sync(~0u, uint32_t(r) & 0x7ffffffu) + (uint64_t(__reduce_add_sync(~0u, uint32_t(r >> 27))) << 27);
      if (!alone && !(a >> 53)) { s.a = a; break; }
      uint64_t upTo = r;   // the totals up to and with the lane's word
#pragma unroll
      for (int o = 1; o < int(kBlockWords); o <<= 1) {
        const uint64_t y = uint64_t(__shfl_up_sync(~0u, uint32_t(upTo), o)) | uint64_t(__shfl_up_sync(~0u, uint32_t(upTo >> 32), o)) << 32;
        if (lane >= uint32_t(o)) upTo += y;
      }
      const uint32_t at = __ffs(alone | __ballot_sync(~0u, (s.a + upTo) >> 53)) - 1;
      const uint64_t less = upTo - r;
      s.a += uint64_t(__shfl_sync(~0u, uint32_t(less), at)) | uint64_t(__shfl_sync(~0u, uint32_t(less >> 32), at)) << 32;
      if (warp == at) {
        add_32(s, p, e, lane);
        if (!lane) left = s;
      }
      __syncthreads();
      s = left;
      from = at + 1;
    }
  }
  if (__syncthreads_or(odd)) {
    if (!threadIdx.x) out[i] = fp64_sum<COS>(t, n, W, i);
  } else if (!threadIdx.x) out[i] = __longlong_as_double((long long)os_bits(s));
}

static uint32_t blocks_of(uint32_t n) { return (n + kReduceBlock - 1) / kReduceBlock; }
constexpr uint32_t kBlockSensors = 450, kBlockDirs = 2048;
template <bool COS, class S>
static void launch_sum_warp(const S& t, uint32_t n, const float* W, double* w64, double* out, cudaStream_t st) {
  uint2* parts = reinterpret_cast<uint2*>(w64);
  k_weight_parts<<<(n + 255) / 256, 256, 0, st>>>(W, n, parts);
  if (t.nc <= kBlockSensors && n >= kBlockDirs) k_sum_block<COS><<<t.nc, 32 * kBlockWords, 0, st>>>(t, n, parts, out);
  else k_sum_warp<COS><<<(t.nc + kSumWarps - 1) / kSumWarps, 32 * kSumWarps, 0, st>>>(t, n, parts, out);
}
// Which form is faster (152 SMs): the thread form waits so many ns a direction for its fma and its reads, whatever the
// sensors, until they fill the SMs (bits of a city's facades, which see little of the sky, 42 and with the cosine 74, of a
// block's 60 and 98; bytes 95 and 112, 119 and 157, a quarter more once they exceed the L2), and 6 us before; the warp form
// costs a sensor 0.106 ns for each word of 32 directions and for fifty words' worth more at the start of its sum, where
// nearly every term doubles it. The rates are about the mean of city's and block's ns over these 0.106 ns, so that near the line
// neither scene loses more than it would gain. us a call, thread / warp, city and block: bits with the cosine 8000 x 1000
// 91 / 88, 123 / 89; 12,345 x 2155 163 / 178, 234 / 174; 20,000 x 5033 362 / 457, 496 / 453; without 5000 x 1000 71 / 73,
// 91 / 70; 8000 x 2155 110 / 125, 151 / 125; 12,345 x 5033 226 / 275, 309 / 269; bytes with the cosine 20,000 x 2155 263 / 264,
// 328 / 269; 25,000 x 2155 249 / 316, 337 / 325; 29,000 x 9066 1254 / 1064, 1507 / 1050; without 16,000 x 2155 223 / 219,
// 285 / 215; 20,000 x 2155 219 / 252, 266 / 254.
// Under 256 directions the start of the sum is most of it (16 sensors x 15 directions: 5 us against 14).
static bool warp_sums(uint32_t nc, uint32_t n, uint64_t rate) { return n >= 256 && uint64_t(nc) * (50 + n / 32) <= rate * (n + 80); }
constexpr uint64_t kL2Bytes = 96000000;   // from here on the L2 (129 MB) no longer holds them: 16,000 x 5033 119 ns a direction, 20,000 x 5033 135

void launch_reduce_bits(const uint32_t* bits, uint32_t nc, uint32_t nWords, uint32_t nDir, const float* N, const float* D, const float* W,
                        int useCos, double* out, cudaStream_t st, double* w64, bool plain) {
  if (w64 && plain && warp_sums(nc, nDir, useCos ? 780 : 475)) {
    if (useCos) launch_sum_warp<true>(BitsTerms<true>{bits, nc, N, D}, nDir, W, w64, out, st);
    else launch_sum_warp<false>(BitsTerms<false>{bits, nc, N, D}, nDir, W, w64, out, st);
  } else if (w64) {
    k_weights64<<<(nDir + 255) / 256, 256, 0, st>>>(W, nDir, w64);
    k_reduce_bits_w64<<<blocks_of(nc), kReduceBlock, 0, st>>>(bits, nc, nWords, N, D, w64, useCos, out);
  } else if (nDir <= kReduceSmemDirs && reduce_smem_ready())
    k_reduce_bits<true><<<(nc + 255) / 256, 256, nDir * sizeof(double), st>>>(bits, nc, nWords, nDir, N, D, W, useCos, out);
  else k_reduce_bits<false><<<(nc + 255) / 256, 256, 0, st>>>(bits, nc, nWords, nDir, N, D, W, useCos, out);
}
void launch_reduce_bytes(const uint8_t* bytes, uint32_t nc, uint32_t nDir, const float* N, const float* D, const float* W, int useCos,
                         double* out, cudaStream_t st, double* w64, bool plain) {
  if (w64 && plain && warp_sums(nc, nDir, (useCos ? 1190 : 1000) * (uint64_t(nc) * nDir > kL2Bytes ? 5 : 4) / 4)) {
    if (useCos) launch_sum_warp<true>(BytesTerms<true>{bytes, nc, N, D}, nDir, W, w64, out, st);
    else launch_sum_warp<false>(BytesTerms<false>{bytes, nc, N, D}, nDir, W, w64, out, st);
  } else if (w64) {
    k_weights64<<<(nDir + 255) / 256, 256, 0, st>>>(W, nDir, w64);
    k_reduce_bytes_w64<<<blocks_of(nc), kReduceBlock, 0, st>>>(bytes, nc, nDir, N, D, w64, useCos, out);
  } else if (nDir <= kReduceSmemDirs && reduce_smem_ready())
    k_reduce_bytes<true><<<(nc + 255) / 256, 256, nDir * sizeof(double), st>>>(bytes, nc, nDir, N, D, W, useCos, out);
  else k_reduce_bytes<false><<<(nc + 255) / 256, 256, 0, st>>>(bytes, nc, nDir, N, D, W, useCos, out);
}
// sky bins: the warp form at every size (2306 bins, both forms, us a call: 500 sensors 673 / 48, 20,011 712 / 156,
// 80,000 2005 / 868: two conversions and two FP64 operations a term against a rounded product)
void launch_reduce_dc(const float* dc, uint32_t nc, uint32_t nBins, const float* W, double* out, cudaStream_t st, double* w64, bool plain) {
  if (plain) launch_sum_warp<false>(DcTerms{dc, nc, nullptr}, nBins, W, w64, out, st);
  else k_reduce_dc<<<(nc + 255) / 256, 256, 0, st>>>(dc, nc, nBins, W, out);
}
void launch_reduce_view(const ViewReduceArgs& a, cudaStream_t st) {
  // shared memory: per warp 2 C + R doubles and C floats per lane (at most 19 classes and 8 reach distances: 111 KB)
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(k_view_reduce, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         int(kViewWarps * 32 * ((2 * KGB_VIEW_CLASSES + 8) * 8 + KGB_VIEW_CLASSES * 4)));
    attr = true;
  }
  const size_t smem = size_t(kViewWarps) * 32 * ((2 * a.nClass + a.nReach) * 8 + a.nClass * 4);
  k_view_reduce<<<(a.nc + kViewWarps - 1) / kViewWarps, kViewWarps * 32, smem, st>>>(a);
  if (a.isoDim) k_iso<<<(a.nc + 7) / 8, 256, 0, st>>>(a);
}

}  // namespace kgb
