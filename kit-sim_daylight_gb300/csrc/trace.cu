// Ray-casting kernels of the engine (compiled with -fmad=false: see rt.cuh):
//  k_bits   visibility bits, any-hit (replaces the reference's __raygen__bits, trace_dev.cu:91-108)
//  k_bytes  transmittance bytes (replaces __raygen__bytes + __anyhit__tr, trace_dev.cu:115-165)
//  k_view   class + distance of the closest hit per view cell (replaces __raygen__view, trace_dev.cu:177-232)
//  k_bounce_paths, k_bounce_rest, k_bounce_accum, k_bounce_accum_few
//           reflected-light paths binned by sky patch (replaces __raygen__bounce, trace_dev.cu:260-311): first
//           segments, then the paths that go on from a queue, to their ends
// The visibility kernels are persistent: each warp takes tasks of 32 consecutive sensors x up to 32 directions from a
// global counter, so a warp traces one direction for 32 neighbouring sensors at a time (coherent rays; k_view: two cells
// for 16). k_bits and k_bytes take a call's sensors in the engine's tracing order (grouped by the orientation of their normals:
// TraceArgs::order), so that a warp's sensors face the same way more often; each result goes to its sensor's column.
#include "engine.h"
#include "rt.cuh"

#include <algorithm>

namespace kgb {

// The sensor (scene index) at lane position i of a launch and its output column (see TraceArgs::order).
__device__ __forceinline__ void task_sensor(const TraceArgs& a, uint32_t i, uint32_t& gi, uint32_t& col) {
  if (!a.order) { gi = a.first + i; col = a.out0 + i; return; }
  const uint32_t p = a.p0 + i;
  uint32_t g = a.pieceG[0];   // the runs' ends do not decrease: the last one passed names the run
  if (p >= a.pieceEnd[0]) g = a.pieceG[1];
  if (p >= a.pieceEnd[1]) g = a.pieceG[2];
  if (p >= a.pieceEnd[2]) g = a.pieceG[3];
  if (p >= a.pieceEnd[3]) g = a.pieceG[4];
  if (p >= a.pieceEnd[4]) g = a.pieceG[5];
  gi = a.order[g + p];
  col = gi - a.callI0;
}

__device__ __forceinline__ uint32_t next_task(uint32_t* counter) {
  uint32_t t = 0;
  if ((threadIdx.x & 31) == 0) t = atomicAdd(counter, 1u);
  return __shfl_sync(~0u, t, 0);
}

// ---------------------------------------------------------------------------------------------------- bits
// Direction d of a sensor is visible when n.d > 0 and every hit from tmin 1e-5 on is an own-plane hit, at most 3.
// A task is 32 sensors x PER directions of a word (32, 16 or 8: task_directions; a template, since the whole word's form
// keeps 80 registers without spills and the general one did not: 2 % of the urban trace); the parts of the last word past
// the last direction are no tasks (199,000 sensors x 14 directions 208 to 201 us). FRONT: the walks start from the
// 32 sensors' frontier (a.frontiers, by position in the launch), which k_frontiers made.
// COUNT: the instrumented variant (same results) that adds up nodes visited, triangles tested and rays traced.
template <bool COUNT, uint32_t PER, bool FRONT>
__global__ void __launch_bounds__(256) k_bits(TraceArgs a) {
  __shared__ Frontier frontier[FRONT ? 8 : 1];
  const Scene s{a.nodes, a.tris, a.nNodes};
  const bool cull = (a.rayFlags & KGB_RAY_CULL_BACK_FACING) != 0;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t cols = (a.nDir + PER - 1) / PER, nTasks = (a.n + 31) / 32 * cols;
  uint32_t overflow = 0;
  Count ctr;
  uint32_t rays = 0;
  for (uint32_t task = next_task(a.counter); task < nTasks; task = next_task(a.counter)) {
    const uint32_t i = task / cols * 32 + lane, d0 = task % cols * PER;
    const bool valid = i < a.n;
    uint32_t gi = 0, col = 0, word = 0;
    F3 n = f3(0.f, 0.f, 0.f), o = n;
    if (valid) {
      task_sensor(a, i, gi, col);
      n = ld3(a.N + 3 * gi);
      o = offset_ray(ld3(a.P + 3 * gi), n);
    }
    if (FRONT) {
      const FrontierRec* rec = a.frontiers + task / cols;
      Frontier& f = frontier[threadIdx.x / 32];
      load_frontier(rec, f, lane);
      const Bounds b = rec->b;
      word = trace_word<COUNT>(s, f, rec->n, b, n, o, valid, a.rayTab, d0, min(d0 + PER, a.nDir), cull, overflow, ctr, rays);
      __syncwarp();   // the frontier is the next task's
    } else if (valid) {
      word = trace_word<COUNT>(s, n, o, a.D, a.rayTab, d0, min(d0 + PER, a.nDir), cull, overflow, ctr, rays);
    }
    if (!valid) continue;
    const uint32_t e0 = task % cols * PER;   // d0 again: not kept through the walks
    uint32_t* out = a.bits + size_t(e0 / 32) * a.stride + col;
    const uint32_t at = e0 % 32;
    if (PER == 32) *out = word;
    else if (PER == 16) {
      reinterpret_cast<uint16_t*>(out)[at / 16] = uint16_t(word >> at);
      if (!at && e0 + 16 >= a.nDir) reinterpret_cast<uint16_t*>(out)[1] = 0;   // no task for the word's second half
    } else {
      reinterpret_cast<uint8_t*>(out)[at / 8] = uint8_t(word >> at);
      if (e0 + 8 >= a.nDir) for (uint32_t k = at / 8 + 1; k < 4; ++k) reinterpret_cast<uint8_t*>(out)[k] = 0;   // no tasks for these
    }
  }
  if (overflow) atomicOr(a.status, (overflow & 1u ? kStatusStackOverflow : 0u) | (overflow & 2u ? kStatusVisitLimit : 0u));
  if (COUNT) {
    unsigned long long* c = reinterpret_cast<unsigned long long*>(a.status + 1);   // ctl words 2..7: three u64 counters
    atomicAdd(c, (unsigned long long)ctr.nodes);
    atomicAdd(c + 1, (unsigned long long)ctr.tris);
    atomicAdd(c + 2, (unsigned long long)rays);
  }
}
// A launch's frontiers: a warp per 32 sensors.
constexpr uint32_t kFrontierWarps = 4;
__global__ void __launch_bounds__(32 * kFrontierWarps) k_frontiers(TraceArgs a) {
  __shared__ Frontier frontier[kFrontierWarps];
  const Scene s{a.nodes, a.tris, a.nNodes};
  const uint32_t lane = threadIdx.x & 31, block = blockIdx.x * kFrontierWarps + threadIdx.x / 32, i = block * 32 + lane;
  if (block * 32 >= a.n) return;   // whole warps
  F3 o = f3(0.f, 0.f, 0.f);
  if (i < a.n) {
    uint32_t gi, col;
    task_sensor(a, i, gi, col);
    o = offset_ray(ld3(a.P + 3 * gi), ld3(a.N + 3 * gi));
  }
  Frontier& f = frontier[threadIdx.x / 32];
  const Bounds b = origin_bounds(o, i < a.n);
  const uint32_t n = build_frontier(s, b, f, lane);
  store_frontier(a.frontiers + block, f, b, n, lane);
}
// A call of few words: a block per 32 sensors x a word, each of its 16 warps two of the directions. Where even tasks of 8
// directions would not give every resident warp one, the call lasts as long as one task: 16 sensors x 4746 directions
// 48 to 10 us, 16 x 15 22 to 8 us.
constexpr uint32_t kFewWarps = 16;
__global__ void __launch_bounds__(32 * kFewWarps) k_bits_few(TraceArgs a) {
  __shared__ uint32_t words[32];
  const Scene s{a.nodes, a.tris, a.nNodes};
  const bool cull = (a.rayFlags & KGB_RAY_CULL_BACK_FACING) != 0;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x / 32, b = blockIdx.x / a.nWords, w = blockIdx.x % a.nWords, i = b * 32 + lane;
  uint32_t overflow = 0, rays = 0, gi = 0, col = 0;
  Count ctr;
  if (warp == 0) words[lane] = 0;
  __syncthreads();
  if (i < a.n) {
    task_sensor(a, i, gi, col);
    const F3 n = ld3(a.N + 3 * gi), o = offset_ray(ld3(a.P + 3 * gi), n);
    uint32_t word = 0;
    for (uint32_t d = w * 32 + warp; d < min(w * 32 + 32, a.nDir); d += kFewWarps)
      word |= trace_word<false>(s, n, o, a.D, a.rayTab, d, d + 1, cull, overflow, ctr, rays);
    if (word) atomicOr(&words[lane], word);
  }
  __syncthreads();
  if (warp == 0 && i < a.n) a.bits[size_t(w) * a.stride + col] = words[lane];
  if (overflow) atomicOr(a.status, (overflow & 1u ? kStatusStackOverflow : 0u) | (overflow & 2u ? kStatusVisitLimit : 0u));
}

// ---------------------------------------------------------------------------------------------------- bytes
// A translucent slot's crossing: tau, 1 on a thin solid's exit face, Radiance glass T(cos) (trace_dev.cu:147-165).
__device__ __forceinline__ float crossing(const kgb_slot* slots, const float2* slotLog, uint32_t nSlots, uint32_t slot, bool front, F3 v0, F3 v1,
                                         F3 v2, F3 d) {
  const kgb_slot sl = slot < nSlots ? slots[slot] : kgb_slot{0.2f, 0.f, 0.f, 0u};
  float T = sl.tau;
  if ((sl.flags & KGB_SLOT_THIN) && front == ((sl.flags & KGB_SLOT_INWARD) != 0)) T = 1.f;
  else if (sl.flags & KGB_SLOT_GLASS) {
    const float ax = v1.x - v0.x, ay = v1.y - v0.y, az = v1.z - v0.z;
    const float bx = v2.x - v0.x, by = v2.y - v0.y, bz = v2.z - v0.z;
    const float nx = ay * bz - az * by, ny = az * bx - ax * bz, nz = ax * by - ay * bx;
    float R;
    glass_TR(fabsf(nx * d.x + ny * d.y + nz * d.z) * (1.f / sqrtf(nx * nx + ny * ny + nz * nz)), sl.tn, slotLog[slot], T, R);
  }
  return T;
}

constexpr int kMaxCross = 16;   // translucent crossings a ray keeps in registers before it walks them in order instead

// Own-plane hits pass (at most 3), an opaque hit blocks, translucent crossings multiply in (t, primitive) order.
// hits(f): calls f for every hit of the ray (origin's normal n, direction dir).
template <class Hits>
__device__ __forceinline__ uint8_t trace_byte(const TraceArgs& a, F3 n, F3 dir, Hits&& hits) {
  bool blocked = false, spill = false;
  int own = 0, nx = 0;
  float ct[kMaxCross], cf[kMaxCross];
  uint32_t cp[kMaxCross];
  hits([&](const Hit& h, F3 v0, F3 v1, F3 v2, uint32_t flags, uint32_t slot) {
    if (own_hit(v0, v1, v2, h, dir, n)) { if (++own <= 3) return false; blocked = true; return true; }
    if (!(flags & kTriTranslucent)) { blocked = true; return true; }
    if (nx < kMaxCross) { ct[nx] = h.t; cp[nx] = h.prim; cf[nx] = crossing(a.slots, a.slotLog, a.nSlots, slot, h.front, v0, v1, v2, dir); ++nx; }
    else spill = true;
    return false;
  });
  if (blocked) return 0;
  float T = 1.f;
  if (!spill) {
    for (int x = 1; x < nx; ++x) {   // insertion sort by (t, primitive)
      const float tx = ct[x], fx = cf[x];
      const uint32_t px = cp[x];
      int y = x - 1;
      while (y >= 0 && (ct[y] > tx || (ct[y] == tx && cp[y] > px))) { ct[y + 1] = ct[y]; cp[y + 1] = cp[y]; cf[y + 1] = cf[y]; --y; }
      ct[y + 1] = tx; cp[y + 1] = px; cf[y + 1] = fx;
    }
    for (int x = 0; x < nx; ++x) {
      T *= cf[x];
      if (!(T >= 1.f / 510.f)) return 0;
    }
    return (uint8_t)__float2uint_rn(T * 255.f);
  }
  // more than kMaxCross crossings: walk them one at a time in (t, primitive) order
  float lastT = -INFINITY;
  uint32_t lastP = 0;
  for (;;) {
    bool found = false;
    float bt = 0.f, bf = 0.f;
    uint32_t bp = 0;
    hits([&](const Hit& h, F3 v0, F3 v1, F3 v2, uint32_t flags, uint32_t slot) {
      if (!(flags & kTriTranslucent) || own_hit(v0, v1, v2, h, dir, n)) return false;
      if (h.t < lastT || (h.t == lastT && h.prim <= lastP)) return false;
      if (!found || h.t < bt || (h.t == bt && h.prim < bp)) {
        found = true; bt = h.t; bp = h.prim;
        bf = crossing(a.slots, a.slotLog, a.nSlots, slot, h.front, v0, v1, v2, dir);
      }
      return false;
    });
    if (!found) break;
    T *= bf;
    if (!(T >= 1.f / 510.f)) return 0;
    lastT = bt; lastP = bp;
  }
  return (uint8_t)__float2uint_rn(T * 255.f);
}

// FRONT: as k_bits.
template <bool FRONT>
__global__ void __launch_bounds__(256, 3) k_bytes(TraceArgs a) {   // 3 blocks an SM: 21.3 ms for a precision chunk, 24.6 at 2 (no spills)
  __shared__ Frontier frontier[FRONT ? 8 : 1];
  const Scene s{a.nodes, a.tris, a.nNodes};
  const bool cull = (a.rayFlags & KGB_RAY_CULL_BACK_FACING) != 0;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t cols = (a.nDir + a.per - 1) / a.per, nTasks = (a.n + 31) / 32 * cols;
  uint32_t overflow = 0;
  for (uint32_t task = next_task(a.counter); task < nTasks; task = next_task(a.counter)) {
    const uint32_t b = task / cols, d0 = task % cols * a.per, i = b * 32 + lane, dEnd = min(d0 + a.per, a.nDir);
    const bool valid = i < a.n;
    if (!FRONT && !valid) continue;
    uint32_t gi = 0, col = 0;
    F3 n = f3(0.f, 0.f, 0.f), o = n;
    if (valid) {
      task_sensor(a, i, gi, col);
      n = ld3(a.N + 3 * gi);
      o = offset_ray(ld3(a.P + 3 * gi), n);
    }
    Frontier& f = frontier[FRONT ? threadIdx.x / 32 : 0];
    uint32_t entries = 0;
    Bounds bounds;
    if (FRONT) {
      const FrontierRec* rec = a.frontiers + b;
      load_frontier(rec, f, lane);
      bounds = rec->b;
      entries = rec->n;
    }
    for (uint32_t d = d0; d < dEnd; ++d) {
      const Ray r = ray_from(a.rayTab, d, o);
      const bool on = n.x * r.d.x + n.y * r.d.y + n.z * r.d.z > 0.f;   // never for a lane without a sensor
      uint8_t out = 0;
      if (FRONT) {
        if (__any_sync(~0u, on)) {
          const Mask64 m = shaft(f, entries, bounds, r, lane);
          if (on)
            out = trace_byte(a, n, r.d, [&](auto&& hit) { frontier_hits<false, true>(s, f, m, r, 1e-5f, INFINITY, cull, hit, overflow, nullptr); });
        }
      } else if (on) {
        out = trace_byte(a, n, r.d, [&](auto&& hit) { for_hits<false, true>(s, r, 1e-5f, INFINITY, cull, hit, overflow); });
      }
      if (valid) a.bytes[size_t(d) * a.stride + col] = out;
    }
    if (FRONT) __syncwarp();   // the frontier is the next task's
  }
  if (overflow) atomicOr(a.status, (overflow & 1u ? kStatusStackOverflow : 0u) | (overflow & 2u ? kStatusVisitLimit : 0u));
}

// ---------------------------------------------------------------------------------------------------- views
// params.h:77-89 (view_cell), sincospif as kgb_sincospi
__device__ __forceinline__ F3 view_cell(uint32_t d, uint32_t col, float rsx, float rsy, float az0, float dAz, bool jitter, uint32_t element, uint32_t side) {
  float a = 0.5f, s = 0.5f * (rsx + rsy);
  if (jitter) { const U3 h = pcg3d(element, d, side); a = u01(h.x); s = rsx + u01(h.y) * (rsy - rsx); }
  float sa, ca;
  kgb_sincospi((az0 + (float(col) + a) * dAz) * (1.f / 180.f), &sa, &ca);
  const float c = sqrtf(fmaxf(0.f, 1.f - s * s));
  return f3(c * sa, c * ca, s);
}

// The reported distance of the hit that ended a view ray. The watertight test's t = T / det rounds with the vertices'
// coordinates relative to the origin, so a triangle whose vertices lie far beyond the hit (a kilometre-long ground quad
// seen from 100 m) gives t off by up to 1e-3 relative. Where a vertex lies more than 4 t from the origin along an axis
// (in float), t is recomputed from the triangle's plane in double, float(dot(v0 - o, ng)) / float(dot(d, ng)) with
// ng = (v1 - v0) x (v2 - v0): the differences and products of float coordinates are exact or within 2^-52 in double,
// so the result lies within 2 ulps of the exact distance. About 9 % of the views city's hits take this path, and every
// distance then lies within 3.2e-6 of a double-precision walk's. The walk (which hits, their order, the own-plane
// rules) keeps the float t; the oracle's view_ray applies the same rule with the same operations.
__device__ __noinline__ float refine_t(F3 o, F3 d, F3 v0, F3 v1, F3 v2, float t) {
  const float reach = fmaxf(fmaxf(fmaxf(fabsf(v0.x - o.x), fabsf(v0.y - o.y)), fmaxf(fabsf(v0.z - o.z), fabsf(v1.x - o.x))),
                            fmaxf(fmaxf(fmaxf(fabsf(v1.y - o.y), fabsf(v1.z - o.z)), fmaxf(fabsf(v2.x - o.x), fabsf(v2.y - o.y))), fabsf(v2.z - o.z)));
  if (!(reach > 4.f * t)) return t;
  const double ex = double(v1.x) - double(v0.x), ey = double(v1.y) - double(v0.y), ez = double(v1.z) - double(v0.z);
  const double fx = double(v2.x) - double(v0.x), fy = double(v2.y) - double(v0.y), fz = double(v2.z) - double(v0.z);
  const double nx = ey * fz - ez * fy, ny = ez * fx - ex * fz, nz = ex * fy - ey * fx;
  const double num = ((double(v0.x) - double(o.x)) * nx + (double(v0.y) - double(o.y)) * ny) + (double(v0.z) - double(o.z)) * nz;
  const double den = (double(d.x) * nx + double(d.y) * ny) + double(d.z) * nz;
  const float r = __fdiv_rn(__double2float_rn(num), __double2float_rn(den));
  return r > 0.f && r < __int_as_float(0x7f800000) ? r : t;
}

// A warp traces kViewSensors neighbouring sensors x two neighbouring cells at a time: the walk is a warp's, and half the
// stretch of facade with cells a few degrees apart diverges less than 32 sensors in one direction. us a call, 32 x 1 / 16 x
// 2: 12,000 sensors, 120 degrees, cells of 2 / 5 / 10 degrees 8865 / 7983, 1532 / 1403, 461 / 430; 25,000 all around in 2 M
// triangles 37,565 / 32,763; 400 at 1 degree 1356 / 1178. 8 x 4 cells was 18 % slower than 32 x 1 (120 degrees, cells of 2).
constexpr uint32_t kViewSensors = 16;
__global__ void __launch_bounds__(256, 3) k_view(ViewArgs a) {   // 3 blocks an SM: more warps to hide latency beat the few spills
  const Scene s{a.nodes, a.tris, a.nNodes};
  const bool cull = (a.rayFlags & KGB_RAY_CULL_BACK_FACING) != 0;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t cols = (a.K + a.per - 1) / a.per, nTasks = (a.n + kViewSensors - 1) / kViewSensors * cols;
  const float inf = __int_as_float(0x7f800000);
  uint32_t overflow = 0;
  for (uint32_t task = next_task(a.counter); task < nTasks; task = next_task(a.counter)) {
    const uint32_t b = task / cols, d0 = task % cols * a.per, i = b * kViewSensors + lane % kViewSensors;
    if (i >= a.n) continue;
    const uint32_t gl = a.first + i;           // sensor within the engine's arrays
    const uint32_t gi = a.i0 + a.out0 + i;     // global sensor index (seeds)
    const uint32_t element = gi / a.nS, side = a.nS == 2 ? gi % 2 : a.back;
    const F3 n = ld3(a.N + 3 * gl), o = offset_ray(ld3(a.P + 3 * gl), n);
    const bool none = !(dot(n, n) > 0.f);
    F3 f, r, u;
    if (a.world) { f = f3(-a.sinN, a.cosN, 0.f); r = f3(a.cosN, a.sinN, 0.f); u = f3(0.f, 0.f, 1.f); }
    else {
      const float l = sqrtf(n.x * n.x + n.y * n.y);
      f = n;
      if (l > 1e-3f) r = f3(n.y / l, -n.x / l, 0.f);
      else {
        r = f3(a.cosN, a.sinN, 0.f);
        if (l > 0.f) { r = sub(r, mul(dot(r, n), n)); r = mul(1.f / sqrtf(dot(r, r)), r); }
      }
      u = f3(r.y * f.z - r.z * f.y, r.z * f.x - r.x * f.z, r.x * f.y - r.y * f.x);
    }
    for (uint32_t d = d0 + lane / kViewSensors; d < d0 + a.per; d += 32 / kViewSensors) {
      if (d >= a.K) break;
      const uint32_t col = d % a.nAz, row = d / a.nAz;
      const F3 l = view_cell(d, col, a.rowSin[2 * row], a.rowSin[2 * row + 1], a.az0, a.dAz, a.jitter != 0, element, side);
      const F3 dir = add(add(mul(l.x, r), mul(l.y, f)), mul(l.z, u));
      uint32_t cl = 2;
      float t = inf;
      if (none || (a.cull && dot(n, dir) <= 0.f)) cl = 254;
      else if (a.vground && dir.z < 0.f && !(o.z > a.groundZ)) { cl = 1; t = 0.1f; }
      else {
        const bool plane = a.vground && dir.z < 0.f;
        const float tg = plane ? (o.z - a.groundZ) / -dir.z : inf;
        const float tmax = plane ? (o.z - a.groundZ + 0.01f) / -dir.z : FLT_MAX;
        float tmin = 1e-5f;
        uint32_t own = 0, panes = 0;
        const Ray ray = make_ray(o, dir);
        ClosestOut c;
        bool byHit = false;   // the walk ended on a hit (not past the last one)
        for (;;) {
          if (!closest(s, ray, tmin, tmax, cull, c, overflow)) { cl = dir.z >= 0.f ? 0 : 1; t = tg; break; }
          t = c.h.t;
          if (own_hit(c.v0, c.v1, c.v2, c.h, dir, n)) { if (++own == 4) { byHit = true; break; } }
          else {
            const uint32_t lb = a.label ? a.label[c.h.prim] : 2u;
            if (lb != KGB_LABEL_PASS) { cl = lb; byHit = true; break; }
            if (++panes > KGB_MAX_PANES) { byHit = true; break; }
          }
          tmin = next_up(t);
        }
        if (byHit) t = refine_t(o, dir, c.v0, c.v1, c.v2, t);
        if (panes) cl |= KGB_VIEW_GLAZED;
      }
      const size_t at = size_t(d) * a.stride + a.out0 + i;
      a.cls[at] = uint8_t(cl);
      a.dist[at] = t;
    }
  }
  if (overflow) atomicOr(a.status, (overflow & 1u ? kStatusStackOverflow : 0u) | (overflow & 2u ? kStatusVisitLimit : 0u));
}

// ---------------------------------------------------------------------------------------------------- bounce
__device__ __forceinline__ F3 cosine_dir(F3 n, float u, float v) {   // trace_dev.cu:235-242 (Duff et al. 2017 basis)
  const float sg = copysignf(1.f, n.z), a = -1.f / (sg + n.z), b = n.x * n.y * a;
  const F3 t = f3(1.f + sg * n.x * n.x * a, sg * b, -sg * n.x), w = f3(b, sg + n.y * n.y * a, -n.y);
  float s, c;
  kgb_sincospi(2.f * v, &s, &c);
  const float r = sqrtf(u);
  return add(add(mul(r * c, t), mul(r * s, w)), mul(sqrtf(fmaxf(0.f, 1.f - u)), n));
}
__constant__ uint32_t kTnaz[7] = {30, 30, 24, 24, 18, 12, 6};
__device__ __forceinline__ uint32_t sky_bin(F3 d, uint32_t mf, uint32_t nBins, float alpha, float cosN, float sinN) {   // trace_dev.cu:248-258
  if (!(d.z >= 0.f)) return 0;
  const uint32_t r = min(uint32_t(kgb_asin(fminf(d.z, 1.f)) / alpha), 7 * mf);
  if (r == 7 * mf) return nBins - 1;
  const uint32_t n = kTnaz[r / mf] * mf;
  uint32_t b = 1 + (r % mf) * n;
  for (uint32_t q = 0; q < r / mf; ++q) b += kTnaz[q] * mf * mf;
  float az = kgb_atan2(d.x * cosN + d.y * sinN, d.y * cosN - d.x * sinN);
  if (az < 0.f) az += 6.28318531f;
  return b + uint32_t(az * (float(n) / 6.28318531f) + .5f) % n;
}

constexpr uint32_t kNoBin = 0xffffffffu;

// A path between segments (48 bytes): where it is, where it goes, its weight and counters.
struct __align__(16) PathState {
  float ox, oy, oz;
  uint32_t gi;       // global sensor index
  float dx, dy, dz;
  uint32_t smp;      // sample
  float w;
  uint32_t k;        // random-number counter
  uint32_t bits;     // diffuse reflections (bits 0-7), reflected (bit 8), segments done (bits 16-31)
  uint32_t at;       // its result's index: contrib[(sample - s0) n + i]
};

// One segment of a path: the body of the reference's per-sample loop (trace_dev.cu:260-311). Returns true when the path
// goes on (o, d, w, k, diffuse, reflected updated), false when it has ended (bin and gain set if it escaped after a
// reflection). nn: the sensor's normal, read on the first segment only.
__device__ __forceinline__ bool bounce_segment(const BounceArgs& a, const Scene& s, bool cull, uint32_t seg, F3 nn, uint32_t gi, uint32_t smp, F3& o,
                                               F3& d, float& w, uint32_t& k, uint32_t& diffuse, bool& reflected, uint32_t& bin, float& gain,
                                               uint32_t& overflow) {
  ClosestOut c;
  const bool found = closest<true>(s, make_ray(o, d), 1e-5f, FLT_MAX, cull, c, overflow);
  if (overflow & 2u) {   // the walk gave up: the first such path leaves its ray for the error message
    uint32_t* diag = a.status + 15;   // ctl words 16..
    if (atomicCAS(diag, 0u, 1u) == 0u) {
      diag[1] = gi; diag[2] = smp; diag[3] = seg;
      diag[4] = __float_as_uint(o.x); diag[5] = __float_as_uint(o.y); diag[6] = __float_as_uint(o.z);
      diag[7] = __float_as_uint(d.x); diag[8] = __float_as_uint(d.y); diag[9] = __float_as_uint(d.z);
    }
    return false;
  }
  if (!found) {
    if (reflected) { bin = sky_bin(d, a.mf, a.nBins, a.alpha, a.cosN, a.sinN); gain = w * (3.14159265f / float(a.M)); }
    return false;
  }
  const kgb_slot sl = c.slot < a.nSlots ? a.slots[c.slot] : kgb_slot{0.2f, 0.f, 0.f, 0u};
  TriHit h;
  if (!tri_geom(c.v0, c.v1, c.v2, c.h, h)) return false;
  if (seg == 0 && own_plane(h, c.h.t, d, nn)) { o = through(h); return true; }
  if ((sl.flags & (KGB_SLOT_THIN | KGB_SLOT_TWIN)) == KGB_SLOT_THIN && h.front == ((sl.flags & KGB_SLOT_INWARD) != 0)) { o = through(h); return true; }
  const bool mirror = (sl.flags & KGB_SLOT_GLASS) != 0;
  float T = sl.tau, R = sl.rho;
  if (mirror) { glass_TR(fabsf(dot(d, h.n)), sl.tn, a.slotLog[c.slot], T, R); if (!(sl.tau > 0.f)) T = 0.f; }
  else if (diffuse == a.nBounce) R = 0.f;
  if (!(T + R > 0.f)) return false;
  const U3 rr = pcg3d(gi, smp, k++);
  w *= T + R;
  if (u01(rr.x) * (T + R) < T) { o = through(h); return true; }
  reflected = true;
  if (mirror) d = sub(d, mul(2.f * dot(d, h.n), h.n));
  else {
    d = cosine_dir(h.n, u01(rr.y), u01(rr.z));
    if (++diffuse >= 2) {
      if (u01(pcg3d(gi, smp, k++).x) >= w) return false;
      w = 1.f;
    }
  }
  o = add(offset_ray(h.p, h.n), h.lift);
  return true;
}

// The warp's paths that go on, appended to the queue in lane order with one atomic per warp.
__device__ __forceinline__ void enqueue(bool go, const PathState& st, PathState* q, uint32_t* count) {
  const uint32_t lane = threadIdx.x & 31, act = __activemask(), m = __ballot_sync(act, go);
  if (!m) return;
  const uint32_t leader = __ffs(act) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(count, __popc(m));
  base = __shfl_sync(act, base, leader);
  if (go) q[base + __popc(m & ((1u << lane) - 1u))] = st;
}

// One mask for the sum and its leader: two reads of __activemask() may see different sets of converged lanes.
__device__ __forceinline__ void add_segments(const BounceArgs& a, uint32_t segments) {
  const uint32_t m = __activemask();
  const uint32_t sum = __reduce_add_sync(m, segments);
  if ((threadIdx.x & 31) == __ffs(m) - 1) atomicAdd(reinterpret_cast<unsigned long long*>(a.status + 1), (unsigned long long)sum);
}

// Paths in two kernels: k_bounce_paths traces every path's first segment, one thread a path; with a.order, sensor
// i = t / S and sample a.order[t % S] (S = s1 - s0): a warp's 32 paths start at one sensor and the order (the host sorts
// the launch's samples by their first direction before the per-sensor rotation) keeps their first directions in a
// narrow cone, so their walks share nodes; without it sensor i = t % n, sample s0 + t / n. The paths that go on are
// compacted into a queue, and k_bounce_rest traces their other segments, at most nBounce + 15 each, one segment of each
// of a warp's paths at a time: a lane whose path has ended takes the next one from the queue, so the lanes stay busy
// whatever the lengths of their paths and one launch sees all paths to their ends. A path's segments are the
// reference's loop body in order with its own counters, so where and when it runs changes no result. A path that ends
// leaves its sky bin (where it escaped after a reflection, or none) and contribution (w x pi / M) in
// contrib[(sample - s0) n + i]; k_bounce_accum adds them to each sensor's rows in sample order, as the reference's
// per-sensor loop over samples does.
__global__ void __launch_bounds__(128) k_bounce_paths(BounceArgs a) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t S = a.s1 - a.s0;
  if (t >= a.n * S) return;
  const uint32_t i = a.order ? t / S : t % a.n, smp = a.order ? a.order[t % S] : a.s0 + t / a.n;
  const Scene s{a.nodes, a.tris, a.nNodes};
  const bool cull = (a.rayFlags & KGB_RAY_CULL_BACK_FACING) != 0;
  const uint32_t gi = a.i0 + i;
  const F3 nn = ld3(a.N + 3 * gi);
  F3 o = offset_ray(ld3(a.P + 3 * gi), nn);
  const U3 rot = pcg3d(gi, ~0u, ~0u);
  const float r0 = u01(rot.x), r1 = u01(rot.y);
  const float u = float(smp) / float(a.M) + r0, v = u01(__brev(smp)) + r1;
  F3 d = cosine_dir(nn, u - floorf(u), v - floorf(v));
  float w = 1.f, gain = 0.f;
  uint32_t k = 0, diffuse = 0, bin = kNoBin, overflow = 0;
  bool reflected = false;
  const uint32_t at = (smp - a.s0) * a.n + i;
  const bool go = bounce_segment(a, s, cull, 0, nn, gi, smp, o, d, w, k, diffuse, reflected, bin, gain, overflow);
  PathState st;
  if (go) {
    st.ox = o.x; st.oy = o.y; st.oz = o.z; st.gi = gi; st.dx = d.x; st.dy = d.y; st.dz = d.z; st.smp = smp;
    st.w = w; st.k = k; st.bits = diffuse | (reflected ? 0x100u : 0u) | (1u << 16); st.at = at;
  } else {
    a.contrib[at] = make_uint2(bin, __float_as_uint(gain));
  }
  enqueue(go, st, a.queue, a.qCount);
  add_segments(a, 1u);
  if (overflow) atomicOr(a.status, (overflow & 1u ? kStatusStackOverflow : 0u) | (overflow & 2u ? kStatusVisitLimit : 0u));
}

// The queue's paths to their ends. The next path's index is a counter, taken once a round for all of a warp's free lanes.
// Bound as the first segments are by the walk's instructions, with the rays of a warp in all directions, and by the last
// paths' chain of segments (about 14 us each) once the queue is empty. A launch per segment over a compacted queue, before,
// paid for that chain and the launches of the segments that no path reaches: 20,011 sensors x 1024 paths 13.3 to 11.5 ms.
// (Ordering the queue by direction and place first: its second segments 4.8 to 4.0 ms, less than a sort costs.)
__global__ void __launch_bounds__(128) k_bounce_rest(BounceArgs a) {
  const Scene s{a.nodes, a.tris, a.nNodes};
  const bool cull = (a.rayFlags & KGB_RAY_CULL_BACK_FACING) != 0;
  const uint32_t count = *a.qCount, lane = threadIdx.x & 31;
  uint32_t overflow = 0, segments = 0;
  const uint64_t start = clock_ns();
  bool have = false, late = false, more = true;
  PathState st{};
  while (true) {
    const uint32_t open = __ballot_sync(0xffffffffu, !have);
    if (open && more) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(a.qNext, uint32_t(__popc(open)));
      base = __shfl_sync(0xffffffffu, base, 0);
      const uint32_t q = base + __popc(open & ((1u << lane) - 1u));
      if (!have && q < count) { st = a.queue[q]; have = true; }
      more = base + __popc(open) < count;
    }
    if (!__any_sync(0xffffffffu, have)) break;
    if (have && !late && clock_ns() - start >= a.limitNs) late = true;
    if (have && late) {   // past the limit: the path ends with no contribution, and the call fails
      a.contrib[st.at] = make_uint2(kNoBin, 0u);
      have = false;
    } else if (have) {
      F3 o = f3(st.ox, st.oy, st.oz), d = f3(st.dx, st.dy, st.dz);
      float gain = 0.f;
      uint32_t diffuse = st.bits & 0xffu, bin = kNoBin;
      bool reflected = (st.bits & 0x100u) != 0;
      const uint32_t seg = st.bits >> 16;
      have = bounce_segment(a, s, cull, seg, f3(0.f, 0.f, 0.f), st.gi, st.smp, o, d, st.w, st.k, diffuse, reflected, bin, gain, overflow) &&
             seg + 1 < a.nBounce + 16;
      ++segments;
      if (have) {
        st.ox = o.x; st.oy = o.y; st.oz = o.z; st.dx = d.x; st.dy = d.y; st.dz = d.z;
        st.bits = diffuse | (reflected ? 0x100u : 0u) | ((seg + 1) << 16);
      } else {
        a.contrib[st.at] = make_uint2(bin, __float_as_uint(gain));
      }
    }
    __syncwarp();
  }
  add_segments(a, segments);
  if (overflow || late)
    atomicOr(a.status, (overflow & 1u ? kStatusStackOverflow : 0u) | (overflow & 2u ? kStatusVisitLimit : 0u) | (late ? kStatusTimeout : 0u));
}

// Per sensor, the launch's samples in order: row[bin] = row[bin] + contribution (the reference's float additions). A warp
// a sensor, 32 samples a round: the lane of a bin's first sample reads the bin's row, adds the round's contributions of
// that bin in lane order and writes it. The rounds' reads are what it waits for; the next round's results are read ahead.
// Against a thread a sensor with its results' reads grouped by eight: calls of 20,011 sensors x 1024 paths 10.7 to 10.4
// ms, 5003 x 1024 3.00 to 2.67, 2000 x 1024 1.39 to 1.09, 30 x 4096 1.09 to 0.34. A launch past its time limit adds nothing.
__global__ void __launch_bounds__(128) k_bounce_accum(BounceArgs a) {
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31, S = a.s1 - a.s0;
  if (i >= a.n || (*a.status & kStatusTimeout)) return;
  float* row = a.dc + i;
  const uint2 none = make_uint2(kNoBin, 0u);
  uint2 next = lane < S ? __ldg(a.contrib + size_t(lane) * a.n + i) : none;
  for (uint32_t q0 = 0; q0 < S; q0 += 32) {
    const uint2 c = next;
    const uint32_t q = q0 + 32 + lane;
    next = q < S ? __ldg(a.contrib + size_t(q) * a.n + i) : none;
    const float gain = __uint_as_float(c.y);
    const uint32_t peers = __match_any_sync(0xffffffffu, c.x);
    const bool first = c.x != kNoBin && lane == __ffs(peers) - 1;
    float* p = row + size_t(c.x) * a.nc;
    uint32_t more = first ? peers & (peers - 1u) : 0u;
    float v = 0.f;
    if (first) v = *p + gain;
    while (__any_sync(0xffffffffu, more != 0)) {
      const float g = __shfl_sync(0xffffffffu, gain, more ? __ffs(more) - 1 : lane);
      if (more) { v = v + g; more &= more - 1u; }
    }
    if (first) *p = v;
    __syncwarp();
  }
}

// The same for launches of few samples (many sensors), a thread a sensor: it reads eight results, then their bins' rows, at
// once, and a bin met again among them goes on from the sum it has. 199,000 sensors x 1 / 2 / 8 paths: 308 / 432 / 1180 us
// against 335 / 453 / 1192 with a warp a sensor, most of whose lanes have no sample.
constexpr uint32_t kAccumFew = 16;
__global__ void __launch_bounds__(64) k_bounce_accum_few(BounceArgs a) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n || (*a.status & kStatusTimeout)) return;
  constexpr uint32_t B = 8;
  float* row = a.dc + i;
  const uint32_t S = a.s1 - a.s0;
  for (uint32_t q0 = 0; q0 < S; q0 += B) {
    uint2 c[B];
    float v[B];
#pragma unroll
    for (uint32_t k = 0; k < B; ++k) c[k] = q0 + k < S ? __ldcs(a.contrib + size_t(q0 + k) * a.n + i) : make_uint2(kNoBin, 0u);
#pragma unroll
    for (uint32_t k = 0; k < B; ++k) v[k] = c[k].x != kNoBin ? row[size_t(c[k].x) * a.nc] : 0.f;
#pragma unroll
    for (uint32_t k = 0; k < B; ++k) {
#pragma unroll
      for (uint32_t j = 0; j < k; ++j) if (c[j].x == c[k].x) v[k] = v[j];
      v[k] = v[k] + __uint_as_float(c[k].y);
    }
#pragma unroll
    for (uint32_t k = 0; k < B; ++k) if (c[k].x != kNoBin) row[size_t(c[k].x) * a.nc] = v[k];
  }
}

// ---------------------------------------------------------------------------------------------------- launches
__global__ void __launch_bounds__(256) k_ray_table(const float* D, uint32_t nDir, RayDir* tab) {
  const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d < nDir) tab[d] = ray_dir_of(ld3(D + 3 * d));
}
// A sensor's orientation class: twice the dominant axis of its normal (x 0, y 1, z 2), plus one when that component is
// positive.
__global__ void k_sensor_classes(const float* N, uint32_t n, uint8_t* cls, uint32_t* flags) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t c = 6;   // no sensor
  if (i < n) {
    const float x = N[3 * i], y = N[3 * i + 1], z = N[3 * i + 2];
    const float ax = fabsf(x), ay = fabsf(y), az = fabsf(z);
    const uint32_t k = (ax >= ay && ax >= az) ? 0u : (ay >= az ? 1u : 2u);
    c = 2u * k + ((k == 0 ? x : k == 1 ? y : z) > 0.f ? 1u : 0u);
    if (cls[i] != c) { cls[i] = uint8_t(c); atomicOr(flags, 1u); }
  }
  for (uint32_t k = 0; k < 6; ++k) {   // counts, one atomic per warp and class
    const uint32_t m = __ballot_sync(~0u, c == k);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(flags + 1 + k, uint32_t(__popc(m)));
  }
}
void launch_sensor_classes(const float* N, uint32_t n, uint8_t* cls, uint32_t* flags, cudaStream_t st) {
  if (n) k_sensor_classes<<<(n + 255) / 256, 256, 0, st>>>(N, n, cls, flags);
}

void launch_ray_table(const float* D, uint32_t nDir, void* tab, cudaStream_t st) {
  if (nDir) k_ray_table<<<(nDir + 255) / 256, 256, 0, st>>>(D, nDir, static_cast<RayDir*>(tab));
}
int bytes_blocks_per_sm() {   // resident blocks of k_bytes per SM
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_bytes<true>, 256, 0) != cudaSuccess || b < 1) b = 1;
  return b;
}
int view_blocks_per_sm() {   // resident blocks of k_view per SM
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_view, 256, 0) != cudaSuccess || b < 1) b = 1;
  return b;
}
int bits_blocks_per_sm() {   // resident blocks of k_bits per SM (its persistent grid fills the GPU once)
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_bits<false, 32, true>, 256, 0) != cudaSuccess || b < 1) b = 1;
  return b;
}
// Directions a task, for `sensors` blocks of 32 sensors x n directions on `warps` resident warps: 32, or fewer where the
// tasks are so few that their uneven lengths (a task turned away from its directions is culled, one along a street walks
// far) would leave warps idle at a launch's end: halved, down to `least`, until there are 64 tasks a warp. Kernel time
// with 32 always / 16 / 32 / 64 / 256 tasks a warp: 20 k sensors x 9066 bytes 16.3 / 15.2 / 14.5 / 14.3 / 14.6 ms, 25 k x
// 3600 views 23.2 / 21.6 / 20.9 / 20.6 / 20.7 ms, 12 k x 10,800 views 21.3 / 19.8 / 19.1 / 18.5 / 18.4 ms, 12 k x 2155
// bits 1.84 / 1.55 / 1.54 / 1.54 / 1.55 ms.
static uint32_t task_directions(size_t sensors, size_t n, size_t warps, uint32_t least) {
  uint32_t per = 32;
  while (per > least && sensors * ((n + per - 1) / per) < 64 * warps) per /= 2;
  return per;
}
static int task_grid(size_t tasks, int resident) { return int(std::min<size_t>(size_t(resident), (tasks + 7) / 8)); }
static void launch_frontiers(const TraceArgs& a, size_t blocks, cudaStream_t st) {
  k_frontiers<<<unsigned((blocks + kFrontierWarps - 1) / kFrontierWarps), 32 * kFrontierWarps, 0, st>>>(a);
}
void launch_bits(const TraceArgs& a, int resident, cudaStream_t st, bool count) {
  const size_t blocks = (size_t(a.n) + 31) / 32, words = blocks * a.nWords, warps = size_t(resident) * 8;
  if (!count && 4 * words < warps) { k_bits_few<<<unsigned(words), 32 * kFewWarps, 0, st>>>(a); return; }
  const uint32_t per = count ? 32u : task_directions(blocks, size_t(a.nWords) * 32, warps, 8);
  const int grid = task_grid(blocks * ((a.nDir + per - 1) / per), resident);
  const bool front = a.frontiers != nullptr;
  if (front) launch_frontiers(a, blocks, st);
  if (count) front ? k_bits<true, 32, true><<<grid, 256, 0, st>>>(a) : k_bits<true, 32, false><<<grid, 256, 0, st>>>(a);
  else if (per == 32) front ? k_bits<false, 32, true><<<grid, 256, 0, st>>>(a) : k_bits<false, 32, false><<<grid, 256, 0, st>>>(a);
  else if (per == 16) front ? k_bits<false, 16, true><<<grid, 256, 0, st>>>(a) : k_bits<false, 16, false><<<grid, 256, 0, st>>>(a);
  else front ? k_bits<false, 8, true><<<grid, 256, 0, st>>>(a) : k_bits<false, 8, false><<<grid, 256, 0, st>>>(a);
}
size_t frontier_bytes() { return sizeof(FrontierRec); }
void launch_bytes(const TraceArgs& args, int resident, cudaStream_t st) {
  TraceArgs a = args;
  const size_t blocks = (size_t(a.n) + 31) / 32;
  a.per = task_directions(blocks, a.nDir, size_t(resident) * 8, 1);
  const int grid = task_grid(blocks * ((a.nDir + a.per - 1) / a.per), resident);
  if (a.frontiers) {
    launch_frontiers(a, blocks, st);
    k_bytes<true><<<grid, 256, 0, st>>>(a);
  } else k_bytes<false><<<grid, 256, 0, st>>>(a);
}
void launch_view(const ViewArgs& args, int resident, cudaStream_t st) {
  ViewArgs a = args;
  const size_t blocks = (size_t(a.n) + kViewSensors - 1) / kViewSensors;
  a.per = task_directions(blocks, a.K, size_t(resident) * 8, 32 / kViewSensors);
  if (blocks * a.K <= size_t(resident) * 8) a.per = 1;   // a warp for each (half empty): 1 sensor x 576 cells 43 to 37 us
  k_view<<<task_grid(blocks * ((size_t(a.K) + a.per - 1) / a.per), resident), 256, 0, st>>>(a);
}
// ln tn of each slot as a float pair (glass_TR's logarithm, once per slot; kgb_ln_pair, as kgb_powf takes it)
__global__ void k_slot_logs(const kgb_slot* slots, uint32_t n, float2* out) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  float h = 0.f, l = 0.f;
  if (slots[s].tn > 0.f) kgb_ln_pair(slots[s].tn, &h, &l);
  out[s] = make_float2(h, l);
}
void launch_slot_logs(const kgb_slot* slots, uint32_t n, float2* out, cudaStream_t st) {
  if (n) k_slot_logs<<<(n + 127) / 128, 128, 0, st>>>(slots, n, out);
}

// The first segments, the other segments of the paths that go on, then the accumulation. qCount: two counters (the
// queue's paths, and the next one to take); queue: n (s1 - s0) paths.
void launch_bounce(const BounceArgs& args, PathState* queue, uint32_t* qCount, int restGrid, cudaStream_t st) {
  BounceArgs a = args;
  const size_t paths = size_t(a.n) * (a.s1 - a.s0);
  a.queue = queue; a.qCount = qCount; a.qNext = qCount + 1;
  cudaMemsetAsync(qCount, 0, 8, st);
  // a warp a block: four-warp blocks, which end with their longest walk, kept 16 warps on an SM of the 20 that its
  // registers allow (20,011 sensors x 1024 paths 10.4 to 10.2 ms)
  k_bounce_paths<<<unsigned((paths + 31) / 32), 32, 0, st>>>(a);
  k_bounce_rest<<<restGrid, 128, 0, st>>>(a);
  if (a.s1 - a.s0 < kAccumFew) k_bounce_accum_few<<<(a.n + 63) / 64, 64, 0, st>>>(a);
  else k_bounce_accum<<<(a.n + 3) / 4, 128, 0, st>>>(a);
}
size_t bounce_state_bytes() { return sizeof(PathState); }
int bounce_rest_blocks_per_sm() {   // resident blocks of k_bounce_rest per SM (its grid fills the GPU once)
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_bounce_rest, 128, 0) != cudaSuccess || b < 1) b = 1;
  return b;
}

}  // namespace kgb
