// Device-side ray casting of the engine: the watertight ray/triangle test, the 8-wide BVH traversal
// (any-hit and closest-hit), and the reference's per-hit rules (own planes, glass, offsets, hashes).
//
// Numerics contract: the code deciding a result (hit or miss, t, own plane, transmittance byte, direction cell, sky
// bin) is a fixed sequence of IEEE-754 float operations: this header is compiled with -fmad=false and divisions /
// square roots are the correctly rounded ones, so the results equal a host restatement compiled without contraction
// bit for bit. Box tests only filter: they are conservative (see kWiden) and may use fused operations.
#pragma once
#include <cfloat>
#include <cstdint>
#include "kgb_detmath.h"
#include "kitsim_gb300.h"
#include "engine.h"

namespace kgb {

// ------------------------------------------------------------------------------------------------ data layout (HBM)
// BVH8 node, 208 bytes = 13 x 16 B:
//   n0: childBase | imask << 24 (childBase: index of the node's first inner child, below 2^24; its inner children are
//       consecutive in slot order; imask bit k: child k is an inner node), triBase (index of the node's first
//       triangle record), meta[8] (leaf child k: count << 5 | offset of its triangles from triBase, below 128; 0: empty
//       slot); bit 7 of meta[0], meta[1], meta[2] holds bit 0, 1, 2 of slots - 1 (slots: 1 + the last slot in use, so
//       these bits fall on slots in use only)
//   n1 n2: lo.x of children 0..3, 4..7 (float)   n3 n4: hi.x
//   n5 n6: lo.y                                  n7 n8: hi.y
//   n9 n10: lo.z                                 n11 n12: hi.z
//   (an empty slot holds lo = +inf, hi = -inf, which no ray enters)
// The child boxes are plain floats: the box test reads a ray's near and far planes straight from the two vectors its
// octant picks (Ray::nearX..: n1 or n3 for x; the far one is the index ^ 2), with no decoding. (The 80-byte form
// with 8-bit child boxes of Ylitie, Karras and Laine 2017 spent most of the box test's instructions decoding bytes.)
// Triangle record, 48 bytes = 3 x 16 B: v0.xyz + primitive index | v1.xyz + flags | v2.xyz + slot.
struct __align__(16) Node8 { uint4 n[kNodeWords / 4]; };
static_assert(sizeof(Node8) == 4 * kNodeWords, "node record size");
struct __align__(16) TriRec { float4 a, b, c; };
enum : uint32_t { kTriTranslucent = 1u };   // TriRec.b.w flag bits: the slot transmitted at build (any-hit)

struct F3 { float x, y, z; };
__device__ __forceinline__ F3 f3(float x, float y, float z) { return F3{x, y, z}; }
__device__ __forceinline__ F3 add(F3 a, F3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ F3 sub(F3 a, F3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ F3 mul(float s, F3 a) { return f3(s * a.x, s * a.y, s * a.z); }
__device__ __forceinline__ float dot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float comp(F3 a, int k) { return k == 0 ? a.x : k == 1 ? a.y : a.z; }
__device__ __forceinline__ F3 ld3(const float* p) { return f3(p[0], p[1], p[2]); }
__device__ __forceinline__ float next_up(float t) { return __uint_as_float(__float_as_uint(t) + 1u); }

// Waechter & Binder 2019 (Ray Tracing Gems, ch. 6), as the reference's offset_ray (trace_dev.cu:16-25).
__device__ __forceinline__ F3 offset_ray(F3 p, F3 n) {
  const float origin = 1.f / 32.f, floatScale = 1.f / 65536.f, intScale = 256.f;
  const int ox = int(intScale * n.x), oy = int(intScale * n.y), oz = int(intScale * n.z);
  const float px = __int_as_float(__float_as_int(p.x) + (p.x < 0.f ? -ox : ox));
  const float py = __int_as_float(__float_as_int(p.y) + (p.y < 0.f ? -oy : oy));
  const float pz = __int_as_float(__float_as_int(p.z) + (p.z < 0.f ? -oz : oz));
  return f3(fabsf(p.x) < origin ? p.x + floatScale * n.x : px, fabsf(p.y) < origin ? p.y + floatScale * n.y : py,
            fabsf(p.z) < origin ? p.z + floatScale * n.z : pz);
}

// Jarzynski & Olano 2020 (JCGT 9(3)): the reference's pcg3d / u01 (params.h:64-71).
struct U3 { uint32_t x, y, z; };
__device__ __forceinline__ U3 pcg3d(uint32_t x, uint32_t y, uint32_t z) {
  x = x * 1664525u + 1013904223u; y = y * 1664525u + 1013904223u; z = z * 1664525u + 1013904223u;
  x += y * z; y += z * x; z += x * y;
  x ^= x >> 16; y ^= y >> 16; z ^= z >> 16;
  x += y * z; y += z * x; z += x * y;
  return U3{x, y, z};
}
__device__ __forceinline__ float u01(uint32_t v) { return float(v >> 8) * (1.f / 16777216.f); }

// Radiance glass (the reference's glass_TR, glass.h:17-25; rad5R4 m_glass.c), powf as kgb_powf. lnTn: the slot's ln tn
// as a float pair (kgb_ln_pair, computed once per slot by k_slot_logs), so tn^(1 / c2) = kgb_pow_ln(lnTn, 1 / c2) is
// kgb_powf's value bit for bit, in float arithmetic only.
__device__ __forceinline__ void glass_TR(float c, float tn, float2 lnTn, float& T, float& R) {
  const float n = 1.52f;
  const float c2 = sqrtf((1.f - 1.f / (n * n)) + c * c / (n * n));
  const float d = tn > 0.f ? kgb_pow_ln(lnTn.x, lnTn.y, 1.f / c2) : 0.f, d2 = d * d;
  float rs = (c - n * c2) / (c + n * c2), rp = (c2 - n * c) / (c2 + n * c);
  rs *= rs; rp *= rp;
  T = .5f * (1.f - rs) * (1.f - rs) * d / (1.f - rs * rs * d2) + .5f * (1.f - rp) * (1.f - rp) * d / (1.f - rp * rp * d2);
  R = .5f * rs * (1.f + (1.f - 2.f * rs) * d2) / (1.f - rs * rs * d2) + .5f * rp * (1.f + (1.f - 2.f * rp) * d2) / (1.f - rp * rp * d2);
}

// x >= 0 as a double, exactly, without the FP64 pipe for a normal float: the exponent rebiased (+896) and the
// mantissa moved up 29 bits by integer operations (zero and subnormals take the conversion instruction).
__device__ __forceinline__ double widen(float x) {
  const uint32_t b = __float_as_uint(x);
  return x >= 1.17549435e-38f ? __hiloint2double(int((b >> 3) + (896u << 20)), int(b << 29)) : (double)x;
}

// ------------------------------------------------------------------------------------------------ the ray
struct Ray {
  F3 o, d;
  int kx, ky, kz;
  float Sx, Sy, Sz;
  F3 inv;     // box test: 1 / d with zero components replaced by +-2^-80
  F3 oinv;    // o * inv
  uint32_t oct;   // sign bits of d (closest-hit child order)
  uint32_t nearX, nearY, nearZ;   // node vectors of the near planes per axis (lo if inv >= 0, else hi); far: ^ 2
};
__device__ __forceinline__ void near_planes(Ray& r) {
  r.nearX = r.inv.x < 0.f ? 3u : 1u;
  r.nearY = r.inv.y < 0.f ? 7u : 5u;
  r.nearZ = r.inv.z < 0.f ? 11u : 9u;
}
__device__ __forceinline__ Ray make_ray(F3 o, F3 d) {
  Ray r;
  r.o = o; r.d = d;
  const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
  r.kz = ax >= ay ? (ax >= az ? 0 : 2) : (ay >= az ? 1 : 2);
  r.kx = r.kz == 2 ? 0 : r.kz + 1;
  r.ky = r.kx == 2 ? 0 : r.kx + 1;
  if (comp(d, r.kz) < 0.f) { const int t = r.kx; r.kx = r.ky; r.ky = t; }
  const float dz = comp(d, r.kz);
  r.Sx = comp(d, r.kx) / dz;
  r.Sy = comp(d, r.ky) / dz;
  r.Sz = 1.f / dz;
  const float tiny = 8.27180613e-25f;   // 2^-80
  const float dx = ax > tiny ? d.x : copysignf(tiny, d.x), dy = ay > tiny ? d.y : copysignf(tiny, d.y), dzz = az > tiny ? d.z : copysignf(tiny, d.z);
  r.inv = f3(1.f / dx, 1.f / dy, 1.f / dzz);
  r.oinv = f3(o.x * r.inv.x, o.y * r.inv.y, o.z * r.inv.z);
  r.oct = (d.x < 0.f ? 1u : 0u) | (d.y < 0.f ? 2u : 0u) | (d.z < 0.f ? 4u : 0u);
  near_planes(r);
  return r;
}

// The direction-only part of a ray (everything but the origin), 48 bytes, computed once per direction table by
// make_ray itself: a = d.xyz, Sx | b = inv.xyz, Sy | c = Sz, kx | ky << 8 | kz << 16 | oct << 24, 0, 0.
struct __align__(16) RayDir { float4 a, b, c; };
__device__ __forceinline__ RayDir ray_dir_of(F3 d) {
  const Ray r = make_ray(f3(0.f, 0.f, 0.f), d);
  RayDir t;
  t.a = make_float4(r.d.x, r.d.y, r.d.z, r.Sx);
  t.b = make_float4(r.inv.x, r.inv.y, r.inv.z, r.Sy);
  t.c = make_float4(r.Sz, __uint_as_float(uint32_t(r.kx) | uint32_t(r.ky) << 8 | uint32_t(r.kz) << 16 | r.oct << 24), 0.f, 0.f);
  return t;
}
// make_ray(o, d) from direction d's precomputed part: the same values, with o * inv the only arithmetic.
__device__ __forceinline__ Ray ray_from(const RayDir* tab, uint32_t d, F3 o) {
  const float4 a = __ldg(&tab[d].a), b = __ldg(&tab[d].b), c = __ldg(&tab[d].c);
  Ray r;
  r.o = o; r.d = f3(a.x, a.y, a.z);
  const uint32_t k = __float_as_uint(c.y);
  r.kx = int(k & 0xffu); r.ky = int((k >> 8) & 0xffu); r.kz = int((k >> 16) & 0xffu); r.oct = k >> 24;
  r.Sx = a.w; r.Sy = b.w; r.Sz = c.x;
  r.inv = f3(b.x, b.y, b.z);
  r.oinv = f3(o.x * r.inv.x, o.y * r.inv.y, o.z * r.inv.z);
  near_planes(r);
  return r;
}

struct Hit { float t, u, v; uint32_t prim; bool front; };

// Woop, Benthin, Wald 2013 (JCGT 2(1)) with a tie rule on edges: the same operation sequence as the oracle's hit_tri.
// x(i), y(i), z(i): vertex i relative to the origin along the ray's axes kx, ky, kz.
template <class X, class Y, class Z>
__device__ __forceinline__ bool hit_tri(const Ray& r, X&& x, Y&& y, Z&& z, float tmin, float tmax, bool cullBack, Hit& h) {
  const float Akz = z(0), Bkz = z(1), Ckz = z(2);
  const float Ax = x(0) - r.Sx * Akz, Ay = y(0) - r.Sy * Akz;
  const float Bx = x(1) - r.Sx * Bkz, By = y(1) - r.Sy * Bkz;
  const float Cx = x(2) - r.Sx * Ckz, Cy = y(2) - r.Sy * Ckz;
  float U = Cx * By - Cy * Bx, V = Ax * Cy - Ay * Cx, W = Bx * Ay - By * Ax;
  if (U == 0.f || V == 0.f || W == 0.f) {
    U = float(double(Cx) * double(By) - double(Cy) * double(Bx));
    V = float(double(Ax) * double(Cy) - double(Ay) * double(Cx));
    W = float(double(Bx) * double(Ay) - double(By) * double(Ax));
  }
  if ((U < 0.f || V < 0.f || W < 0.f) && (U > 0.f || V > 0.f || W > 0.f)) return false;
  const float det = U + V + W;
  if (det == 0.f) return false;
  if (cullBack && det < 0.f) return false;
  if (U == 0.f || V == 0.f || W == 0.f) {   // the ray meets an edge's line: one of the two triangles sharing it takes it
    const float s = det > 0.f ? 1.f : -1.f;
    if (U == 0.f) { const float ex = s * (Cx - Bx), ey = s * (Cy - By); if (!(ey > 0.f || (ey == 0.f && ex > 0.f))) return false; }
    if (V == 0.f) { const float ex = s * (Ax - Cx), ey = s * (Ay - Cy); if (!(ey > 0.f || (ey == 0.f && ex > 0.f))) return false; }
    if (W == 0.f) { const float ex = s * (Bx - Ax), ey = s * (By - Ay); if (!(ey > 0.f || (ey == 0.f && ex > 0.f))) return false; }
  }
  const float Az = r.Sz * Akz, Bz = r.Sz * Bkz, Cz = r.Sz * Ckz;
  const float T = U * Az + V * Bz + W * Cz;
  const float t = T / det;
  if (!(t >= tmin && t <= tmax)) return false;
  h.t = t; h.u = V / det; h.v = W / det; h.front = det > 0.f;
  return true;
}

// The reference's hit_triangle (trace_dev.cu:37-52): point, unit normal on the ray's side (1/sqrt), ext, lift.
struct TriHit { F3 p, n, lift; float ext; bool front; };
__device__ __forceinline__ bool tri_geom(F3 v0, F3 v1, F3 v2, const Hit& hh, TriHit& h) {
  const F3 e1 = sub(v1, v0), e2 = sub(v2, v0);
  const F3 ng = f3(e1.y * e2.z - e1.z * e2.y, e1.z * e2.x - e1.x * e2.z, e1.x * e2.y - e1.y * e2.x);
  const float l2 = dot(ng, ng);
  if (!(l2 > 0.f)) return false;
  const float inv = 1.f / sqrtf(l2);
  h.front = hh.front;
  h.n = mul(h.front ? inv : -inv, ng);
  h.p = add(add(v0, mul(hh.u, e1)), mul(hh.v, e2));
  h.ext = fmaxf(fmaxf(fmaxf(fabsf(e1.x), fabsf(e1.y)), fmaxf(fabsf(e1.z), fabsf(e2.x))), fmaxf(fabsf(e2.y), fabsf(e2.z)));
  h.lift = mul(h.ext * 9.5367432e-7f, h.n);
  return true;
}
// own_plane / own_hit / through (trace_dev.cu:60-72, 63)
__device__ __forceinline__ bool own_plane(const TriHit& h, float t, F3 d, F3 n) {
  return t * fabsf(dot(d, h.n)) < h.ext * 2.3841858e-7f && dot(n, h.n) <= 0.f;
}
__device__ __forceinline__ bool own_hit(F3 v0, F3 v1, F3 v2, const Hit& hh, F3 d, F3 n) {
  if (!(hh.t * dot(n, d) < 1.f / 32.f)) return false;
  TriHit h;
  return tri_geom(v0, v1, v2, hh, h) && own_plane(h, hh.t, d, n);
}
__device__ __forceinline__ F3 through(const TriHit& h) { return sub(offset_ray(h.p, mul(-1.f, h.n)), h.lift); }

// ------------------------------------------------------------------------------------------------ BVH8 traversal
__device__ __forceinline__ uint32_t byte_of(uint32_t w, int k) { return (w >> (8 * k)) & 0xffu; }

// The helpers below hold inline PTX; their host branches (plain C++, the same values) let tests and tools compile
// this header for the CPU.
__device__ __forceinline__ float max3f(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
#else
  return fmaxf(fmaxf(a, b), c);
#endif
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
#else
  return fminf(fminf(a, b), c);
#endif
}

// Two floats in one 64-bit register pair, for the packed FP32 instructions (add / mul / fma .f32x2, sm_100 and
// later): each half is rounded exactly as the scalar instruction rounds it.
__device__ __forceinline__ unsigned long long pk2(float a, float b) {
#if defined(__CUDA_ARCH__)
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
#else
  return (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32);
#endif
}
__device__ __forceinline__ void up2(unsigned long long r, float& a, float& b) {
#if defined(__CUDA_ARCH__)
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
#else
  a = __uint_as_float(uint32_t(r)); b = __uint_as_float(uint32_t(r >> 32));
#endif
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
#if defined(__CUDA_ARCH__)
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
#else
  float a0, a1, b0, b1, c0, c1;
  up2(a, a0, a1); up2(b, b0, b1); up2(c, c0, c1);
  return pk2(fmaf(a0, b0, c0), fmaf(a1, b1, c1));
#endif
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
#if defined(__CUDA_ARCH__)
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
#else
  float a0, a1, b0, b1;
  up2(a, a0, a1); up2(b, b0, b1);
  return pk2(a0 * b0, a1 * b1);
#endif
}
// Two words as one packed pair (the low word first).
__device__ __forceinline__ unsigned long long pku(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
  return r;
#else
  return (unsigned long long)a | ((unsigned long long)b << 32);
#endif
}

// What the box test owes a hit that the triangle test computes, with u = 2^-24 (a float's half ulp), t the hit's
// distance, L the triangle's extent, K = L^2 / (2 area), M the scene's largest coordinate:
//  - the triangle test signs its edge functions exactly for vertices slightly off where they are relative to the ray:
//    subtracting the origin, shearing and rounding the result move them by at most 4 u t |d_a| + 6 u L along axis a
//    (Sx times the depth is t |d_a| up to L, and so is the vertex's offset). So the ray's line passes within that of the
//    triangle, and 4 u t |d_a| is 4 u of the axis's slab distance;
//  - t is the depth of the vertices weighted by the edge functions. A weight is off by some u L^2 over the triangle's area
//    as seen along the ray, and t by as much of L: up to some u L K / s, s the sine of the ray against the triangle's plane;
//  - not so for a triangle perpendicular to an axis: its sheared coordinates across that axis are its depths times the
//    shear (plus its one distance from the origin), so their errors shrink with s as that area does. The weights move t by
//    at most 12 u L K, the other roundings by 14 u L and a few u of itself, at any incidence;
//  - a slab distance fma(plane, 1 / d, -o / d) is off by 3 u of itself and, for a coordinate |o_a| up to 6 M, by 7 u M in
//    distance (the products' rounding and the planes'); past 6 M that too is a small part of the slab distance.
// The exit distance is widened by kWiden, 1 + 32 u, which covers the parts relative to t on both sides of the interval;
// the triangles' boxes are expanded by prim_eps, which covers the others: 8 u M + 32 u L K for triangles perpendicular to
// an axis, 256 u M for the others. That leaves out, of the others, hits of s < L K / 8 M at worst whose t is off by more: the
// ray starts within some 30 u L K of the triangle's plane, past its edge, and leaves it nearly along the plane. A walk may
// miss such a hit, and then that of another tree may not (three of 8 million rays made for it).
// With 256 u M for every triangle, 6 mm on a 400 m block, more than the 0.1 to 4 mm by which offset_ray lifts a sensor off
// its face, every ray began inside the boxes of its own wall and walked down to its triangles. With the walls' boxes behind
// the sensors the urban block's rays visit about 6.9 nodes instead of 8.2 and test 0.9 triangles instead of 1.9 (trace 57.5
// to 43.3 ms); the boxes of walls turned against the axes hold their sensors either way. (The smaller expansion only along
// the axis that the triangle is perpendicular to: 7 % slower on the block; for every triangle: the turned ones lose grazing
// hits that 256 u M keeps, 220 of the 8 million rays, for 0.5 to 2 % of the views' time.)
constexpr float kWiden = 1.0000019073486328125f;   // 1 + 2^-19

// Child boxes of the node at p against the ray in [tmin, tmax] (tmin >= 0): returns the mask of hit children (bit k),
// their entry distances in tn[8]. Per axis the slab distance of a plane is fma(plane, inv, -o inv); the near planes
// are the low ones when inv >= 0, else the high ones, and the ray's nearX.. index picks their vector (the far one is
// the other). Children go in pairs through the packed fma: per pair one fma.f32x2 per plane, per child one 3-input max
// and one 3-input min. Empty child slots (lo +inf, hi -inf) fail the test; a leaf slot without triangles that passes
// tests nothing.
// CLIP: the exit is also clipped at tmax (closest hit: the best hit so far times kWiden, as a box's entry may lie that
// much past a hit in it). Without it boxes beyond tmax pass as well, which is conservative: the triangle test applies
// tmax (the any-hit walks run to infinity).
// 1 + the node's last slot in use, from bit 7 of its first three meta bytes (the word of meta[0..3]).
__device__ __forceinline__ uint32_t node_slots(uint32_t meta03) {
  return 1u + (((meta03 >> 7) & 1u) | ((meta03 >> 14) & 2u) | ((meta03 >> 21) & 4u));
}

// SKIP: slots past the node's last child (empty boxes, which fail the test anyway) are neither read nor tested. The
// byte-mode trace and the bounce's walks run faster with it (10.5 against 9.8 G rays/s, 1283 against 1200 M paths/s);
// the visibility bits' walk and the views' closest hits run slower (the extra branches cost more than the tests they
// save: 64.9 against 61.0 ms for the urban trace), so those test every slot.
template <bool CLIP = true, bool SKIP = false>
__device__ __forceinline__ uint32_t node_hits(const uint4* p, const Ray& r, float tmin, float tmax, uint32_t slots, float* tn) {
  const unsigned long long IX = pk2(r.inv.x, r.inv.x), IY = pk2(r.inv.y, r.inv.y), IZ = pk2(r.inv.z, r.inv.z);
  const unsigned long long OX = pk2(-r.oinv.x, -r.oinv.x), OY = pk2(-r.oinv.y, -r.oinv.y), OZ = pk2(-r.oinv.z, -r.oinv.z);
  const unsigned long long WIDEN = pk2(kWiden, kWiden);
  const uint32_t fX = r.nearX ^ 2u, fY = r.nearY ^ 2u, fZ = r.nearZ ^ 2u;
  uint32_t mask = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {   // children 4h .. 4h + 3: the second vector of each plane set
    if (SKIP && 4 * h >= int(slots)) break;
    const uint4 nx = __ldg(p + r.nearX + h), fx = __ldg(p + fX + h);
    const uint4 ny = __ldg(p + r.nearY + h), fy = __ldg(p + fY + h);
    const uint4 nz = __ldg(p + r.nearZ + h), fz = __ldg(p + fZ + h);
#pragma unroll
    for (int j = 0; j < 2; ++j) {   // the pair 4h + 2j, 4h + 2j + 1
      const int k = 4 * h + 2 * j;
      if (SKIP && k >= int(slots)) break;
      float tnx[2], tny[2], tnz[2], tfx[2], tfy[2], tfz[2];
      up2(fma2(j ? pku(nx.z, nx.w) : pku(nx.x, nx.y), IX, OX), tnx[0], tnx[1]);
      up2(fma2(j ? pku(fx.z, fx.w) : pku(fx.x, fx.y), IX, OX), tfx[0], tfx[1]);
      up2(fma2(j ? pku(ny.z, ny.w) : pku(ny.x, ny.y), IY, OY), tny[0], tny[1]);
      up2(fma2(j ? pku(fy.z, fy.w) : pku(fy.x, fy.y), IY, OY), tfy[0], tfy[1]);
      up2(fma2(j ? pku(nz.z, nz.w) : pku(nz.x, nz.y), IZ, OZ), tnz[0], tnz[1]);
      up2(fma2(j ? pku(fz.z, fz.w) : pku(fz.x, fz.y), IZ, OZ), tfz[0], tfz[1]);
      // exit widened to tfar kWiden; a negative tfar fails against tnear >= tmin >= 0 either way
      float tf[2];
      up2(mul2(pk2(min3f(tfx[0], tfy[0], tfz[0]), min3f(tfx[1], tfy[1], tfz[1])), WIDEN), tf[0], tf[1]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float tnear = max3f(tnx[e], tny[e], fmaxf(tnz[e], tmin));
        const float tfar = CLIP ? fminf(tf[e], tmax) : tf[e];
        if (tnear <= tfar) { mask |= 1u << (k + e); tn[k + e] = tnear; }
      }
    }
  }
  return mask;
}

__device__ __forceinline__ void load_tri(const TriRec* tris, uint32_t j, F3& v0, F3& v1, F3& v2, uint32_t& prim, uint32_t& flags, uint32_t& slot) {
  const float4* p = reinterpret_cast<const float4*>(tris + j);
  const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
  v0 = f3(a.x, a.y, a.z); v1 = f3(b.x, b.y, b.z); v2 = f3(c.x, c.y, c.z);
  prim = __float_as_uint(a.w); flags = __float_as_uint(b.w); slot = __float_as_uint(c.w);
}

// The triangle at rec (a record) against the ray, its coordinates read along the ray's axes, one by one.
__device__ __forceinline__ bool hit_record(const TriRec* rec, const Ray& r, float tmin, float tmax, bool cull, Hit& h) {
  const float ox = comp(r.o, r.kx), oy = comp(r.o, r.ky), oz = comp(r.o, r.kz);
  const float* p = reinterpret_cast<const float*>(rec);
  const float *px = p + r.kx, *py = p + r.ky, *pz = p + r.kz;
  return hit_tri(r, [&](int i) { return __ldg(px + 4 * i) - ox; }, [&](int i) { return __ldg(py + 4 * i) - oy; },
                 [&](int i) { return __ldg(pz + 4 * i) - oz; }, tmin, tmax, cull, h);
}
// The triangle of vertices v0 v1 v2 against the ray.
__device__ __forceinline__ bool hit_vertices(const Ray& r, F3 v0, F3 v1, F3 v2, float tmin, float tmax, bool cull, Hit& h) {
  const F3 A = sub(v0, r.o), B = sub(v1, r.o), C = sub(v2, r.o);
  const auto at = [&](int i, int k) { return comp(i == 0 ? A : i == 1 ? B : C, k); };
  return hit_tri(r, [&](int i) { return at(i, r.kx); }, [&](int i) { return at(i, r.ky); }, [&](int i) { return at(i, r.kz); }, tmin, tmax, cull, h);
}

struct Scene {
  const Node8* nodes;
  const TriRec* tris;
  uint32_t nNodes;    // 0: empty scene, every ray misses
};

// the GPU's nanosecond clock (kernels with a wall-time limit read it)
__device__ __forceinline__ uint64_t clock_ns() {
#if defined(__CUDA_ARCH__)
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
#else
  return 0;
#endif
}

constexpr int kStack = 48;   // node-group stack entries (one per level at most)
// Node visits of one query past which the traversal gives up (overflow bit 2): a query visits a node of a tree at
// most once, so more than the node count (or 2^20) means a damaged walk; it ends at once instead of running on.
constexpr uint32_t kMaxVisits = 1u << 20;
__device__ __forceinline__ uint32_t visit_cap(const Scene& s) { return min(kMaxVisits, s.nNodes + 8u); }

// Traversal counters of the instrumented kernels (nodes visited, triangles tested); compiled out otherwise.
struct Count {
  uint32_t nodes = 0, tris = 0;
};

// A leaf's triangle is tested by 5 to 8 of a warp's 32 lanes, and these tests are a third to two fifths of a walk's
// instructions (a test is some 90, 18 of them picking the coordinates along the ray's axes). LATE: hit_record, which reads
// them in place, and the whole record only for a hit: bounce 13.9 to 13.3 ms, views 18.5 to 18.25 ms (all around) and 20.5
// to 20.4 (fov 120); the visibility bits' walk spills with it (2 % slower).
// The triangles of a leaf: f(hit, v0, v1, v2, flags, slot) for every hit in [tmin, tmax]; true when f returned true.
template <bool COUNT, bool LATE, class Fn>
__device__ __forceinline__ bool leaf_hits(const Scene& s, const Ray& r, float tmin, float tmax, bool cull, uint32_t first, uint32_t cnt, Fn&& f,
                                          Count* ctr) {
  for (uint32_t j = first; j < first + cnt; ++j) {
    if (COUNT) ctr->tris++;
    Hit h;
    if (LATE) {
      if (hit_record(s.tris + j, r, tmin, tmax, cull, h)) {
        F3 v0, v1, v2;
        uint32_t prim, flags, slot;
        load_tri(s.tris, j, v0, v1, v2, prim, flags, slot);
        h.prim = prim;
        if (f(h, v0, v1, v2, flags, slot)) return true;
      }
    } else {
      F3 v0, v1, v2;
      uint32_t prim, flags, slot;
      load_tri(s.tris, j, v0, v1, v2, prim, flags, slot);
      if (hit_vertices(r, v0, v1, v2, tmin, tmax, cull, h)) {
        h.prim = prim;
        if (f(h, v0, v1, v2, flags, slot)) return true;
      }
    }
  }
  return false;
}

// Visit every triangle hit in [tmin, tmax] (any order) under the nodes that `next` gives one after the other (false: no
// more; ONE: it gives one node only); f(hit, v0, v1, v2, flags, slot) returns true to stop.
template <bool COUNT, bool SKIP, bool ONE, class Next, class Fn>
__device__ __forceinline__ void walk_hits(const Scene& s, const Ray& r, float tmin, float tmax, bool cull, Next&& next, Fn&& f, uint32_t& overflow,
                                          Count* ctr) {
  uint2 stack[kStack];   // node group: x = childBase, y = imask << 8 | remaining inner children
  int sp = 0;
  uint32_t cur;          // node to visit
  if (!next(cur)) return;
  const uint32_t cap = visit_cap(s);
  for (uint32_t visits = 0;; ++visits) {
    if (visits >= cap || cur >= s.nNodes) { overflow |= 2u; return; }
    const uint4* np = reinterpret_cast<const uint4*>(s.nodes + cur);
    const uint4 hd = __ldg(np);
    if (COUNT) ctr->nodes++;
    float tn[8];
    const uint32_t hit = node_hits<false, SKIP>(np, r, tmin, tmax, SKIP ? node_slots(hd.z) : 8u, tn);
    const uint32_t imask = hd.x >> 24, childBase = hd.x & 0xffffffu;
    uint32_t leaves = hit & ~imask;
    while (leaves) {
      const int k = __ffs(leaves) - 1;
      leaves &= leaves - 1;
      const uint32_t meta = byte_of(k < 4 ? hd.z : hd.w, k & 3);
      if (leaf_hits<COUNT, SKIP>(s, r, tmin, tmax, cull, hd.y + (meta & 31u), (meta >> 5) & 3u, f, ctr)) return;
    }
    const uint32_t inner = hit & imask;
    if (inner) {
      const int k = __ffs(inner) - 1;
      const uint32_t rest = inner & (inner - 1);
      if (rest) {
        if (sp < kStack) stack[sp++] = make_uint2(childBase, (imask << 8) | rest);
        else overflow = 1;
      }
      cur = childBase + __popc(imask & ((1u << k) - 1u));
      continue;
    }
    if (!sp) {
      if (ONE || !next(cur)) return;
      continue;
    }
    uint2& g = stack[sp - 1];
    const uint32_t rem = g.y & 0xffu, im = g.y >> 8;
    const int k = __ffs(rem) - 1;
    cur = g.x + __popc(im & ((1u << k) - 1u));
    const uint32_t left = rem & (rem - 1);
    if (left) g.y = (im << 8) | left; else --sp;
  }
}
// ... of the whole scene, from the root
template <bool COUNT = false, bool SKIP = false, class Fn>
__device__ __forceinline__ void for_hits(const Scene& s, const Ray& r, float tmin, float tmax, bool cull, Fn&& f, uint32_t& overflow,
                                         Count* ctr = nullptr) {
  if (!s.nNodes) return;
  walk_hits<COUNT, SKIP, true>(s, r, tmin, tmax, cull, [](uint32_t& cur) { cur = 0; return true; }, f, overflow, ctr);
}

// The closest hit in [tmin, tmax], ties broken by the smaller primitive index. Children are visited near to far: the
// nearest inner child next, the others pushed far to near; a node whose entry lies beyond the best hit so far is
// skipped. The visiting order changes nothing but the work: the result is the closest hit of the whole hit set.
struct ClosestOut { Hit h; F3 v0, v1, v2; uint32_t flags, slot; };
template <bool SKIP = false>
__device__ __forceinline__ bool closest(const Scene& s, const Ray& r, float tmin, float tmax, bool cull, ClosestOut& out, uint32_t& overflow) {
  if (!s.nNodes) return false;
  struct Entry { uint32_t node; float t; };
  Entry stack[kStack * 4];
  int sp = 0;
  bool any = false;
  float best = tmax, lim = tmax * kWiden;   // lim: the boxes' bound on the entry distance
  uint32_t cur = 0, visits = 0;
  const uint32_t cap = visit_cap(s);
  for (;;) {
    if (++visits > cap || cur >= s.nNodes) { overflow |= 2u; return any; }
    const uint4* np = reinterpret_cast<const uint4*>(s.nodes + cur);
    const uint4 hd = __ldg(np);
    float tn[8];
    const uint32_t hit = node_hits<true, SKIP>(np, r, tmin, lim, SKIP ? node_slots(hd.z) : 8u, tn);
    const uint32_t imask = hd.x >> 24, childBase = hd.x & 0xffffffu;
    uint32_t leaves = hit & ~imask;
    while (leaves) {
      const int k = __ffs(leaves) - 1;
      leaves &= leaves - 1;
      const uint32_t meta = byte_of(k < 4 ? hd.z : hd.w, k & 3);
      const uint32_t first = hd.y + (meta & 31u), cnt = (meta >> 5) & 3u;
      for (uint32_t j = first; j < first + cnt; ++j) {
        Hit h;
        if (hit_record(s.tris + j, r, tmin, best, cull, h)) {
          F3 v0, v1, v2;
          uint32_t prim, flags, slot;
          load_tri(s.tris, j, v0, v1, v2, prim, flags, slot);
          h.prim = prim;
          if (!any || h.t < out.h.t || (h.t == out.h.t && prim < out.h.prim)) {
            out.h = h; out.v0 = v0; out.v1 = v1; out.v2 = v2; out.flags = flags; out.slot = slot;
            any = true;
            best = h.t;
            lim = best * kWiden;
          }
        }
      }
    }
    // inner children still in front of the best hit, sorted far to near: the nearest is visited next
    uint32_t inner = hit & imask;
    Entry ch[8];
    int m = 0;
    while (inner) {
      const int k = __ffs(inner) - 1;
      inner &= inner - 1;
      if (tn[k] > lim) continue;
      const Entry x{childBase + __popc(imask & ((1u << k) - 1u)), tn[k]};
      int b = m - 1;
      while (b >= 0 && ch[b].t < x.t) { ch[b + 1] = ch[b]; --b; }
      ch[b + 1] = x;
      ++m;
    }
    if (m) {
      if (sp + m - 1 > kStack * 4) { overflow |= 1u; m = 1; }
      for (int a = 0; a < m - 1; ++a) stack[sp++] = ch[a];
      cur = ch[m - 1].node;
      continue;
    }
    for (;;) {   // the next pushed node still in front of the best hit
      if (!sp) return any;
      const Entry e = stack[--sp];
      if (e.t <= lim) { cur = e.node; break; }
    }
  }
}

// ------------------------------------------------------------------------------------------------ a warp's frontier
// The rays of a warp start close together, so each of them would walk the same nodes from the root down to where they
// start, testing the same subtrees' boxes on the way (a block's ray: 4 of 7 node visits; a city's 6 of 10). A warp opens
// those nodes once, for all its directions: its frontier is the set of subtrees (or leaves) left, which together hold
// every triangle. Per direction the warp tests the frontier's boxes against the shaft of all its rays (a lane per box), and
// each ray tests the few that are left (5 to 9 of 40 to 60) and walks into those it enters. Urban block: node visits a
// ray 6.4 to 3.1, trace 43.4 to 36.7 ms; city bits 4.23 to 3.29 ms. A warp whose sensors stand far apart against the
// scene's detail opens little and gains little (12 k sensors on the block 1.54 to 1.55 ms). Opening nodes down to half the
// origins' extent instead of all of it: 38.8 ms (more entries for each ray to test), to twice 36.6, to five times 39.0.
// The closest-hit walk of the views gained nothing by it: its rays differ in direction, which widens the shaft, and the
// nearer entries have to come first.
constexpr int kEntries = 64;   // subtrees a frontier holds; a node is opened while its up to 8 children fit
struct __align__(16) Frontier {   // in shared memory, one a warp
  float2 x[kEntries], y[kEntries], z[kEntries];   // an entry's box: lo, hi
  uint2 ref[kEntries];         // a node, 0 | a leaf's first triangle record, its triangles
  float open[kEntries];        // the extent of a node to open, else 0
};
#if defined(__CUDACC__)
__device__ __forceinline__ uint32_t order_bits(float f) {   // floats as unsigned integers of the same order
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_order_bits(uint32_t u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u); }

struct Bounds { F3 lo, hi; };   // of a warp's ray origins
// An origin that is not finite is left out: its rays hit nothing wherever they walk (hit_tri's t is not a number), and the
// bounds of the others stay finite, without which shaft would drop entries that their rays enter.
__device__ __forceinline__ Bounds origin_bounds(F3 o, bool valid) {
  Bounds b;
  valid = valid && fabsf(o.x) <= FLT_MAX && fabsf(o.y) <= FLT_MAX && fabsf(o.z) <= FLT_MAX;
  const uint32_t none = order_bits(INFINITY), no = order_bits(-INFINITY);
  b.lo.x = from_order_bits(__reduce_min_sync(~0u, valid ? order_bits(o.x) : none));
  b.lo.y = from_order_bits(__reduce_min_sync(~0u, valid ? order_bits(o.y) : none));
  b.lo.z = from_order_bits(__reduce_min_sync(~0u, valid ? order_bits(o.z) : none));
  b.hi.x = from_order_bits(__reduce_max_sync(~0u, valid ? order_bits(o.x) : no));
  b.hi.y = from_order_bits(__reduce_max_sync(~0u, valid ? order_bits(o.y) : no));
  b.hi.z = from_order_bits(__reduce_max_sync(~0u, valid ? order_bits(o.z) : no));
  return b;
}

// The frontier of a warp's rays: from the root, the largest node that holds some of the origins' bounds and is larger
// than them is opened, until none is or the entries are used up: at most kEntries nodes, so that it ends in a damaged tree
// too (the entries hold every triangle after each). Returns the entries. Every lane calls it.
__device__ __forceinline__ uint32_t build_frontier(const Scene& s, const Bounds& b, Frontier& f, uint32_t lane) {
  if (!s.nNodes) return 0;
  const float size = fmaxf(fmaxf(b.hi.x - b.lo.x, b.hi.y - b.lo.y), b.hi.z - b.lo.z);
  uint32_t n = 1, node = 0, at = 0;   // the entry that is opened holds `node`
  for (int opened = 0;;) {
    const uint4* np = reinterpret_cast<const uint4*>(s.nodes + node);
    const uint4 hd = __ldg(np);
    const uint32_t k = lane & 7u, imask = hd.x >> 24, meta = byte_of(k < 4 ? hd.z : hd.w, k & 3u) & 0x7fu;
    const bool inner = imask >> k & 1u, used = lane < 8 && (inner || meta);
    const uint32_t in = __ballot_sync(~0u, used);
    if (used) {
      const uint32_t rank = __popc(in & ((1u << lane) - 1u)), e = rank ? n + rank - 1 : at;
      const float* p = reinterpret_cast<const float*>(np) + 4 + k;
      const float2 x = make_float2(__ldg(p), __ldg(p + 8)), y = make_float2(__ldg(p + 16), __ldg(p + 24)), z = make_float2(__ldg(p + 32), __ldg(p + 40));
      const float ext = fmaxf(fmaxf(x.y - x.x, y.y - y.x), z.y - z.x);
      const uint32_t child = (hd.x & 0xffffffu) + __popc(imask & ((1u << k) - 1u));
      f.x[e] = x; f.y[e] = y; f.z[e] = z;
      f.ref[e] = inner ? make_uint2(child, 0u) : make_uint2(hd.y + (meta & 31u), meta >> 5);
      f.open[e] = inner && child < s.nNodes && ext > size && x.x <= b.hi.x && x.y >= b.lo.x && y.x <= b.hi.y && y.y >= b.lo.y && z.x <= b.hi.z &&
                  z.y >= b.lo.z ? ext : 0.f;
    }
    if (in) n += __popc(in) - 1;
    else if (!opened) return 0;                 // a root without children
    else if (lane == 0) f.open[at] = 0.f;       // such a node stays an entry
    __syncwarp();
    if (n + 7 > kEntries || ++opened == kEntries) break;
    const uint32_t x = lane < n ? __float_as_uint(f.open[lane]) : 0u, y = lane + 32 < n ? __float_as_uint(f.open[lane + 32]) : 0u;
    const uint32_t top = __reduce_max_sync(~0u, max(x, y));
    if (!top) break;
    at = __shfl_sync(~0u, x == top ? lane : lane + 32, __ffs(__ballot_sync(~0u, x == top || y == top)) - 1);
    node = f.ref[at].x;
    __syncwarp();
  }
  return n;
}

// A box's entry distance (at least tmin) against its widened exit; lo and hi planes have offsets of their own (o.x, o.y).
// Near and far planes are told apart by the distances: they order as the planes do, rounding included.
__device__ __forceinline__ bool box_entered(float2 x, float2 y, float2 z, const Ray& r, float2 ox, float2 oy, float2 oz, float tmin) {
  float x0, x1, y0, y1, z0, z1;
  up2(fma2(pk2(x.x, x.y), pk2(r.inv.x, r.inv.x), pk2(ox.x, ox.y)), x0, x1);
  up2(fma2(pk2(y.x, y.y), pk2(r.inv.y, r.inv.y), pk2(oy.x, oy.y)), y0, y1);
  up2(fma2(pk2(z.x, z.y), pk2(r.inv.z, r.inv.z), pk2(oz.x, oz.y)), z0, z1);
  const float near = max3f(fminf(x0, x1), fminf(y0, y1), fmaxf(fminf(z0, z1), tmin));
  return near <= min3f(fmaxf(x0, x1), fmaxf(y0, y1), fmaxf(z0, z1)) * kWiden;
}
// A frontier in global memory (k_frontiers), for launches whose tasks would each build the same ones.
struct __align__(16) FrontierRec {
  float4 box[3][32];   // x, y, z of two entries a lane
  uint4 ref[32];
  Bounds b;
  uint32_t n, pad;
};
__device__ __forceinline__ void load_frontier(const FrontierRec* rec, Frontier& f, uint32_t lane) {
  const float4 x = __ldg(&rec->box[0][lane]), y = __ldg(&rec->box[1][lane]), z = __ldg(&rec->box[2][lane]);
  const uint4 r = __ldg(&rec->ref[lane]);
  reinterpret_cast<float4*>(f.x)[lane] = x;
  reinterpret_cast<float4*>(f.y)[lane] = y;
  reinterpret_cast<float4*>(f.z)[lane] = z;
  reinterpret_cast<uint4*>(f.ref)[lane] = r;
  __syncwarp();
}
__device__ __forceinline__ void store_frontier(FrontierRec* rec, const Frontier& f, const Bounds& b, uint32_t n, uint32_t lane) {
  rec->box[0][lane] = reinterpret_cast<const float4*>(f.x)[lane];
  rec->box[1][lane] = reinterpret_cast<const float4*>(f.y)[lane];
  rec->box[2][lane] = reinterpret_cast<const float4*>(f.z)[lane];
  rec->ref[lane] = reinterpret_cast<const uint4*>(f.ref)[lane];
  if (lane == 0) { rec->b = b; rec->n = n; }
}

// The entries that some ray from within the bounds in r's direction may enter (all the warp's rays have it), as a mask:
// each ray's own test passes on a subset, rounding included, since every operation is monotonic (from finite origins).
struct Mask64 { uint32_t lo, hi; };
__device__ __forceinline__ Mask64 shaft(const Frontier& f, uint32_t n, const Bounds& b, const Ray& r, uint32_t lane) {
  // the near plane (lo when the direction is positive) against the origin farthest along, the far one against the first
  const float2 ox = make_float2(-(b.hi.x * r.inv.x), -(b.lo.x * r.inv.x)), oy = make_float2(-(b.hi.y * r.inv.y), -(b.lo.y * r.inv.y)),
               oz = make_float2(-(b.hi.z * r.inv.z), -(b.lo.z * r.inv.z));
  Mask64 m;
  m.lo = __ballot_sync(~0u, lane < n && box_entered(f.x[lane], f.y[lane], f.z[lane], r, ox, oy, oz, 0.f));
  m.hi = n > 32 ? __ballot_sync(~0u, lane + 32 < n && box_entered(f.x[lane + 32], f.y[lane + 32], f.z[lane + 32], r, ox, oy, oz, 0.f)) : 0u;
  return m;
}
// for_hits over the entries of a mask
template <bool COUNT, bool SKIP, class Fn>
__device__ __forceinline__ void frontier_hits(const Scene& s, const Frontier& fr, Mask64 entries, const Ray& r, float tmin, float tmax, bool cull, Fn&& f,
                                              uint32_t& overflow, Count* ctr) {
  const float2 ox = make_float2(-r.oinv.x, -r.oinv.x), oy = make_float2(-r.oinv.y, -r.oinv.y), oz = make_float2(-r.oinv.z, -r.oinv.z);
  // the same entry for every lane: its leaf's triangles are tested together
  const auto half = [&](uint32_t m, uint32_t base, uint32_t& mine) {
    mine = 0;
    for (; m; m &= m - 1) {
      const uint32_t k = __ffs(m) - 1, e = base + k;
      if (!box_entered(fr.x[e], fr.y[e], fr.z[e], r, ox, oy, oz, tmin)) continue;
      const uint2 ref = fr.ref[e];
      if (!ref.y) mine |= 1u << k;
      else if (leaf_hits<COUNT, SKIP>(s, r, tmin, tmax, cull, ref.x, ref.y, f, ctr)) return true;
    }
    return false;
  };
  uint32_t lo, hi;
  if (half(entries.lo, 0, lo) || half(entries.hi, 32, hi)) return;
  walk_hits<COUNT, SKIP, false>(s, r, tmin, tmax, cull, [&](uint32_t& cur) {
    if (lo) { cur = fr.ref[__ffs(lo) - 1].x; lo &= lo - 1; return true; }
    if (hi) { cur = fr.ref[31 + __ffs(hi)].x; hi &= hi - 1; return true; }
    return false;
  }, f, overflow, ctr);
}
#endif

// Bits of one visibility word, those of directions d0 .. dEnd - 1: bit d % 32 = direction d of a sensor (normal n, ray
// origin o) passes the hemisphere cull and every hit from tmin 1e-5 on is an own-plane hit, at most 3 (the reference's
// __raygen__bits, trace_dev.cu:91-108, restated over the ray's hit set). COUNT adds traversal counters and rays traced.
// D: the directions, tab: their precomputed RayDir entries.
template <bool COUNT>
__device__ __forceinline__ uint32_t trace_word(const Scene& s, F3 n, F3 o, const float* D, const RayDir* tab, uint32_t d0, uint32_t dEnd,
                                               bool cull, uint32_t& overflow, Count& ctr, uint32_t& rays) {
  uint32_t word = 0;
  for (uint32_t d = d0; d < dEnd; ++d) {
    const F3 dir = ld3(D + 3 * d);
    if (!(n.x * dir.x + n.y * dir.y + n.z * dir.z > 0.f)) continue;
    const Ray r = ray_from(tab, d, o);
    bool blocked = false;
    int own = 0;
    if (COUNT) ++rays;
    for_hits<COUNT>(s, r, 1e-5f, INFINITY, cull, [&](const Hit& h, F3 v0, F3 v1, F3 v2, uint32_t, uint32_t) {
      if (own_hit(v0, v1, v2, h, dir, n) && ++own <= 3) return false;
      blocked = true;
      return true;
    }, overflow, &ctr);
    if (!blocked) word |= 1u << (d & 31u);
  }
  return word;
}

#if defined(__CUDACC__)
// The same from the warp's frontier (entries of it in fr, b the bounds of the warp's origins); every lane calls it.
template <bool COUNT>
__device__ __forceinline__ uint32_t trace_word(const Scene& s, const Frontier& fr, uint32_t entries, const Bounds& b, F3 n, F3 o, bool valid,
                                               const RayDir* tab, uint32_t d0, uint32_t dEnd, bool cull, uint32_t& overflow, Count& ctr, uint32_t& rays) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t word = 0;
  for (uint32_t d = d0; d < dEnd; ++d) {
    const Ray r = ray_from(tab, d, o);
    const bool on = valid && n.x * r.d.x + n.y * r.d.y + n.z * r.d.z > 0.f;
    if (!__any_sync(~0u, on)) continue;
    const Mask64 m = shaft(fr, entries, b, r, lane);
    if (!on) continue;
    bool blocked = false;
    int own = 0;
    if (COUNT) ++rays;
    frontier_hits<COUNT, false>(s, fr, m, r, 1e-5f, INFINITY, cull, [&](const Hit& h, F3 v0, F3 v1, F3 v2, uint32_t, uint32_t) {
      if (own_hit(v0, v1, v2, h, r.d, n) && ++own <= 3) return false;
      blocked = true;
      return true;
    }, overflow, &ctr);
    if (!blocked) word |= 1u << (d & 31u);
  }
  return word;
}
#endif

}  // namespace kgb
