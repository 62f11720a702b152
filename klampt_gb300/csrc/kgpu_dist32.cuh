// kgpu_dist32.cuh — FP32 distance helpers shared by the distance kernels
// (kgpu_dist.cu: link-obstacle and link-link distances; kgpu_geom.cu:
// distances between two free geometries).  Values only: the closest
// features and the reported distances always come from the canonical FP64
// arithmetic of include/kgpu_exact.h; these FP32 values prune and select
// candidates, with the error bands their callers add.
#pragma once

#include <cfloat>
#include <climits>

#include "kgpu_device.cuh"

namespace kgpu {

__device__ __forceinline__ float box_dist32(const Box32& A, float3 c, float3 h)
{
  float gx = fmaxf(0.f, fabsf(A.c.x - c.x) - A.h.x - h.x);
  float gy = fmaxf(0.f, fabsf(A.c.y - c.y) - A.h.y - h.y);
  float gz = fmaxf(0.f, fabsf(A.c.z - c.z) - A.h.z - h.z);
  return root_below32(gx * gx + gy * gy + gz * gz);
}

__device__ __forceinline__ float warp_min(float v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---- FP32 triangle distance (value only; features come from FP64) --------
// The parameters use the fast reciprocal divide (__fdividef): a parameter off
// by a few ulp moves the evaluated points along their segments by a few ulp of
// the edge length, well inside the 128 u x span band the callers allow for the
// FP32 value (at an interior optimum the error is even second order).
__device__ __forceinline__ float clamp01f(float x) { return fminf(1.f, fmaxf(0.f, x)); }

static __device__ float seg_seg2_32(float3 p1, float3 d1, float3 p2, float3 d2)
{
  const float3 r = sub3(p1, p2);
  const float a = dot3(d1, d1), e = dot3(d2, d2), f = dot3(d2, r);
  float s, t;
  if (a <= 1e-30f && e <= 1e-30f) {
    s = 0.f; t = 0.f;
  } else if (a <= 1e-30f) {
    s = 0.f; t = clamp01f(__fdividef(f, e));
  } else {
    const float c = dot3(d1, r);
    if (e <= 1e-30f) {
      t = 0.f; s = clamp01f(__fdividef(-c, a));
    } else {
      const float b = dot3(d1, d2);
      const float den = a * e - b * b;
      s = den > 0.f ? clamp01f(__fdividef(b * f - c * e, den)) : 0.f;
      t = __fdividef(b * s + f, e);
      if (t < 0.f) { t = 0.f; s = clamp01f(__fdividef(-c, a)); }
      else if (t > 1.f) { t = 1.f; s = clamp01f(__fdividef(b - c, a)); }
    }
  }
  const float3 w = make_float3(r.x + d1.x * s - d2.x * t, r.y + d1.y * s - d2.y * t, r.z + d1.z * s - d2.z * t);
  return dot3(w, w);
}

// The callers take the value with its band as an upper bound.  So the foot is
// a point of the triangle whatever its shape (weights clamped: a sliver's are
// rounding noise), and it is formed relative to the vertices, never in world
// coordinates: its rounding then scales with the span, as the band does, not
// with the distance from the origin (a 0.1 mm triangle at 0.3 m was off by up
// to 2e-8 beyond that band).
static __device__ float pt_tri2_32(float3 p, float3 a, float3 b, float3 c)
{
  const float3 ab = sub3(b, a), ac = sub3(c, a), ap = sub3(p, a);
  const float d1 = dot3(ab, ap), d2 = dot3(ac, ap);
  float3 w;  // p - foot
  if (d1 <= 0.f && d2 <= 0.f) { w = ap; goto done; }
  {
    const float3 bp = sub3(p, b);
    const float d3 = dot3(ab, bp), d4 = dot3(ac, bp);
    if (d3 >= 0.f && d4 <= d3) { w = bp; goto done; }
    const float vc = d1 * d4 - d3 * d2;
    if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) {
      const float v = __fdividef(d1, d1 - d3);
      w = make_float3(ap.x - ab.x * v, ap.y - ab.y * v, ap.z - ab.z * v);
      goto done;
    }
    const float3 cp = sub3(p, c);
    const float d5 = dot3(ab, cp), d6 = dot3(ac, cp);
    if (d6 >= 0.f && d5 <= d6) { w = cp; goto done; }
    const float vb = d5 * d2 - d1 * d6;
    if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) {
      const float t = __fdividef(d2, d2 - d6);
      w = make_float3(ap.x - ac.x * t, ap.y - ac.y * t, ap.z - ac.z * t);
      goto done;
    }
    const float va = d3 * d6 - d5 * d4;
    if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f) {
      const float t = __fdividef(d4 - d3, (d4 - d3) + (d5 - d6));
      w = make_float3(bp.x - (c.x - b.x) * t, bp.y - (c.y - b.y) * t, bp.z - (c.z - b.z) * t);
      goto done;
    }
    const float den = __fdividef(1.f, va + vb + vc);
    const float v = clamp01f(vb * den), t = fminf(clamp01f(vc * den), 1.f - v);
    w = make_float3(ap.x - (ab.x * v + ac.x * t), ap.y - (ab.y * v + ac.y * t), ap.z - (ab.z * v + ac.z * t));
  }
done:
  return dot3(w, w);
}

// squared distance of two separated triangles: 9 edge-edge + 6 vertex-face.
// The vertices come by value: through pointers they live in local memory, which
// the loops' selections then read over and over (the distance kernels' L1, cut
// short by their shared memory, missed 4 of 5 of those loads).
static __device__ __noinline__ float tri_dist2_32(float3 P0, float3 P1, float3 P2, float3 Q0, float3 Q1, float3 Q2)
{
  float best = FLT_MAX;
#pragma unroll 1
  for (int k = 0; k < 9; ++k) {
    const int i = k / 3, j = k % 3;
    const float3 pa = sel3(i, P0, P1, P2), pb = sel3(i == 2 ? 0 : i + 1, P0, P1, P2);
    const float3 qa = sel3(j, Q0, Q1, Q2), qb = sel3(j == 2 ? 0 : j + 1, Q0, Q1, Q2);
    best = fminf(best, seg_seg2_32(pa, sub3(pb, pa), qa, sub3(qb, qa)));
  }
#pragma unroll 1
  for (int k = 0; k < 3; ++k) {
    best = fminf(best, pt_tri2_32(sel3(k, P0, P1, P2), Q0, Q1, Q2));
    best = fminf(best, pt_tri2_32(sel3(k, Q0, Q1, Q2), P0, P1, P2));
  }
  return best;
}

// ---- which features the canonical FP64 distance still has to look at --------
// kx_tri_tri_dist2 is the minimum over 15 features (9 edge-edge, 3 vertices of
// P against Q, 3 of Q against P; bit 3 i + j, 9 + k, 12 + k), taken in that
// order with strict comparisons (tri_dist2_masked64).  An FP64 operation
// occupies the SM for 19 cycles per warp whatever the number of active lanes, and all 15 features
// plus the 17 overlap axes are ~2,300 of them; in FP32 the features are a few
// hundred full-rate instructions.  Measured (before -> after): 8,192 humanoid
// self distances 28.4 -> 20.0 ms, soft-min over 6,400 waypoints 190.5 -> 140.1
// ms, 32,768 terrain clearances 47.9 -> 43.7 ms.  The mask keeps the features
// whose FP32 squared distance is at most thr2 (the caller's upper bound on the pair's
// minimum with its bands); the dropped ones cannot be the minimum.
//
// An FP32 feature value exceeds the feature's exact one by the placement and
// evaluation bands (in thr2) and by the error of the FP32 parameters.  For
// edges with den >= 1e-3 a e the parameter s is off by at most
// 8u 10^3 (r / sqrt(a) + 1), which raises the squared distance by at most
// a ds^2 <= 2.3e-7 (r + sqrt(a))^2 < 2e-6 span^2; for a vertex and a triangle
// of |n|^2 >= 0.01 L^4 (L its longest edge) the foot moves by at most
// min(L, 6u p^2 / (0.01 L)), p <= span, within 2e-5 span^2 as well.  thr2
// includes 2e-5 span^2; features worse conditioned than that are always kept.
// kFeatFlat is set when a triangle has no area: the canonical overlap test can
// report a contact of such triangles that are apart (its axes vanish), so the
// pair is left to the whole canonical function.
static __device__ __noinline__ unsigned tri_feature_mask32(float3 P0, float3 P1, float3 P2, float3 Q0, float3 Q1,
                                                              float3 Q2, float thr2)
{
  unsigned mask = 0;
#pragma unroll 1
  for (int k = 0; k < 9; ++k) {
    const int i = k / 3, j = k % 3;
    const float3 pa = sel3(i, P0, P1, P2), pb = sel3(i == 2 ? 0 : i + 1, P0, P1, P2);
    const float3 qa = sel3(j, Q0, Q1, Q2), qb = sel3(j == 2 ? 0 : j + 1, Q0, Q1, Q2);
    const float3 d1 = sub3(pb, pa), d2 = sub3(qb, qa);
    const float a = dot3(d1, d1), e = dot3(d2, d2), b = dot3(d1, d2);
    if (!(a * e - b * b >= 1e-3f * a * e) || !(seg_seg2_32(pa, d1, qa, d2) > thr2)) mask |= 1u << k;
  }
#pragma unroll 1
  for (int t = 0; t < 2; ++t) {
    // t = 0: vertices of P against Q, t = 1: vertices of Q against P
    const float3 a = t ? P0 : Q0, b = t ? P1 : Q1, c = t ? P2 : Q2;
    const float3 ab = sub3(b, a), ac = sub3(c, a), bc = sub3(c, b);
    const float3 n = cross3(ab, ac);
    const float L2 = fmaxf(dot3(ab, ab), fmaxf(dot3(ac, ac), dot3(bc, bc)));
    const float n2 = dot3(n, n);
    const bool thin = !(n2 >= 0.01f * L2 * L2);
    if (!(n2 > 1e-8f * L2 * L2)) mask |= kFeatFlat;  // (a single point too)
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
      const float3 p = t ? sel3(k, Q0, Q1, Q2) : sel3(k, P0, P1, P2);
      if (thin || !(pt_tri2_32(p, a, b, c) > thr2)) mask |= 1u << (9 + 3 * t + k);
    }
  }
  return mask;
}

// The threshold of tri_feature_mask32: m32 bounds the pair's minimum up to
// the placement bound `place` and the evaluation band of this triangle pair.
__device__ __forceinline__ float feature_thr2(const float3* P, const float3* Q, float m32, float place)
{
  float3 lo = P[0], hi = P[0];
#pragma unroll
  for (int k = 1; k < 6; ++k) {
    const float3 v = k < 3 ? P[k] : Q[k - 3];
    lo = make_float3(fminf(lo.x, v.x), fminf(lo.y, v.y), fminf(lo.z, v.z));
    hi = make_float3(fmaxf(hi.x, v.x), fmaxf(hi.y, v.y), fmaxf(hi.z, v.z));
  }
  const float span = fmaxf(fmaxf(hi.x - lo.x, hi.y - lo.y), hi.z - lo.z);
  const float thr = m32 * (1.f + 2e-5f) + 2.f * (place + 128.f * kU * span) + 1e-6f;
  return thr * thr * (1.f + 1e-5f) + 2e-5f * span * span;  // (FLT_MAX bounds overflow to inf: every feature kept)
}

// Non-negative doubles compare like their bits (integer instructions: an FP64
// comparison occupies the SM for 19 cycles)
__device__ __forceinline__ unsigned long long double_bits(double d) { return (unsigned long long)__double_as_longlong(d); }

// lexicographic (d2, a, b) minimum across the warp, d2 as double_bits; result
// in every lane
__device__ __forceinline__ void warp_lexmin(unsigned long long& d2, int& a, int& b, int& src, int lane)
{
  src = lane;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long od = __shfl_xor_sync(0xffffffffu, d2, o);
    const int oa = __shfl_xor_sync(0xffffffffu, a, o);
    const int ob = __shfl_xor_sync(0xffffffffu, b, o);
    const int os = __shfl_xor_sync(0xffffffffu, src, o);
    const bool take = od < d2 || (od == d2 && (oa < a || (oa == a && (ob < b || (ob == b && os < src)))));
    if (take) { d2 = od; a = oa; b = ob; src = os; }
  }
}

// Lower bound on the distance of two triangles from the separating direction
// through their centroids (projections onto a unit vector are 1-Lipschitz);
// nearly tight for facing triangles, which the box bound is not.  The FP32
// rounding of the centroids, the normalisation (rsqrtf: 2 ulp) and the
// projections is covered by the (1 - 16u) factor and the 16 u span term.
__device__ __forceinline__ float tri_axis_lb32(const float3* P, const float3* Q, float span)
{
  const float k3 = 1.f / 3.f;
  const float3 cP = make_float3((P[0].x + P[1].x + P[2].x) * k3, (P[0].y + P[1].y + P[2].y) * k3,
                                (P[0].z + P[1].z + P[2].z) * k3);
  const float3 cQ = make_float3((Q[0].x + Q[1].x + Q[2].x) * k3, (Q[0].y + Q[1].y + Q[2].y) * k3,
                                (Q[0].z + Q[1].z + Q[2].z) * k3);
  float3 u = sub3(cQ, cP);
  const float nn = dot3(u, u);
  if (!(nn > 1e-30f)) return 0.f;
  const float inv = rsqrtf(nn);
  u = make_float3(u.x * inv, u.y * inv, u.z * inv);
  float pm = -FLT_MAX, qm = FLT_MAX;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    pm = fmaxf(pm, dot3(sub3(P[k], cP), u));
    qm = fminf(qm, dot3(sub3(Q[k], cP), u));
  }
  return (qm - pm) * (1.f - 16.f * kU) - 16.f * kU * span;
}

}  // namespace kgpu
