// The ray-triangle tests: Moller-Trumbore in float with a forward error bound,
// and the reference's in double, operation by operation.
#pragma once

#include <cuda_runtime.h>

namespace skw {
namespace {

// Forward error bound of the float triangle test: with u = 2^-24, the edge
// and offset vectors carry <= u relative error, the cross products <= 4u of
// their magnitude sums, and det, n1, n2, nt <= 8u of the matching
// magnitude dot products (first order); 10u leaves room for the second-order
// terms and for the bounds being evaluated in float.  A double ray rounded
// to float (d by u relative, o by u |o|) moves the cross product with d by
// another u of its magnitude sum and the offset o - v0 by u (|o| + |o - v0|)
// instead of u |o - v0|: with |o - v0| + |o| in the magnitude sums 12u covers
// every term (9u to first order).
//
// A double ray's test decides the same as the double test at any scale, so
// what a float rounds in its subnormal range is bounded too: by g / 2 an
// operation (g = 2^-149), whatever the operands.  With S1 = |e1| + |e2| summed
// over the components and S = 1 + S1 + sum |o - v0| + sum |o| + sum |d|: d's
// and o's own rounding and two products move a cross product by at most
// g (1 + S1), the dot product with it adds 2g, and the other operand's rounding
// g / 2 times the other cross product, so that det, n1, n2 and nt are off by
// at most 3g (1 + S1) S.  Their bounds get 8g (1 + S1) S (tri_under, from the
// scene's largest coordinate B): the rest is for the roundings of the bounds
// themselves, in that range too.  (200,001 closest hits over 1.1M triangles,
// with the walk's guard for distances beyond a float: 539 us without, 556 with.)
constexpr float kTriErr = 10.0f * 5.9604645e-8f, kTriErrD = 12.0f * 5.9604645e-8f;
constexpr double kDblEps = 2.220446049250313e-16;

enum : int { kMiss = 0, kHit = 1, kAmbiguous = 2 };

struct RayF {
  float ox, oy, oz, dx, dy, dz, tmin, tmax;
};

// The subnormal range's part of a double ray's bounds (above); o, d: the sums
// of its origin's and direction's components' magnitudes.
__device__ __forceinline__ float tri_under(float scene_abs, float o, float d) {
  return 1.1210388e-44f * (1.0f + 12.0f * scene_abs) * (1.0f + 15.0f * scene_abs + 2.0f * o + d);  // 8 * 2^-149
}

// Float triangle test with a forward error bound.  Returns kMiss when the
// reference's double test certainly rejects (barycentrics or t < tmin),
// kHit when its barycentric tests and t >= tmin certainly pass (t and a bound
// et on |t - t_exact| are returned), else kAmbiguous.  ROUNDED: r is a double
// ray rounded to float (tmin down), and the bounds cover that rounding and what
// is rounded in the subnormal range (under: tri_under of the ray).
template <bool ROUNDED>
__device__ __forceinline__ int tri_test32(const RayF &r, float3 v0, float3 v1, float3 v2, float &t, float &et,
                                          float under = 0.0f) {
  t = __int_as_float(0x7fffffff);  // NaN until computed
  et = 0.0f;
  const float e1x = v1.x - v0.x, e1y = v1.y - v0.y, e1z = v1.z - v0.z;
  const float e2x = v2.x - v0.x, e2y = v2.y - v0.y, e2z = v2.z - v0.z;
  const float s1x = r.dy * e2z - r.dz * e2y;
  const float s1y = r.dz * e2x - r.dx * e2z;
  const float s1z = r.dx * e2y - r.dy * e2x;
  const float det = s1x * e1x + s1y * e1y + s1z * e1z;
  const float ddx = r.ox - v0.x, ddy = r.oy - v0.y, ddz = r.oz - v0.z;
  const float n1 = ddx * s1x + ddy * s1y + ddz * s1z;
  const float s2x = ddy * e1z - ddz * e1y;
  const float s2y = ddz * e1x - ddx * e1z;
  const float s2z = ddx * e1y - ddy * e1x;
  const float n2 = r.dx * s2x + r.dy * s2y + r.dz * s2z;
  const float nt = e2x * s2x + e2y * s2y + e2z * s2z;
  // Componentwise magnitude bounds of the cross products.
  const float adx = fabsf(r.dx), ady = fabsf(r.dy), adz = fabsf(r.dz);
  const float a2x = fabsf(e2x), a2y = fabsf(e2y), a2z = fabsf(e2z);
  const float a1x = fabsf(e1x), a1y = fabsf(e1y), a1z = fabsf(e1z);
  const float aox = ROUNDED ? fabsf(ddx) + fabsf(r.ox) : fabsf(ddx), aoy = ROUNDED ? fabsf(ddy) + fabsf(r.oy) : fabsf(ddy),
              aoz = ROUNDED ? fabsf(ddz) + fabsf(r.oz) : fabsf(ddz);
  constexpr float kErr = ROUNDED ? kTriErrD : kTriErr;
  const float A1x = ady * a2z + adz * a2y, A1y = adz * a2x + adx * a2z, A1z = adx * a2y + ady * a2x;
  const float A2x = aoy * a1z + aoz * a1y, A2y = aoz * a1x + aox * a1z, A2z = aox * a1y + aoy * a1x;
  const float D = fabsf(det);
  const float rest = ROUNDED ? 1e-15f * D + under : 1e-15f * D;
  const float edet = kErr * (a1x * A1x + a1y * A1y + a1z * A1z) + rest;
  const float en1 = kErr * (aox * A1x + aoy * A1y + aoz * A1z) + rest;
  const float en2 = kErr * (adx * A2x + ady * A2y + adz * A2z) + rest;
  const float et0 = kErr * (a2x * A2x + a2y * A2y + a2z * A2z), ent = ROUNDED ? et0 + under : et0;
  if (ROUNDED) {
    // (beyond 1e37 the reciprocal would be subnormal; below 8 bounds of det,
    // 1 / det's own error would not be covered by t's bound)
    if (!(D > 8.0f * edet && D < 1e37f)) return kAmbiguous;
  } else {
    if (!(D > 2.0f * edet)) return kAmbiguous;  // nearly parallel (or degenerate)
  }
  const float sgn = det < 0.0f ? -1.0f : 1.0f;
  const float N1 = sgn * n1, N2 = sgn * n2, NT = sgn * nt;
  if (N1 + en1 < 0.0f || N2 + en2 < 0.0f) return kMiss;
  if (N1 - en1 > D + edet) return kMiss;
  if ((N1 + N2) - (en1 + en2) > D + edet) return kMiss;
  const float inv = 1.0f / D;
  t = NT * inv;
  et = (ent + fabsf(t) * edet) * inv * 1.0001f + fabsf(t) * 2.4e-7f + 1e-30f;
  if (t + et < r.tmin) return kMiss;
  if (N1 - en1 > 0.0f && N2 - en2 > 0.0f && (N1 + N2) + (en1 + en2) < D - edet &&
      (ROUNDED ? t - et > r.tmin : t - et >= r.tmin))  // rounded: above tmin rounded down is above tmin
    return kHit;
  return kAmbiguous;
}

// A ray given in double (skw_ray_d): origin, direction, tmin, tmax.
struct RayD {
  double ox, oy, oz, dx, dy, dz, tmin, tmax;
};

// The reference's double-precision Moller-Trumbore test, operation by
// operation (TriangleAccelerator.cpp:240-273).  Intrinsics keep every
// product and sum separately rounded, as in the x86-64 SSE2 build.
__device__ __forceinline__ bool tri_test64v(double ox, double oy, double oz, double dx, double dy, double dz,
                                            float3 v0f, float3 v1f, float3 v2f, double tmin, double tmax,
                                            double &t_out) {
  const double v0x = v0f.x, v0y = v0f.y, v0z = v0f.z;
  const double e1x = __dsub_rn((double)v1f.x, v0x), e1y = __dsub_rn((double)v1f.y, v0y),
               e1z = __dsub_rn((double)v1f.z, v0z);
  const double e2x = __dsub_rn((double)v2f.x, v0x), e2y = __dsub_rn((double)v2f.y, v0y),
               e2z = __dsub_rn((double)v2f.z, v0z);
  const double s1x = __dsub_rn(__dmul_rn(dy, e2z), __dmul_rn(dz, e2y));
  const double s1y = __dsub_rn(__dmul_rn(dz, e2x), __dmul_rn(dx, e2z));
  const double s1z = __dsub_rn(__dmul_rn(dx, e2y), __dmul_rn(dy, e2x));
  const double divisor = __dadd_rn(__dadd_rn(__dmul_rn(s1x, e1x), __dmul_rn(s1y, e1y)), __dmul_rn(s1z, e1z));
  const double inv = __ddiv_rn(1.0, divisor);
  const double ddx = __dsub_rn(ox, v0x), ddy = __dsub_rn(oy, v0y), ddz = __dsub_rn(oz, v0z);
  const double b1 =
      __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(ddx, s1x), __dmul_rn(ddy, s1y)), __dmul_rn(ddz, s1z)), inv);
  if (b1 > -kDblEps && b1 < (1.0 + kDblEps)) {
    const double s2x = __dsub_rn(__dmul_rn(ddy, e1z), __dmul_rn(ddz, e1y));
    const double s2y = __dsub_rn(__dmul_rn(ddz, e1x), __dmul_rn(ddx, e1z));
    const double s2z = __dsub_rn(__dmul_rn(ddx, e1y), __dmul_rn(ddy, e1x));
    const double b2 =
        __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, s2x), __dmul_rn(dy, s2y)), __dmul_rn(dz, s2z)), inv);
    if (b2 > -kDblEps && __dadd_rn(b1, b2) < (1.0 + kDblEps)) {
      const double t =
          __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(e2x, s2x), __dmul_rn(e2y, s2y)), __dmul_rn(e2z, s2z)), inv);
      if (t >= tmin && t <= tmax) {
        t_out = t;
        return true;
      }
    }
  }
  return false;
}

}  // namespace
}  // namespace skw
