// Closest-hit and any-hit traversal of the ternary bbox kd-tree on sm_103a.
//
// Semantics follow TriangleAccelerator::_NodeIntersect / _NodeIntersectTest
// (Raytracer/Core/TriangleAccelerator.cpp:154-293, 354-462):
//   * a stack of nodes; each popped node's AABB is tested against the ray's
//     [tmin, current tmax] with the reference's twelve slab comparisons;
//   * an internal node pushes its present children so that the child on the
//     ray's near side of the split axis is popped first;
//   * a leaf tests its triangles in order with Moller-Trumbore; a hit with
//     tmin <= t <= current tmax replaces the current one (so among exactly
//     equal t the last tested triangle wins) and becomes the new tmax.
//
// The reference does all of this in double precision over float data.  Here
// the node tests run in float: a plane distance is fma(coordinate, 1/d,
// -o/d -+ w) with the per-ray absolute widening w = 6u (B + |o|) |1/d|
// (u = 2^-24, B = the scene's largest absolute coordinate; see SlabRay),
// which bounds the float error for every node, so a node is culled only if
// the reference culls it too.  The triangle test runs in float with a
// forward error bound on every quantity; only when a decision
// (inside/outside an edge, t inside [tmin, tmax], which of two hits is
// nearer) falls inside that bound is the triangle re-tested with the
// reference's exact double-precision arithmetic (round-to-nearest
// intrinsics, no fused multiply-add).  Such hits are flagged
// SKW_HIT_FP64_DECIDED.
//
// Layout: nodes are 32-byte DevNode records, one 32-byte load each; a
// triangle slot is 3 x float4 (v0|prim, v1|tri, v2|slot); rays are 2 x float4.
// The traversal stack holds 12-byte entries (node words 6-7 and the widened
// entry distance): the first SKW_TRAV_SCAP (8) of each thread in shared
// memory, deeper ones in local memory.  Its capacity CAP is chosen on the
// host as >= 2 * tree depth + 1, which bounds its use (at most two entries
// are pushed per level).
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <mutex>
#include <unordered_map>

#include "accel_build.h"
#include "kernels.h"
#include "tri_test.cuh"

namespace skw {
namespace {

// Launch shape: threads per block and the minimum resident blocks per SM
// that bounds the register budget.  Six blocks (80 registers) leave the node
// step without spills: measured on 4,194,304 closest hits over 1.1M triangles
// with 10 / 8 / 7 / 6 / 5 / 4 blocks per SM: 4.00 / 3.85 / 3.82 / 3.69 / 3.77
// / 4.42 ms, on 1,000 rays: 98 / 88 / 79 / 77 / 73 / 77 us.
#ifndef SKW_TRAV_BLOCK
#define SKW_TRAV_BLOCK 128
#endif
#ifndef SKW_TRAV_MINB
#define SKW_TRAV_MINB 6
#endif

// Rays and results stream through once: with SKW_TRAV_STREAMING they are
// loaded and stored with the evict-first policy so that they do not push the
// tree out of L2.
#ifndef SKW_TRAV_STREAMING
#define SKW_TRAV_STREAMING 1
#endif
#if SKW_TRAV_STREAMING
#define SKW_LD_STREAM(p) __ldcs(p)
#define SKW_ST_STREAM(p, v) __stcs(p, v)
#else
#define SKW_LD_STREAM(p) __ldg(p)
#define SKW_ST_STREAM(p, v) (*(p) = (v))
#endif

__device__ __forceinline__ RayF load_ray(const float4 *__restrict__ rays, int64_t i) {
  const float4 a = SKW_LD_STREAM(rays + 2 * i);
  const float4 b = SKW_LD_STREAM(rays + 2 * i + 1);
  return RayF{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
}

__device__ __forceinline__ RayD load_ray_d(const float4 *__restrict__ rays, int64_t i) {
  const double2 *p = reinterpret_cast<const double2 *>(rays) + 4 * i;
  const double2 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2), d = __ldg(p + 3);
  return RayD{a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y};
}

__device__ __forceinline__ void load_tri(const float4 *__restrict__ tris, uint32_t slot, float3 &v0, float3 &v1,
                                         float3 &v2, int &prim, int &tri) {
  const float4 a = __ldg(tris + 3 * slot);
  const float4 b = __ldg(tris + 3 * slot + 1);
  const float4 c = __ldg(tris + 3 * slot + 2);
  v0 = make_float3(a.x, a.y, a.z);
  v1 = make_float3(b.x, b.y, b.z);
  v2 = make_float3(c.x, c.y, c.z);
  prim = __float_as_int(a.w);
  tri = __float_as_int(b.w);
}

// Per-ray data for the slab test.  A plane distance is computed as
// fma(coordinate, 1/d, offset) with the offset -o/d -+ w folded in, where the
// per-axis widening w = 6u (B + |o|) |1/d| (u = 2^-24, B = largest absolute
// coordinate in the scene) bounds the float result's distance from the exact
// value for every node of the scene; the reference's double result is within
// a far smaller distance of the exact one.  The near plane of each axis is
// selected by the sign of 1/d, which is the reference's "swap if
// tNear > tFar" for every non-NaN slab.  Together with tmin, tmax and the
// near-child side of each axis this is all the node walk needs, so the
// ray's origin and direction can stay out of registers while it runs.
struct SlabRay {
  float ix, iy, iz;  // 1/d
  float nx, ny, nz;  // near-plane offsets: -o/d - w
  float fx, fy, fz;  // far-plane offsets:  -o/d + w
  float tmin, tmax;
  // bits 0-2: !(d[axis] > 0), the reference pops the right child first;
  // bits 3-5: 1/d[axis] < 0, the near plane is the box maximum
  uint32_t bits;
};

// The widening is 6u for a float ray; 9u for a double ray rounded to float
// (ROUNDED), whose rounding moves a plane distance by at most
// u |o| |1/d| (origin) + u |b - o| |1/d| (direction) more, and whose plane
// distances, beyond a float's range on an axis, leave that axis out.
template <bool ROUNDED>
__device__ __forceinline__ SlabRay make_slab_ray(const RayF &r, float scene_abs) {
  SlabRay s;
  s.ix = 1.0f / r.dx;
  s.iy = 1.0f / r.dy;
  s.iz = 1.0f / r.dz;
  constexpr float c = (ROUNDED ? 9.0f : 6.0f) * 5.9604645e-8f;
  const float wx = c * (scene_abs + fabsf(r.ox)) * fabsf(s.ix);
  const float wy = c * (scene_abs + fabsf(r.oy)) * fabsf(s.iy);
  const float wz = c * (scene_abs + fabsf(r.oz)) * fabsf(s.iz);
  const float ox = -r.ox * s.ix, oy = -r.oy * s.iy, oz = -r.oz * s.iz;
  s.nx = ox - wx;
  s.ny = oy - wy;
  s.nz = oz - wz;
  s.fx = ox + wx;
  s.fy = oy + wy;
  s.fz = oz + wz;
  constexpr float most = c * 1.0e38f;  // the distances are within w / c
  if (ROUNDED && !(wx + wy + wz < most)) {
    const float inf = __int_as_float(0x7f800000);
    if (!(wx < most)) s.ix = 0.0f, s.nx = -inf, s.fx = inf;
    if (!(wy < most)) s.iy = 0.0f, s.ny = -inf, s.fy = inf;
    if (!(wz < most)) s.iz = 0.0f, s.nz = -inf, s.fz = inf;
  }
  s.tmin = r.tmin;
  s.tmax = r.tmax;
  s.bits = (r.dx > 0.0f ? 0u : 1u) | (r.dy > 0.0f ? 0u : 2u) | (r.dz > 0.0f ? 0u : 4u) |
           (signbit(s.ix) ? 8u : 0u) | (signbit(s.iy) ? 16u : 0u) | (signbit(s.iz) ? 32u : 0u);
  return s;
}

// The reference's slab test (TriangleAccelerator.cpp:176-192) on the widened
// interval: true when the node must be visited.  `lo` receives the widened
// entry distance max(tnear_x, tnear_y, tnear_z, tmin), all that a later
// re-test against a smaller tmax needs.  fmaxf/fminf drop NaN operands
// (0 * inf slabs), as the reference's comparisons are all false on NaN.
__device__ __forceinline__ bool node_visit(const float4 na, const float4 nb, const SlabRay &s, float tcull,
                                           float &lo) {
  const bool sx = s.bits & 8u, sy = s.bits & 16u, sz = s.bits & 32u;
  const float tn0 = fmaf(sx ? na.w : na.x, s.ix, s.nx), tf0 = fmaf(sx ? na.x : na.w, s.ix, s.fx);
  const float tn1 = fmaf(sy ? nb.x : na.y, s.iy, s.ny), tf1 = fmaf(sy ? na.y : nb.x, s.iy, s.fy);
  const float tn2 = fmaf(sz ? nb.y : na.z, s.iz, s.nz), tf2 = fmaf(sz ? na.z : nb.y, s.iz, s.fz);
  lo = fmaxf(fmaxf(tn0, tn1), fmaxf(tn2, s.tmin));
  const float hi = fminf(fminf(tf0, tf1), fminf(tf2, tcull));
  return !(lo > hi);
}

#ifndef SKW_TRAV_SCAP
#define SKW_TRAV_SCAP 8
#endif
#ifndef SKW_TRAV_REFILL
#define SKW_TRAV_REFILL 8
#endif
// A walk round ends once at most SKW_TRAV_LAG walking lanes still have no
// leaf; those keep their place and go on walking in the next round.
#ifndef SKW_TRAV_LAG
#define SKW_TRAV_LAG 12
#endif
// Traversal stack: the first SCAP entries of each thread live in shared
// memory as arrays indexed [entry][thread] (so lanes never conflict on a
// bank), deeper entries in local memory.  An entry holds a node's words 6-7
// and its widened entry distance.
template <int CAP>
struct Stack {
  static constexpr int SCAP = CAP < SKW_TRAV_SCAP ? CAP : SKW_TRAV_SCAP;
  uint2 (*sw)[SKW_TRAV_BLOCK];
  float (*slo)[SKW_TRAV_BLOCK];
  uint4 ovf[CAP - SCAP > 0 ? CAP - SCAP : 1];
  int sp;

  __device__ __forceinline__ void push(uint32_t a, uint32_t b, float lo, unsigned *status) {
    if (sp < SCAP) {
      sw[sp][threadIdx.x] = make_uint2(a, b);
      slo[sp][threadIdx.x] = lo;
    } else if (sp < CAP) {
      ovf[sp - SCAP] = make_uint4(a, b, __float_as_uint(lo), 0u);
    } else {
      atomicOr(status, 1u);  // never: CAP covers the tree's depth
      return;
    }
    ++sp;
  }
  // Pops until an entry survives the re-cull against tcull (the reference
  // culls the others when it pops them).  A ray that has just found its hit
  // drops most of its stack here, usually on its own in the warp, so the
  // loop over the shared entries reads nothing but their distances.
  __device__ __forceinline__ bool pop(float tcull, uint32_t &a, uint32_t &b, float &lo) {
    while (sp > SCAP) {
      --sp;
      const uint4 e = ovf[sp - SCAP];
      a = e.x;
      b = e.y;
      lo = __uint_as_float(e.z);
      if (!(lo > tcull)) return true;
    }
    while (sp > 0) {
      --sp;
      lo = slo[sp][threadIdx.x];
      if (!(lo > tcull)) {
        const uint2 e = sw[sp][threadIdx.x];
        a = e.x;
        b = e.y;
        return true;
      }
    }
    return false;
  }
};

// A 32-byte node (32-byte aligned) in one load.
__device__ __forceinline__ void load_node(const float4 *__restrict__ nodes, uint32_t i, float4 &a, float4 &b) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(nodes + 2 * (size_t)i));
}

// Expands the internal node (cur_a, cur_b): box-tests its present children,
// makes the first passing one (in the reference's pop order) current and
// pushes the others; false when none passes.  cur_lo is the current node's
// widened entry distance.
//
// Visit order equals the reference's (TriangleAccelerator.cpp:170-211): the
// reference pushes an internal node's children and pops the near-side one
// first, testing each node's box when it is popped.  Here the present
// children (contiguous) are box-tested right away.  A pushed entry keeps its
// widened entry distance and is re-culled on pop against the tmax of that
// moment -- the only part of the reference's pop-time test that can change
// after the push, since tmax only shrinks.
template <int CAP>
__device__ __forceinline__ bool expand(const float4 *__restrict__ nodes, const SlabRay &s, float tcull,
                                       Stack<CAP> &st, uint32_t &cur_a, uint32_t &cur_b, float &cur_lo,
                                       unsigned *status) {
  const uint32_t type = cur_b & 3u, mask = (cur_b >> 2) & 7u;
  const bool near_right = (s.bits >> (type - 1u)) & 1u;  // the reference pops left first when d[axis] > 0
  const uint32_t sL = cur_a, sM = cur_a + (mask & 1u), sR = sM + ((mask >> 1) & 1u);
  // far, middle, near: the reverse of the pop order
  const uint32_t slot[3] = {near_right ? sL : sR, sM, near_right ? sR : sL};
  const bool present[3] = {(mask & (near_right ? 1u : 4u)) != 0u, (mask & 2u) != 0u,
                           (mask & (near_right ? 4u : 1u)) != 0u};
  bool have = false;
  float4 ca[3], cb[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) load_node(nodes, present[k] ? slot[k] : sL, ca[k], cb[k]);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float lo;
    if (node_visit(ca[k], cb[k], s, tcull, lo) && present[k]) {
      if (have) st.push(cur_a, cur_b, cur_lo, status);
      have = true;
      cur_a = __float_as_uint(cb[k].z);
      cur_b = __float_as_uint(cb[k].w);
      cur_lo = lo;
    }
  }
  return have;
}

// The exact (double) decisions of a lane's ray.  They are out of line and
// read the ray and the triangles from memory again, so that the walk's
// registers are not laid out around their double temporaries: inline, the
// kernel spilled in its hot loop.
template <bool DRAY>
__device__ __forceinline__ RayD exact_ray(const float4 *__restrict__ rays, int ray_i) {
  if (DRAY) return load_ray_d(rays, ray_i);
  const RayF r = load_ray(rays, ray_i);
  return RayD{r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, r.tmin, r.tmax};
}

__device__ __forceinline__ bool tri_test64(const float4 *__restrict__ tris, const RayD &r, int slot, double tmax,
                                           double &t_out) {
  const float4 a = __ldg(tris + 3 * slot), b = __ldg(tris + 3 * slot + 1), c = __ldg(tris + 3 * slot + 2);
  return tri_test64v(r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, make_float3(a.x, a.y, a.z), make_float3(b.x, b.y, b.z),
                     make_float3(c.x, c.y, c.z), r.tmin, tmax, t_out);
}

// t of the hit on slot `slot` (its barycentric tests are known to pass).
template <bool DRAY>
__device__ __noinline__ double exact_t(const float4 *__restrict__ tris, const float4 *__restrict__ rays, int ray_i,
                                       int slot, float fallback) {
  double t;
  return tri_test64(tris, exact_ray<DRAY>(rays, ray_i), slot, 1.0e308, t) ? t : (double)fallback;
}

// Whether the triangle in `slot` is hit no farther than the current tmax:
// the ray's own (best < 0) or the t of the best hit so far.  On a hit lo / hi
// bracket its t and `flags` has bit 0 set, and bit 1 where the two t are
// within 1e-12 relative; no hit: flags = 0.
struct ExactHit {
  float lo, hi;
  uint32_t flags;
};
template <bool DRAY>
__device__ __noinline__ ExactHit exact_hit(const float4 *__restrict__ tris, const float4 *__restrict__ rays, int ray_i,
                                           int slot, int best, float fallback) {
  const RayD r = exact_ray<DRAY>(rays, ray_i);
  double cur_max = r.tmax, t;
  if (best >= 0) cur_max = tri_test64(tris, r, best, 1.0e308, t) ? t : (double)fallback;
  if (!tri_test64(tris, r, slot, cur_max, t)) return ExactHit{0.0f, 0.0f, 0u};
  return ExactHit{__double2float_rd(t), __double2float_ru(t),
                  best >= 0 && fabs(t - cur_max) <= 1e-12 * fabs(t) ? 3u : 1u};
}

// Persistent traversal.  The rays form groups of consecutive rays; a warp
// takes the launch's next group from the launch's counter (`work`, one
// atomicAdd per group) when its current group is used up, and a lane whose
// ray is finished takes the next ray of the warp's group when at least
// SKW_TRAV_REFILL lanes are idle (or all are), so lanes rarely idle while
// long rays finish and warps that drew cheap rays take more.  A finished
// lane keeps its result until then, so that the results of several lanes
// are written together.  No cross-warp waits.
//
// Closest-hit state is kept small: the slot of the current best hit and a
// float interval [lo_t, hi_t] that contains the reference's current tmax
// (the best hit's double t).  Where a decision needs that tmax exactly, it is
// recomputed from the slot with the exact test.
//
// surf: the rays leave surfaces with tmin from next_min_t (the renders'
// shadow, BSDF, specular and gather rays, photon bounces).
//
// DRAY: the rays are skw_ray_d (double).  The walk and the triangle tests
// run on the ray rounded to float (origin and direction to nearest, tmin
// down, tmax up) with the bounds of make_slab_ray and tri_test32 for rounded
// rays, so a node is still culled only if the reference culls it and a
// triangle is decided in float only where the double test decides the same;
// the rest is decided on the double ray (read again from memory).
// Closest-hit results are skw_hit_d (the exact double t, prim, tri).
//
// What bounds it: the latency of the divergent walk (ncu, 1M closest hits:
// 0.49 instructions issued per cycle and scheduler, 42 % of the stalls on node
// loads, 11 of 32 lanes, L1 at 57 % of its peak, DRAM at 2 %).  What the shape of the step is
// for, measured on 4,194,304 closest / 2,000,003 any hits over 1.1M triangles
// (3.99 / 1.71 ms before): one place that pops, children loaded and tested
// without branches, one 32-byte load per node and no spills in the step:
// 3.47 / 1.33 ms.  200,001 double rays: 3.25 -> 0.53 ms with the float
// decisions (87 % of the kernel was double triangle tests), 0.55 with bounds that
// hold at any scale.
template <int CAP, bool CLOSEST, bool DRAY>
__global__ void __launch_bounds__(SKW_TRAV_BLOCK, SKW_TRAV_MINB)
    k_trace(const float4 *__restrict__ nodes, const float4 *__restrict__ tris, const float4 *__restrict__ rays,
            int n, const int *__restrict__ n_dev, float scene_abs, const int32_t *__restrict__ out_index,
            void *__restrict__ out, unsigned *__restrict__ status, unsigned *__restrict__ work, int surf,
            unsigned long long *__restrict__ traced) {
  if (n_dev) n = min(n, *n_dev);  // a queue whose length lives on the device
  if (traced && blockIdx.x == 0 && threadIdx.x == 0 && n > 0) atomicAdd(traced, (unsigned long long)n);
  constexpr int SCAP = Stack<CAP>::SCAP;
  __shared__ uint2 s_w[SCAP][SKW_TRAV_BLOCK];
  __shared__ float s_lo[SCAP][SKW_TRAV_BLOCK];
  Stack<CAP> st;
  st.sw = s_w;
  st.slo = s_lo;
  st.sp = 0;

  const unsigned lane = threadIdx.x & 31u;
  // Rays per group: 32, or fewer where that leaves warps of the grid without
  // rays (see the launch).
  const int n_warps = (int)(gridDim.x * (unsigned)(SKW_TRAV_BLOCK / 32));
  const int group = (int)min(32u, max(1u, ((unsigned)n + (unsigned)n_warps - 1u) / (unsigned)n_warps));
  // next / end are positions in the current group [gbase, gbase + group);
  // end = -1 once the rays are gone.
  int next = 0, end = 0;
  unsigned gbase = 0;

  int ray_i = -1;    // the lane's ray
  bool fin = true;   // its walk is over; its result waits while ray_i >= 0
  bool hit = false;  // any hit: the result
  RayF r{};          // read only by the triangle tests
  uint32_t cur_a = 0, cur_b = 0;
  float cur_lo = 0.0f;
  int best_slot = -1;
  float lo_t = 0.0f, hi_t = 0.0f;  // bracket of the reference's current tmax
  uint32_t flags = 0;              // SKW_HIT_* bits; bit 3: [lo_t, hi_t] brackets an exact double

  while (true) {
    const unsigned idle = __ballot_sync(0xffffffffu, fin);
    if (idle != 0u && (__popc(idle) >= SKW_TRAV_REFILL || idle == 0xffffffffu)) {
      // the finished lanes' results
      if (fin && ray_i >= 0) {
        const int o = out_index ? SKW_LD_STREAM(out_index + ray_i) : ray_i;
        if (!CLOSEST) {
          ((uint8_t *)out)[o] = hit ? 1 : 0;
        } else {
          int4 h = DRAY ? make_int4(0, 0x7ff00000, -1, -1)  // t = +inf, a miss
                        : make_int4(0x7f800000, -1, -1, (int)(flags & 7u));
          if (best_slot >= 0) {
            const int prim = __float_as_int(__ldg(tris + 3 * best_slot).w),
                      tri = __float_as_int(__ldg(tris + 3 * best_slot + 1).w);
            float tout = 0.5f * lo_t + 0.5f * hi_t;
            if (DRAY) {
              const long long t64 =
                  __double_as_longlong(exact_t<DRAY>(tris, rays, ray_i, best_slot, tout));
              h = make_int4((int)(t64 & 0xffffffffll), (int)(t64 >> 32), prim, tri);
            } else {
              // A float-decided hit whose bracket is wider than the 1e-5 reporting
              // tolerance (grazing incidence) takes t from the exact test.
              if (!(flags & 8u) && hi_t - lo_t > 1.0e-5f * fabsf(tout)) {
                tout = (float)exact_t<DRAY>(tris, rays, ray_i, best_slot, tout);
                flags |= 4u;
              }
              h = make_int4(__float_as_int(tout), prim, tri, (int)(flags & 7u));
            }
          }
          SKW_ST_STREAM((int4 *)out + o, h);
        }
        ray_i = -1;
      }
      // new rays
      if (end >= 0 && next >= end) {
        if (lane == 0) gbase = atomicAdd(work, (unsigned)group);
        gbase = __shfl_sync(0xffffffffu, gbase, 0);
        next = 0;
        end = gbase < (unsigned)n ? min(group, n - (int)gbase) : -1;
      }
      if (next < end) {
        const int mine = next + __popc(idle & ((1u << lane) - 1u));
        next += __popc(idle);
        if (fin && mine < end) {
          ray_i = (int)gbase + mine;
          if (DRAY) {
            const RayD rd = load_ray_d(rays, ray_i);
            r = RayF{(float)rd.ox, (float)rd.oy, (float)rd.oz, (float)rd.dx, (float)rd.dy, (float)rd.dz,
                     __double2float_rd(rd.tmin), __double2float_ru(rd.tmax)};
            lo_t = __double2float_rd(rd.tmax);
          } else {
            r = load_ray(rays, ray_i);
            lo_t = r.tmax;
          }
          hi_t = r.tmax;
          const SlabRay s = make_slab_ray<DRAY>(r, scene_abs);
          best_slot = -1;
          flags = 8u;
          hit = false;
          st.sp = 0;
          const float4 na = __ldg(nodes), nb = __ldg(nodes + 1);
          cur_a = __float_as_uint(nb.z);
          cur_b = __float_as_uint(nb.w);
          fin = !node_visit(na, nb, s, r.tmax, cur_lo);  // root culled: a miss
        }
      }
    }
    const unsigned busy = __ballot_sync(0xffffffffu, !fin);
    if (busy == 0u) {
      if (end < 0 && __ballot_sync(0xffffffffu, ray_i >= 0) == 0u) break;
      continue;
    }
    if (fin) continue;
    // Independent thread scheduling does not promise that the busy lanes run
    // the rest of the iteration as one group; without an explicit sync they
    // were measured to split into 2-3 groups that each walked on their own.
    __syncwarp(busy);
    // The slab data (14 words) is made from the ray in every round instead of
    // being held through the triangle tests (measured at 80 registers, 4M
    // closest hits: 3.69 -> 3.50 ms).
    const SlabRay s = make_slab_ray<DRAY>(r, scene_abs);

    // Node steps continue past a lane's first leaf (postponed) until all but
    // SKW_TRAV_LAG walking lanes hold one, or the lane reaches a second leaf;
    // the leaves are then tested in the order they were reached, which is
    // the reference's order.  (Waiting for the last few lanes to find a leaf
    // left most of the warp idle: with 32 lanes the round length is the
    // slowest lane's.)  Nodes stepped through before the postponed leaf
    // is tested see a larger tmax than the reference's -- a superset of its
    // visits, whose extra triangles all lie beyond the final tmax.
    //
    // Every busy lane is walking when the round starts.  All of them stay in
    // the loop -- a lane that is done idles -- and vote on every step over
    // the busy mask, so they stay one group (a vote over __activemask() would
    // only cover whatever fragment happens to be running together) and one
    // vote per step suffices.
    const float tcull = CLOSEST ? hi_t : s.tmax;
    const int lag = min(SKW_TRAV_LAG, __popc(busy) >> 1);
    bool walking = true, trav = true, has_post = false;
    uint32_t post_a = 0, post_cnt = 0;
    while (true) {
      if (walking) {
        bool pop = true;
        if ((cur_b & 3u) == 0u) {  // a leaf
          if (has_post) {
            walking = pop = false;  // a second leaf: it waits for the next round
          } else if (!(cur_lo > tcull)) {
            post_a = cur_a;
            post_cnt = cur_b >> 8;
            has_post = true;
          }
        } else if (!(cur_lo > tcull)) {
          pop = !expand(nodes, s, tcull, st, cur_a, cur_b, cur_lo, status);
        }
        if (pop) walking = trav = st.pop(tcull, cur_a, cur_b, cur_lo);
      }
      if (__popc(__ballot_sync(busy, walking && !has_post)) <= lag) break;
    }
    __syncwarp(busy);
    if (has_post) {
      const float under = DRAY ? tri_under(scene_abs, fabsf(r.ox) + fabsf(r.oy) + fabsf(r.oz),
                                           fabsf(r.dx) + fabsf(r.dy) + fabsf(r.dz))
                               : 0.0f;
      for (uint32_t k = 0; k < post_cnt; ++k) {
        const int slot = (int)(post_a + k);
        float3 v0, v1, v2;
        int prim, tri;
        load_tri(tris, (uint32_t)slot, v0, v1, v2, prim, tri);
        float t, et;
        const int res = tri_test32<DRAY>(r, v0, v1, v2, t, et, under);
        if (res == kMiss) continue;
        // A ray leaving a surface (surf) starts at an upper bound of the
        // reference's GetNextMinT: a triangle whose t cannot be told apart
        // from that tmin in float lies on the ray's own plane crossing --
        // the triangle it leaves, or geometry touching it there -- and is
        // skipped, as the reference's tmin skips the triangle it leaves.
        if (surf && res == kAmbiguous && t - et < r.tmin) continue;
        if (CLOSEST) {
          if (res == kHit) {
            if (__fsub_rd(t, et) > hi_t) continue;  // certainly beyond the current tmax
            if (__fadd_ru(t, et) < lo_t) {          // certainly nearer: accept in float
              best_slot = slot;
              lo_t = __fsub_rd(t, et);
              hi_t = __fadd_ru(t, et);
              flags &= ~8u;
              continue;
            }
          }
          // Exact re-test against the reference's exact current tmax.
          const ExactHit x = exact_hit<DRAY>(tris, rays, ray_i, slot, best_slot, hi_t);
          if (x.flags != 0u) {
            best_slot = slot;
            lo_t = x.lo;
            hi_t = x.hi;
            flags |= x.flags | 8u;
          }
        } else {
          if (res == kHit) {
            if (t + et < r.tmax) {
              hit = true;
              break;
            }
            if (t - et > r.tmax) continue;
          }
          if (exact_hit<DRAY>(tris, rays, ray_i, slot, -1, 0.0f).flags != 0u) {
            hit = true;
            break;
          }
        }
      }
    }
    fin = hit || !trav;
  }
}

// --------------------------------------------------------------------------
// Accelerators with instances (meshes shared by several primitives) are
// traversed by k_trace_inst: one ray per thread, the reference's
// _NodeIntersect / _NodeIntersectTest restated in double throughout
// (TriangleAccelerator.cpp:154-293, 354-462) -- the slab test of every
// node, the children pushed in the reference's order, at a leaf first its
// instances (the ray taken to mesh space by the instance's world-to-mesh
// Transform, TriangleAccelerator.cpp:213-233, and the instance's subtree
// traversed with it) and then its triangles, all with the reference's
// double Moller-Trumbore.  Exact but slow: instanced scenes are rare and
// the float walk of k_trace does not apply to rays in mesh space.

struct InstDev {
  double m[16];  // world to mesh, row-major
  uint32_t root;
  int32_t prim;
  uint32_t pad[2];
};

// Transform::operator() on a point (with the w division) and a vector
// (Math/Transform.h:239-269), every sum and product rounded separately.
__device__ __forceinline__ void xf_point(const double *m, double x, double y, double z, double *o) {
  const double xp = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(m[0], x), __dmul_rn(m[1], y)), __dmul_rn(m[2], z)), m[3]);
  const double yp = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(m[4], x), __dmul_rn(m[5], y)), __dmul_rn(m[6], z)), m[7]);
  const double zp = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(m[8], x), __dmul_rn(m[9], y)), __dmul_rn(m[10], z)), m[11]);
  const double w = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(m[12], x), __dmul_rn(m[13], y)), __dmul_rn(m[14], z)), m[15]);
  o[0] = xp;
  o[1] = yp;
  o[2] = zp;
  if (w != 1.0) {
    const double inv = __ddiv_rn(1.0, w);
    o[0] = __dmul_rn(xp, inv);
    o[1] = __dmul_rn(yp, inv);
    o[2] = __dmul_rn(zp, inv);
  }
}
__device__ __forceinline__ void xf_vector(const double *m, double x, double y, double z, double *o) {
  o[0] = __dadd_rn(__dadd_rn(__dmul_rn(m[0], x), __dmul_rn(m[1], y)), __dmul_rn(m[2], z));
  o[1] = __dadd_rn(__dadd_rn(__dmul_rn(m[4], x), __dmul_rn(m[5], y)), __dmul_rn(m[6], z));
  o[2] = __dadd_rn(__dadd_rn(__dmul_rn(m[8], x), __dmul_rn(m[9], y)), __dmul_rn(m[10], z));
}

// The reference's slab test (TriangleAccelerator.cpp:176-192): true when
// the node is culled.
__device__ __forceinline__ bool slab_culled(float4 na, float4 nb, const double *o, const double *inv, double tmin,
                                            double tmax) {
  const double lo[3] = {na.x, na.y, na.z}, hi[3] = {na.w, nb.x, nb.y};
  double tn[3], tf[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    tn[k] = __dmul_rn(__dsub_rn(lo[k], o[k]), inv[k]);
    tf[k] = __dmul_rn(__dsub_rn(hi[k], o[k]), inv[k]);
    if (tn[k] > tf[k]) {
      const double t = tn[k];
      tn[k] = tf[k];
      tf[k] = t;
    }
  }
  return tmin > tf[0] || tn[0] > tf[1] || tn[1] > tf[0] || tn[2] > tf[0] || tmin > tf[1] || tn[0] > tf[2] ||
         tn[1] > tf[2] || tn[2] > tf[1] || tmin > tf[2] || tn[0] > tmax || tn[1] > tmax || tn[2] > tmax;
}

// One (sub)tree walk from `root` for the ray (o, d, tmin, tmax): closest hit
// updates tmax and the hit's slot (best_slot; the instance's primitive in
// best_prim when inside an instance), any hit returns on the first.  Leaves
// of the top tree may hold instances (INNER = false); a subtree's do not.
// Returns false on stack overflow.
template <int CAP, bool CLOSEST, bool INNER>
__device__ bool walk_exact(const float4 *__restrict__ nodes, const float4 *__restrict__ tris,
                           const InstDev *__restrict__ inst, const uint4 *__restrict__ ext, uint32_t root,
                           const double *o, const double *d, double tmin, double &tmax, int &best_slot,
                           int &best_prim, bool &hit, uint32_t *stk) {
  const double inv[3] = {__ddiv_rn(1.0, d[0]), __ddiv_rn(1.0, d[1]), __ddiv_rn(1.0, d[2])};
  int sp = 0;
  stk[sp++] = root;
  while (sp > 0) {
    const uint32_t ni = stk[--sp];
    const float4 na = __ldg(nodes + 2 * ni), nb = __ldg(nodes + 2 * ni + 1);
    if (slab_culled(na, nb, o, inv, tmin, tmax)) continue;
    const uint32_t a = __float_as_uint(nb.z), b = __float_as_uint(nb.w);
    if (b & 3u) {
      const uint32_t axis = (b & 3u) - 1u, mask = (b >> 2) & 7u;
      const uint32_t sL = a, sM = a + (mask & 1u), sR = sM + ((mask >> 1) & 1u);
      if (sp + 3 > CAP) return false;
      if (d[axis] > 0.0) {  // children pushed in reverse so that the left one pops first
        if (mask & 4u) stk[sp++] = sR;
        if (mask & 2u) stk[sp++] = sM;
        if (mask & 1u) stk[sp++] = sL;
      } else {
        if (mask & 1u) stk[sp++] = sL;
        if (mask & 2u) stk[sp++] = sM;
        if (mask & 4u) stk[sp++] = sR;
      }
      continue;
    }
    uint32_t tf = a, tc = b >> 8, i0 = 0, ic = 0;
    if (!INNER && (b & kLeafExt)) {
      const uint4 e = __ldg(ext + a);
      tf = e.x;
      tc = e.y;
      i0 = e.z;
      ic = e.w;
    }
    for (uint32_t k = 0; k < ic && !INNER; ++k) {
      const InstDev *I = inst + i0 + k;
      double mo[3], md[3];
      xf_point(I->m, o[0], o[1], o[2], mo);
      xf_vector(I->m, d[0], d[1], d[2], md);
      int slot = -1, pr = -1;
      bool h2 = false;
      if (!walk_exact<CAP, CLOSEST, true>(nodes, tris, inst, ext, I->root, mo, md, tmin, tmax, slot, pr, h2,
                                          stk + sp))
        return false;
      if (h2) {
        hit = true;
        if (!CLOSEST) return true;
        best_slot = slot;
        best_prim = I->prim;
      }
    }
    for (uint32_t k = 0; k < tc; ++k) {
      const int slot = (int)(tf + k);
      float3 v0, v1, v2;
      int prim, tri;
      load_tri(tris, (uint32_t)slot, v0, v1, v2, prim, tri);
      double t64;
      if (tri_test64v(o[0], o[1], o[2], d[0], d[1], d[2], v0, v1, v2, tmin, tmax, t64)) {
        hit = true;
        if (!CLOSEST) return true;
        tmax = t64;
        best_slot = slot;
        best_prim = prim;
      }
    }
  }
  return true;
}

template <int CAP, bool CLOSEST, bool DRAY>
__global__ void __launch_bounds__(128)
    k_trace_inst(const float4 *__restrict__ nodes, const float4 *__restrict__ tris, const InstDev *__restrict__ inst,
                 const uint4 *__restrict__ ext, const float4 *__restrict__ rays, int n, const int *__restrict__ n_dev,
                 const int32_t *__restrict__ out_index, void *__restrict__ out, unsigned *__restrict__ status,
                 unsigned long long *__restrict__ traced) {
  if (n_dev) n = min(n, *n_dev);
  if (traced && blockIdx.x == 0 && threadIdx.x == 0 && n > 0) atomicAdd(traced, (unsigned long long)n);
  uint32_t stk[2 * CAP];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double o[3], d[3], tmin, tmax;
    if (DRAY) {
      const RayD r = load_ray_d(rays, i);
      o[0] = r.ox, o[1] = r.oy, o[2] = r.oz, d[0] = r.dx, d[1] = r.dy, d[2] = r.dz, tmin = r.tmin, tmax = r.tmax;
    } else {
      const RayF r = load_ray(rays, i);
      o[0] = r.ox, o[1] = r.oy, o[2] = r.oz, d[0] = r.dx, d[1] = r.dy, d[2] = r.dz, tmin = r.tmin, tmax = r.tmax;
    }
    int slot = -1, prim = -1;
    bool hit = false;
    if (!walk_exact<CAP, CLOSEST, false>(nodes, tris, inst, ext, 0u, o, d, tmin, tmax, slot, prim, hit, stk))
      atomicOr(status, 1u);
    const int oi = out_index ? out_index[i] : i;
    if (!CLOSEST) {
      ((uint8_t *)out)[oi] = hit ? 1 : 0;
    } else if (DRAY) {
      int4 h = make_int4(0, 0x7ff00000, -1, -1);
      if (hit) {
        const long long tb = __double_as_longlong(tmax);
        h = make_int4((int)(tb & 0xffffffffll), (int)(tb >> 32), prim, __float_as_int(__ldg(tris + 3 * slot + 1).w));
      }
      ((int4 *)out)[oi] = h;
    } else {
      int4 h = make_int4(0x7f800000, -1, -1, 0);
      if (hit) h = make_int4(__float_as_int((float)tmax), prim, __float_as_int(__ldg(tris + 3 * slot + 1).w), 1);
      ((int4 *)out)[oi] = h;
    }
  }
}

// Per-device launch facts, computed once per device on first use and read
// without a lock afterwards (launches may come from several host threads).
constexpr int kMaxDevices = 64;

std::mutex &prepare_mutex() {
  static std::mutex m;
  return m;
}

cudaError_t current_device(int &dev) {
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  return dev < 0 || dev >= kMaxDevices ? cudaErrorInvalidDevice : cudaSuccess;
}

// The kernel of a variant: bit 0 closest hit, bit 1 double rays.
template <int CAP>
const void *trace_kernel(int variant) {
  switch (variant) {
    case 0: return (const void *)k_trace<CAP, false, false>;
    case 1: return (const void *)k_trace<CAP, true, false>;
    case 2: return (const void *)k_trace<CAP, false, true>;
    default: return (const void *)k_trace<CAP, true, true>;
  }
}

// Resident CTAs per SM of each variant on each device (0 = not yet known).
template <int CAP>
std::atomic<int> &cap_occupancy(int dev, int variant) {
  static std::atomic<int> blocks_per_sm[kMaxDevices][4];
  return blocks_per_sm[dev][variant];
}

template <int CAP>
cudaError_t cap_prepare(int dev) {
  bool known = true;
  for (int v = 0; v < 4; ++v) known = known && cap_occupancy<CAP>(dev, v).load(std::memory_order_acquire) != 0;
  if (known) return cudaSuccess;
  std::lock_guard<std::mutex> lock(prepare_mutex());
  for (int v = 0; v < 4; ++v) {
    std::atomic<int> &slot = cap_occupancy<CAP>(dev, v);
    if (slot.load(std::memory_order_relaxed) != 0) continue;
    int occ = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, trace_kernel<CAP>(v), SKW_TRAV_BLOCK, 0);
    if (e != cudaSuccess) return e;
    slot.store(occ < 1 ? 1 : occ, std::memory_order_release);
  }
  return cudaSuccess;
}

// SM count of each device (0 = not yet known).
cudaError_t device_sms(int dev, int &sms) {
  static std::atomic<int> cache[kMaxDevices];
  sms = cache[dev].load(std::memory_order_acquire);
  if (sms != 0) return cudaSuccess;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  cache[dev].store(sms, std::memory_order_release);
  return cudaSuccess;
}

// Device tables of the accelerators that have instances, by their node
// array (the traversal launches receive the node pointer).
// Per-accelerator launch tables, keyed by the device node array: the
// instance tables (null: no instances) and the accelerator's traced-ray
// counter (null: none).
struct InstTables {
  const void *inst = nullptr;
  const void *ext = nullptr;
  unsigned long long *traced = nullptr;
};
std::mutex &inst_mutex() {
  static std::mutex m;
  return m;
}
std::unordered_map<const void *, InstTables> &inst_registry() {
  static std::unordered_map<const void *, InstTables> r;
  return r;
}
bool find_instances(const void *nodes, InstTables &t) {
  std::lock_guard<std::mutex> lock(inst_mutex());
  auto &r = inst_registry();
  if (r.empty()) return false;
  auto it = r.find(nodes);
  if (it == r.end()) return false;
  t = it->second;
  return true;
}

template <int CAP>
cudaError_t launch_inst(int variant, const void *nodes, const void *tris, const InstTables &T, const void *rays,
                        int64_t n, const int *n_dev, const int32_t *out_index, void *out, unsigned *status,
                        cudaStream_t stream, int sms) {
  const int64_t want = (n + 127) / 128, cap = (int64_t)sms * 16;
  const dim3 grid((unsigned)(want < cap ? want : cap)), block(128);
  const float4 *nd = (const float4 *)nodes, *tr = (const float4 *)tris, *ry = (const float4 *)rays;
  const InstDev *in = (const InstDev *)T.inst;
  const uint4 *ex = (const uint4 *)T.ext;
  switch (variant) {
    case 0:
      k_trace_inst<CAP, false, false><<<grid, block, 0, stream>>>(nd, tr, in, ex, ry, (int)n, n_dev, out_index, out, status, T.traced);
      break;
    case 1:
      k_trace_inst<CAP, true, false><<<grid, block, 0, stream>>>(nd, tr, in, ex, ry, (int)n, n_dev, out_index, out, status, T.traced);
      break;
    case 2:
      k_trace_inst<CAP, false, true><<<grid, block, 0, stream>>>(nd, tr, in, ex, ry, (int)n, n_dev, out_index, out, status, T.traced);
      break;
    default:
      k_trace_inst<CAP, true, true><<<grid, block, 0, stream>>>(nd, tr, in, ex, ry, (int)n, n_dev, out_index, out, status, T.traced);
  }
  return cudaGetLastError();
}

template <int CAP>
cudaError_t launch_cap(int variant, const void *nodes, const void *tris, const void *rays, int64_t n,
                       const int *n_dev, float scene_abs, const int32_t *out_index, void *out, unsigned *status,
                       cudaStream_t stream, int ctas_per_sm, int *work, int surf) {
  if (!work) return cudaErrorInvalidValue;
  int dev = 0, sms = 0;
  cudaError_t e = current_device(dev);
  if (e != cudaSuccess || (e = cap_prepare<CAP>(dev)) != cudaSuccess || (e = device_sms(dev, sms)) != cudaSuccess)
    return e;
  InstTables T;
  if (find_instances(nodes, T) && T.inst)
    return launch_inst<CAP>(variant, nodes, tris, T, rays, n, n_dev, out_index, out, status, stream, sms);
  int per_sm = cap_occupancy<CAP>(dev, variant).load(std::memory_order_acquire);
  if (ctas_per_sm > 0 && ctas_per_sm < per_sm) per_sm = ctas_per_sm;
  const int64_t warps_per_block = SKW_TRAV_BLOCK / 32;
  int64_t blocks = (int64_t)per_sm * sms;
  // A launch of fewer rays than the grid has lanes spreads them over all
  // resident warps, down to one ray per warp: a warp's time is the sum of its
  // lanes' divergent paths (1,000 rays over 18,000 triangles: 142 us in groups
  // of 16, 106 us in groups of 1).
  const int64_t needed = (n + warps_per_block - 1) / warps_per_block;
  if (blocks > needed) blocks = needed;
  if ((e = cudaMemsetAsync(work, 0, sizeof(int), stream)) != cudaSuccess) return e;
  const float4 *nd = (const float4 *)nodes, *tr = (const float4 *)tris, *ry = (const float4 *)rays;
  const dim3 grid((unsigned)blocks), block(SKW_TRAV_BLOCK);
  switch (variant) {
    case 0:
      k_trace<CAP, false, false><<<grid, block, 0, stream>>>(nd, tr, ry, (int)n, n_dev, scene_abs, out_index, out,
                                                             status, (unsigned *)work, surf, T.traced);
      break;
    case 1:
      k_trace<CAP, true, false><<<grid, block, 0, stream>>>(nd, tr, ry, (int)n, n_dev, scene_abs, out_index, out,
                                                            status, (unsigned *)work, surf, T.traced);
      break;
    case 2:
      k_trace<CAP, false, true><<<grid, block, 0, stream>>>(nd, tr, ry, (int)n, n_dev, scene_abs, out_index, out,
                                                            status, (unsigned *)work, surf, T.traced);
      break;
    default:
      k_trace<CAP, true, true><<<grid, block, 0, stream>>>(nd, tr, ry, (int)n, n_dev, scene_abs, out_index, out,
                                                           status, (unsigned *)work, surf, T.traced);
  }
  return cudaGetLastError();
}

cudaError_t launch_variant(int variant, int stack_cap, const void *nodes, const void *tris, const void *rays,
                           int64_t n, const int *n_dev, float scene_abs, const int32_t *out_index, void *out,
                           unsigned *status, cudaStream_t stream, int ctas_per_sm, int *work, int surf) {
  if (n <= 0) return cudaSuccess;
  switch (stack_cap) {
    case 48:
      return launch_cap<48>(variant, nodes, tris, rays, n, n_dev, scene_abs, out_index, out, status, stream,
                            ctas_per_sm, work, surf);
    case 96:
      return launch_cap<96>(variant, nodes, tris, rays, n, n_dev, scene_abs, out_index, out, status, stream,
                            ctas_per_sm, work, surf);
    case 192:
      return launch_cap<192>(variant, nodes, tris, rays, n, n_dev, scene_abs, out_index, out, status, stream,
                             ctas_per_sm, work, surf);
    default:
      return launch_cap<416>(variant, nodes, tris, rays, n, n_dev, scene_abs, out_index, out, status, stream,
                             ctas_per_sm, work, surf);
  }
}

}  // namespace

cudaError_t prepare_traversal(int stack_cap) {
  int dev = 0, sms = 0;
  cudaError_t e = current_device(dev);
  if (e != cudaSuccess || (e = device_sms(dev, sms)) != cudaSuccess) return e;
  switch (stack_cap) {
    case 48: return cap_prepare<48>(dev);
    case 96: return cap_prepare<96>(dev);
    case 192: return cap_prepare<192>(dev);
    default: return cap_prepare<416>(dev);
  }
}

int traversal_max_ctas_per_sm(int stack_cap) {
  int dev = 0;
  if (current_device(dev) != cudaSuccess || prepare_traversal(stack_cap) != cudaSuccess) return 1;
  switch (stack_cap) {
    case 48: return cap_occupancy<48>(dev, 1).load();
    case 96: return cap_occupancy<96>(dev, 1).load();
    case 192: return cap_occupancy<192>(dev, 1).load();
    default: return cap_occupancy<416>(dev, 1).load();
  }
}

int traversal_stack_capacity(int max_depth) {
  const int need = 2 * max_depth + 1;
  if (need <= 48) return 48;
  if (need <= 96) return 96;
  if (need <= 192) return 192;
  return 416;  // the reference's depth limit 200 needs 401 entries
}

cudaError_t launch_traversal(bool closest, int stack_cap, const void *nodes, const void *tris, const void *rays,
                             int64_t n, const int *n_dev, float scene_abs, const int32_t *out_index, void *out,
                             unsigned *status, cudaStream_t stream, int ctas_per_sm, int *work, bool surface) {
  return launch_variant(closest ? 1 : 0, stack_cap, nodes, tris, rays, n, n_dev, scene_abs, out_index, out, status,
                        stream, ctas_per_sm, work, surface ? 1 : 0);
}

void register_instances(const void *nodes, const void *inst, const void *ext) {
  std::lock_guard<std::mutex> lock(inst_mutex());
  InstTables &t = inst_registry()[nodes];
  t.inst = inst;
  t.ext = ext;
}

void register_ray_counter(const void *nodes, unsigned long long *traced) {
  std::lock_guard<std::mutex> lock(inst_mutex());
  inst_registry()[nodes].traced = traced;
}

void unregister_instances(const void *nodes) {
  std::lock_guard<std::mutex> lock(inst_mutex());
  inst_registry().erase(nodes);
}

cudaError_t launch_traversal_d(bool closest, int stack_cap, const void *nodes, const void *tris, const void *rays,
                               int64_t n, float scene_abs, void *out, unsigned *status, cudaStream_t stream,
                               int *work) {
  return launch_variant(closest ? 3 : 2, stack_cap, nodes, tris, rays, n, nullptr, scene_abs, nullptr, out, status,
                        stream, 0, work, 0);
}

}  // namespace skw
