// Construction of the ternary bbox kd-tree on the GPU: node for node the
// tree of the host build (accel_build.cpp), which restates the reference's
// TriangleAccelerator build (Raytracer/Core/TriangleAccelerator.cpp:470-729):
// node box, leaf rule, bucketed split search with its float / double
// arithmetic, and the in-place three-way partition's exact element order.
//
// Layout: the triangles' float boxes in slot order (6 floats: lo xyz,
// hi xyz) and each slot's triangle; every slot carries the range [b, e) of
// the node it is in (b = -1 once that node is a leaf), so a level of the
// tree is a fixed sequence of slot-parallel launches and 64-bit scans, and
// a node's own values live at its first slot b.  Per level:
//   * node boxes: a warp-segmented reduction of 64-bit keys (value order,
//     then slot) merged with atomics — the reference's min / max keep the
//     first of equal values (it matters only for the sign of a zero);
//   * leaf rule (<= 4 triangles, all three axes split through the middle,
//     depth 200), candidate count tries = min(200, 2n), per-axis scale;
//   * split search, by node size: per candidate plane the left / middle /
//     right boxes and counts (box unions and counts do not depend on the
//     order they are formed in), then the costs in the reference's double
//     arithmetic, which only the planes that could be the least by their
//     float costs need.  Up to 32 triangles one warp holds the node's boxes
//     and each lane a plane (k_split_small); up to 4,096 a block per axis
//     fills buckets in shared memory (k_split_mid); above that blocks of 4,096
//     triangles do and merge them into global ones (k_fill_big, k_score_big);
//   * partition: the reference's sequential swap loop (left to the front in
//     order of processing, right to the back, a rotating middle block)
//     computed in parallel.  Elements are processed from the front, except
//     that after each right-class element the loop takes elements from the
//     back until it meets one that is not right-class: with prefix counts
//     over the front stream (right-class elements so far) and the back
//     stream (its runs), each element's processing step follows; left and
//     right destinations are ranks in that order, and a middle element's
//     destination follows the chain "moved to the block's end when the
//     block's front reaches it" by pointer jumping.
// Accelerators whose meshes are shared by several primitives (instancing)
// are built on the host.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "accel_build.h"
#include "kernels.h"

namespace skw {
namespace {

constexpr int kB = 256;
constexpr int kTries = 200;    // TriangleAccelerator.h:131
constexpr int kLeafMax = 4;    // TriangleAccelerator.h:128
constexpr int kDepthMax = 200; // TriangleAccelerator.h:134
// Split search by node size.  Below 33 triangles a node has at most 64
// planes, two per lane; a chunk of 4,096 triangles outweighs the 4,200 words
// of an axis' buckets that its block empties and merges.
constexpr int kSmall = 32, kMid = 4096;

// Order-preserving key of a float (NaN excluded by the callers).
__device__ __forceinline__ uint32_t okey(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float okey_inv(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}
// Bucket keys: min identity 0xFFFFFFFF (decodes to +inf), max identity 0
// (decodes to -inf), as the reference's empty BBox3D.
__device__ __forceinline__ float lo_of(uint32_t k) { return k == 0xFFFFFFFFu ? INFINITY : okey_inv(k); }
__device__ __forceinline__ float hi_of(uint32_t k) { return k == 0u ? -INFINITY : okey_inv(k); }

// (size_t) of a double as the reference's x86-64 build computes it: NaN ->
// 2^63, values >= 2^64 -> 0 (the same rule as the host build's cast_size).
__device__ __forceinline__ uint64_t cast_size(double v) {
  if (isnan(v)) return 1ull << 63;
  if (v >= 18446744073709551616.0) return 0ull;
  if (v >= 9223372036854775808.0) return (uint64_t)__double2ll_rz(v - 9223372036854775808.0) + (1ull << 63);
  return (uint64_t)__double2ll_rz(v);
}

// BBox3D<double>::Area of a box with float corners.
__device__ __forceinline__ double area_d(const float *lo, const float *hi) {
  const double x = fabs(__dsub_rn((double)hi[0], (double)lo[0]));
  const double y = fabs(__dsub_rn((double)hi[1], (double)lo[1]));
  const double z = fabs(__dsub_rn((double)hi[2], (double)lo[2]));
  return __dmul_rn(2.0, __dadd_rn(__dadd_rn(__dmul_rn(x, y), __dmul_rn(x, z)), __dmul_rn(y, z)));
}
// BBox3D<float>::Area.
__device__ __forceinline__ float area_f(const float *lo, const float *hi) {
  const float x = fabsf(__fsub_rn(hi[0], lo[0]));
  const float y = fabsf(__fsub_rn(hi[1], lo[1]));
  const float z = fabsf(__fsub_rn(hi[2], lo[2]));
  return __fmul_rn(2.0f, __fadd_rn(__fadd_rn(__fmul_rn(x, y), __fmul_rn(x, z)), __fmul_rn(y, z)));
}
// std::min(1.0, v)
__device__ __forceinline__ double min1(double v) { return v < 1.0 ? v : 1.0; }

struct Dev {
  int64_t n;
  float *box, *box2;          // 6 floats per slot
  uint32_t *perm, *perm2;     // triangle of each slot
  int2 *seg;                  // node range of each slot ((-1, -1): in a leaf)
  uint8_t *smask, *sord;      // node's middle-split axes; child ordinal in its parent
  int32_t *spar;              // parent node id (-1: the root)
  // per node, at its first slot
  unsigned long long *hkeys;  // 6 box keys
  float *hbox;                // 6 floats
  double *hcoef;              // 3 per node
  double *hsplit;
  int32_t *hid, *htries, *haxis, *hbase;  // hbase: a big node's first bucket
  uint32_t *hnl, *hnr;
  uint8_t *hleaf;
  double *bcost, *bpos;       // 3 per node
  uint32_t *buckets;          // big nodes, 7 words per bucket: lo keys, hi keys, count
  // The level's nodes to split, by size (their first slots), and the chunks
  // of the big ones (first slot of the node, chunk); count: their numbers.
  uint32_t *small, *mid, *big;
  uint2 *chunks;
  int *count;                 // small, mid, big, chunks
  // per level
  uint8_t *cls;
  uint64_t *cnt, *cnt2, *cnt3, *sums;  // n + 1 each (sums: block totals)
  uint32_t *tarr, *jarr, *ord, *iarr, *f0, *f1, *lmb, *dest;
  int *err;
  int *maxseg;                // the level's largest node (triangles)
  unsigned long long *n_leaves;
  // node records, by node id
  float *rbox;
  uint32_t *rtb, *rte;
  uint8_t *rflags;
  int32_t *rchild;
};

inline unsigned grid_of(int64_t m) { return (unsigned)((m + kB - 1) / kB); }

// The primitives' meshes: their arrays, where their triangles lie among all,
// their primitive and matrix.
struct DevMesh {
  const float *v;
  const int32_t *ix;
  int64_t n_vertices, t0;
  double m[16];
  int32_t prim, has_m;
};

__device__ __forceinline__ const DevMesh &mesh_of(const DevMesh *__restrict__ ms, int n_meshes, int64_t t) {
  int lo = 0, hi = n_meshes;  // the last mesh whose first triangle is not past t
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (ms[mid].t0 <= t) lo = mid;
    else hi = mid;
  }
  return ms[lo];
}

// Whether TriangleMesh keeps a triangle: indices in range and not repeated
// (TriangleMesh.cpp:176-182).
__global__ void k_keep(const DevMesh *__restrict__ ms, int n_meshes, int64_t total, uint64_t *cnt) {
  const int64_t t = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (t > total) return;
  uint64_t keep = 0;
  if (t < total) {
    const DevMesh &m = mesh_of(ms, n_meshes, t);
    const int32_t *ix = m.ix + 3 * (t - m.t0);
    const int32_t i = ix[0], j = ix[1], k = ix[2];
    keep = i >= 0 && j >= 0 && k >= 0 && i < m.n_vertices && j < m.n_vertices && k < m.n_vertices && i != j &&
           i != k && j != k;
  }
  cnt[t] = keep;
}

// One row of Matrix4x4 * Point3D<float> in the host build's order.
__device__ __forceinline__ float row_d(const double *m, float x, float y, float z) {
  return (float)__dadd_rn(
      __dadd_rn(__dadd_rn(__dmul_rn(m[0], x), __dmul_rn(m[1], y)), __dmul_rn(m[2], z)), m[3]);
}

// The kept triangles in world space (cnt: how many are kept before each) as
// slot records in input order, their boxes and the root's state.  Bound by
// its scattered vertex reads and 101 bytes of writes a triangle: 0.04 ms with
// k_keep for 1,098,576 triangles; the same loop on the host's threads and the
// copy of its boxes took 6.2.
__global__ void k_collect(Dev D, const DevMesh *__restrict__ ms, int n_meshes, int64_t total, DevTri *__restrict__ src) {
  const int64_t t = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (t >= total) return;
  const uint64_t o = D.cnt[t];
  if (D.cnt[t + 1] == o) return;
  const DevMesh &m = mesh_of(ms, n_meshes, t);
  const int32_t *ix = m.ix + 3 * (t - m.t0);
  float v[9], lo[3], hi[3];
  for (int a = 0; a < 3; ++a) {
    lo[a] = INFINITY;
    hi[a] = -INFINITY;
  }
  for (int q = 0; q < 3; ++q) {
    const float *p = m.v + 3 * (int64_t)ix[q];
    float x = p[0], y = p[1], z = p[2];
    if (m.has_m) {  // Transform on Point3D<float>: a divide by w is a product with its double reciprocal
      const float xp = row_d(m.m, x, y, z), yp = row_d(m.m + 4, x, y, z), zp = row_d(m.m + 8, x, y, z);
      const float wp = row_d(m.m + 12, x, y, z);
      x = xp;
      y = yp;
      z = zp;
      if (!(wp == 1.0f)) {
        const double inv = __ddiv_rn(1.0, (double)wp);
        x = (float)__dmul_rn((double)xp, inv);
        y = (float)__dmul_rn((double)yp, inv);
        z = (float)__dmul_rn((double)zp, inv);
      }
    }
    v[3 * q] = x;
    v[3 * q + 1] = y;
    v[3 * q + 2] = z;
    for (int a = 0; a < 3; ++a) {  // std::min / std::max: the first of equal values, NaN skipped
      lo[a] = v[3 * q + a] < lo[a] ? v[3 * q + a] : lo[a];
      hi[a] = hi[a] < v[3 * q + a] ? v[3 * q + a] : hi[a];
    }
  }
  float4 *r = (float4 *)(src + o);
  r[0] = make_float4(v[0], v[1], v[2], __int_as_float(m.prim));
  r[1] = make_float4(v[3], v[4], v[5], __int_as_float((int32_t)(o - D.cnt[m.t0])));
  r[2] = make_float4(v[6], v[7], v[8], 0.0f);
  for (int a = 0; a < 3; ++a) {
    D.box[o * 6 + a] = lo[a];
    D.box[o * 6 + 3 + a] = hi[a];
  }
  D.perm[o] = (uint32_t)o;
  D.seg[o] = make_int2(0, (int)D.n);
  D.smask[o] = 0;
  D.sord[o] = 0;
  D.spar[o] = -1;
}

// Heads of the level's nodes: their rank (a scan) gives the node id.
__global__ void k_heads(Dev D) {
  const int64_t s = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (s > D.n) return;
  uint64_t h = 0;
  if (s < D.n && D.seg[s].x == (int)s) {
    h = 1;
    atomicMax(D.maxseg, D.seg[s].y - (int)s);
    for (int c = 0; c < 3; ++c) {
      D.hkeys[s * 6 + c] = ~0ull;
      D.hkeys[s * 6 + 3 + c] = 0ull;
    }
  }
  D.cnt[s] = h;
}

// Node boxes: keys (value, slot) so that the first of equal values wins,
// as in the reference's min / max over the node's triangles in slot order;
// -0 and +0 compare equal, NaN is skipped.  Runs of lanes in one node are
// reduced with shuffles, then merged with atomics.
__global__ void k_node_box(Dev D) {
  const int64_t s = (int64_t)blockIdx.x * kB + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int b = -1;
  unsigned long long k[6];
  for (int c = 0; c < 3; ++c) {
    k[c] = ~0ull;
    k[3 + c] = 0ull;
  }
  if (s < D.n) {
    b = D.seg[s].x;
    if (b >= 0) {
      for (int c = 0; c < 3; ++c) {
        const float lo = D.box[s * 6 + c], hi = D.box[s * 6 + 3 + c];
        if (!isnan(lo)) k[c] = ((unsigned long long)okey(lo == 0.0f ? 0.0f : lo) << 32) | (uint32_t)s;
        if (!isnan(hi))
          k[3 + c] = ((unsigned long long)okey(hi == 0.0f ? 0.0f : hi) << 32) | (0xFFFFFFFFu - (uint32_t)s);
      }
    }
  }
  for (int o = 1; o < 32; o <<= 1) {
    const int ob = __shfl_up_sync(0xffffffffu, b, o);
    unsigned long long t[6];
    for (int c = 0; c < 6; ++c) t[c] = __shfl_up_sync(0xffffffffu, k[c], o);
    if (lane >= o && ob == b) {
      for (int c = 0; c < 3; ++c) {
        k[c] = t[c] < k[c] ? t[c] : k[c];
        k[3 + c] = t[3 + c] > k[3 + c] ? t[3 + c] : k[3 + c];
      }
    }
  }
  const int nb = __shfl_down_sync(0xffffffffu, b, 1);
  if (b >= 0 && (lane == 31 || nb != b)) {
    for (int c = 0; c < 3; ++c) {
      atomicMin(&D.hkeys[(int64_t)b * 6 + c], k[c]);
      atomicMax(&D.hkeys[(int64_t)b * 6 + 3 + c], k[3 + c]);
    }
  }
}

// A node's record and leaf decision (Node::Node, TriangleAccelerator.cpp:
// 621-636); internal nodes get their candidate count and per-axis scale
// (_DetermineBestSplit, :512-530) and go to the list of their size.
__global__ void k_head_setup(Dev D, int64_t level_base, int depth) {
  const int64_t s = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (s < D.n && D.seg[s].x == (int)s) {
    const int2 r = D.seg[s];
    const int64_t id = level_base + (int64_t)D.cnt[s];
    D.hid[s] = (int32_t)id;
    float lo[3], hi[3];
    for (int c = 0; c < 3; ++c) {
      const unsigned long long kl = D.hkeys[s * 6 + c], kh = D.hkeys[s * 6 + 3 + c];
      lo[c] = kl == ~0ull ? INFINITY : D.box[(int64_t)(uint32_t)kl * 6 + c];
      hi[c] = kh == 0ull ? -INFINITY : D.box[(int64_t)(0xFFFFFFFFu - (uint32_t)kh) * 6 + 3 + c];
      D.hbox[s * 6 + c] = lo[c];
      D.hbox[s * 6 + 3 + c] = hi[c];
      D.rbox[id * 6 + c] = lo[c];
      D.rbox[id * 6 + 3 + c] = hi[c];
    }
    D.rtb[id] = (uint32_t)r.x;
    D.rte[id] = (uint32_t)r.y;
    for (int c = 0; c < 3; ++c) D.rchild[id * 3 + c] = -1;
    const int32_t par = D.spar[s];
    if (par >= 0) D.rchild[(int64_t)par * 3 + D.sord[s]] = (int32_t)id;
    const int count = r.y - r.x;
    const unsigned mask = D.smask[s];
    if (count <= kLeafMax || mask == 7u || depth >= kDepthMax) {
      D.hleaf[s] = 1;
      D.rflags[id] = 0;
      atomicAdd(D.n_leaves, 1ull);
    } else {
      D.hleaf[s] = 0;
      const int tries = min(kTries, 2 * count);
      D.htries[s] = tries;
      for (int a = 0; a < 3; ++a) {
        // size_t / float converts the count to float: a float division
        D.hcoef[s * 3 + a] = (double)__fdiv_rn((float)tries, __fsub_rn(hi[a], lo[a]));
      }
      if (count <= kSmall) {
        D.small[atomicAdd(D.count, 1)] = (uint32_t)s;
      } else if (count <= kMid) {
        D.mid[atomicAdd(D.count + 1, 1)] = (uint32_t)s;
      } else {
        const int k = atomicAdd(D.count + 2, 1), nc = (count + kMid - 1) / kMid;
        D.big[k] = (uint32_t)s;
        D.hbase[s] = k * 9 * kTries;
        const int c0 = atomicAdd(D.count + 3, nc);
        for (int c = 0; c < nc; ++c) D.chunks[c0 + c] = make_uint2((uint32_t)s, (uint32_t)c);
      }
    }
  }
}

// Union of two bucket boxes with counts (the order of unions does not
// change a union of float boxes).
struct BoxN {
  float lo[3], hi[3];
  uint32_t n;
};
__device__ __forceinline__ BoxN box_empty() {
  BoxN b;
  for (int c = 0; c < 3; ++c) {
    b.lo[c] = INFINITY;
    b.hi[c] = -INFINITY;
  }
  b.n = 0;
  return b;
}
__device__ __forceinline__ void box_unite(BoxN &a, const BoxN &b) {
  for (int c = 0; c < 3; ++c) {
    a.lo[c] = fminf(a.lo[c], b.lo[c]);
    a.hi[c] = fmaxf(a.hi[c], b.hi[c]);
  }
  a.n += b.n;
}
__device__ __forceinline__ BoxN box_keys(const uint32_t *r) {  // a bucket as filled (keys)
  BoxN b;
  for (int c = 0; c < 3; ++c) {
    b.lo[c] = lo_of(r[c]);
    b.hi[c] = hi_of(r[3 + c]);
  }
  b.n = r[6];
  return b;
}
__device__ __forceinline__ BoxN box_shfl_up(const BoxN &a, int o) {
  BoxN b;
  for (int c = 0; c < 3; ++c) {
    b.lo[c] = __shfl_up_sync(0xffffffffu, a.lo[c], o);
    b.hi[c] = __shfl_up_sync(0xffffffffu, a.hi[c], o);
  }
  b.n = __shfl_up_sync(0xffffffffu, a.n, o);
  return b;
}
__device__ __forceinline__ BoxN box_shfl_down(const BoxN &a, int o) {
  BoxN b;
  for (int c = 0; c < 3; ++c) {
    b.lo[c] = __shfl_down_sync(0xffffffffu, a.lo[c], o);
    b.hi[c] = __shfl_down_sync(0xffffffffu, a.hi[c], o);
  }
  b.n = __shfl_down_sync(0xffffffffu, a.n, o);
  return b;
}

// min(tries, (size_t)((double)d * coef + 1.0)) (_DetermineBestSplit, :536-540).
// coef is a float, so the product is exact in double; in float the fused
// multiply-add is the correctly rounded sum, and where that is not within its
// rounding of a whole number both have the same whole part.
__device__ __forceinline__ int plane_of(float d, double coef, int tries) {
  const float v = fmaf(d, (float)coef, 1.0f);
  if (v >= 1.0f && v < 4194304.0f && fabsf(v - rintf(v)) > v * 2.4e-7f) return min(tries, (int)v);
  return (int)min((uint64_t)tries, cast_size(__dadd_rn(__dmul_rn((double)d, coef), 1.0)));
}

// The cost of a plane, sum(n_child * area_child / area_node) with the 0.8
// bonus for an empty side, in the reference's double arithmetic.
__device__ __forceinline__ double plane_cost(const BoxN &l, const BoxN &m, const BoxN &r, double inv_area) {
  const double p1 = min1(__dmul_rn(area_d(l.lo, l.hi), inv_area));
  const double p2 = min1(__dmul_rn(area_d(m.lo, m.hi), inv_area));
  const double p3 = min1(__dmul_rn(area_d(r.lo, r.hi), inv_area));
  const double cost =
      __dadd_rn(__dadd_rn(__dmul_rn((double)l.n, p1), __dmul_rn((double)m.n, p2)), __dmul_rn((double)r.n, p3));
  return l.n == 0 || r.n == 0 ? __dmul_rn(cost, 0.8) : cost;
}
// The same in float: all terms are positive, so it is within 20u of the
// double cost (u = 2^-24) unless an area underflows or is not finite; lo / hi
// bound the double cost (-inf / +inf where that is not certain).
__device__ __forceinline__ void plane_cost_bounds(const BoxN &l, const BoxN &m, const BoxN &r, float inv_area,
                                                  float &lo, float &hi) {
  const BoxN *b[3] = {&l, &m, &r};
  float cost = 0.0f;
  bool sure = true;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (b[k]->n == 0u) continue;  // an empty box counts 0 * 1
    const float a = area_f(b[k]->lo, b[k]->hi), v = a * inv_area;
    sure = sure && a > 1e-30f && a < 1e30f;
    cost += (float)b[k]->n * (v < 1.0f ? v : 1.0f);
  }
  if (l.n == 0u || r.n == 0u) cost *= 0.8f;
  sure = sure && inv_area > 1e-30f && inv_area < 1e30f;
  lo = sure ? cost * (1.0f - 1.3e-6f) : -INFINITY;
  hi = sure ? cost * (1.0f + 1.3e-6f) : INFINITY;
}

// The least (cost, plane) of a warp.
__device__ __forceinline__ void warp_least(double &cost, int &plane) {
  for (int o = 16; o > 0; o >>= 1) {
    const double oc = __shfl_xor_sync(0xffffffffu, cost, o);
    const int oi = __shfl_xor_sync(0xffffffffu, plane, o);
    if (oc < cost || (oc == cost && oi < plane)) {
      cost = oc;
      plane = oi;
    }
  }
}
__device__ __forceinline__ float warp_min(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// min + i * (max - min) / tries, evaluated in float; 0 where no plane has a
// finite cost.
__device__ __forceinline__ double plane_position(int i, float nlo, float nhi, int tries) {
  if (i >= tries) return 0.0;
  const float ext = __fsub_rn(nhi, nlo);
  return (double)__fadd_rn(nlo, __fdiv_rn(__fmul_rn((float)i, ext), (float)tries));
}

// The split search of a node of at most 32 triangles, one warp: the boxes and
// their first / last planes wait in shared memory, every lane unites the
// boxes on the two sides of its plane (lane + 32 in a second round) and across
// it.  Every (node, axis) is bound by these 32 n updates; the double costs are
// made for a round only if one of its planes could still be the least.
// All three sizes together, bucket fill and scores before: 18.8 -> 6.3 ms for
// 1,098,576 triangles.
constexpr int kSmallWarps = 4;
__global__ void __launch_bounds__(kSmallWarps * 32) k_split_small(Dev D) {
  __shared__ float4 s_lo[kSmallWarps][32], s_hi[kSmallWarps][32];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const int64_t w = (int64_t)blockIdx.x * kSmallWarps + wi;
  if (w >= D.count[0]) return;  // whole warps
  const int64_t b = D.small[w];
  const int n = D.seg[b].y - (int)b, tries = D.htries[b];
  const unsigned mask = D.smask[b];
  float lo[3] = {0.0f, 0.0f, 0.0f}, hi[3] = {0.0f, 0.0f, 0.0f}, nlo[3], nhi[3];
  for (int c = 0; c < 3; ++c) {
    if (lane < n) {
      lo[c] = D.box[(b + lane) * 6 + c];
      hi[c] = D.box[(b + lane) * 6 + 3 + c];
    }
    nlo[c] = D.hbox[b * 6 + c];
    nhi[c] = D.hbox[b * 6 + 3 + c];
  }
  const float area = area_f(nlo, nhi), inv_f = 1.0f / area;
  const double inv_area = __ddiv_rn(1.0, (double)area);
  double best = INFINITY;
  int bi = 0x7FFFFFFF, ba = 0;
  for (int a = 0; a < 3; ++a) {
    if (mask & (1u << a)) continue;
    const double coef = D.hcoef[b * 3 + a];
    int first = 0, last = 0;  // planes >= first have the box on their left, planes < last on their right
    if (lane < n) {
      first = plane_of(__fsub_rn(hi[a], nlo[a]), coef, tries);
      last = plane_of(__fsub_rn(lo[a], nlo[a]), coef, tries);
    }
    __syncwarp();
    s_lo[wi][lane] = make_float4(lo[0], lo[1], lo[2], __int_as_float(first));
    s_hi[wi][lane] = make_float4(hi[0], hi[1], hi[2], __int_as_float(last));
    __syncwarp();
    for (int i0 = 0; i0 < tries; i0 += 32) {
      const int i = i0 + lane;
      BoxN L = box_empty(), M = box_empty(), R = box_empty();
      for (int t = 0; t < n; ++t) {
        const float4 p = s_lo[wi][t], q = s_hi[wi][t];
        BoxN x;
        x.lo[0] = p.x, x.lo[1] = p.y, x.lo[2] = p.z;
        x.hi[0] = q.x, x.hi[1] = q.y, x.hi[2] = q.z;
        x.n = 1u;
        const bool left = i >= __float_as_int(p.w), right = i < __float_as_int(q.w);
        if (left) box_unite(L, x);
        if (right) box_unite(R, x);  // (both: only where the planes per unit of length are infinite)
        if (!left && !right) box_unite(M, x);
      }
      float cl = INFINITY, ch = INFINITY;
      if (i < tries) plane_cost_bounds(L, M, R, inv_f, cl, ch);
      const float least = fminf(warp_min(ch), __double2float_ru(best));
      if (__ballot_sync(0xffffffffu, cl <= least) == 0u) continue;
      double cost = INFINITY;
      int plane = 0x7FFFFFFF;
      if (i < tries && cl <= least) {
        const double c = plane_cost(L, M, R, inv_area);
        if (c < INFINITY) {
          cost = c;
          plane = i;
        }
      }
      warp_least(cost, plane);
      if (cost < best) {
        best = cost;
        bi = plane;
        ba = a;
      }
    }
  }
  if (lane == 0) {
    D.haxis[b] = ba;
    D.hsplit[b] = plane_position(bi, nlo[ba], nhi[ba], tries);
    D.rflags[D.hid[b]] = (uint8_t)(ba + 1);
  }
}

// Adds triangle boxes to the buckets of one axis in shared memory (L at
// 0, M at tries, R at 2 tries, 7 words each): a box goes to the right bucket
// of its first candidate plane, the left one of its last, and the middle ones
// of the planes it straddles (NaN coordinates take no part, as in the
// reference's min / max).
__device__ __forceinline__ void bucket_add(uint32_t *r, const uint32_t *kl, const uint32_t *kh) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (kl[c] < r[c]) atomicMin(r + c, kl[c]);  // (a stale read only costs the atomic)
    if (kh[c] > r[3 + c]) atomicMax(r + 3 + c, kh[c]);
  }
  atomicAdd(r + 6, 1u);
}
__device__ __forceinline__ void fill_buckets(const Dev &D, uint32_t *sb, int64_t b, int64_t s0, int64_t s1, int a,
                                             int tries) {
  for (int i = threadIdx.x; i < 21 * tries; i += blockDim.x) {
    const int k = i % 7;
    sb[i] = k < 3 ? 0xFFFFFFFFu : 0u;
  }
  __syncthreads();
  const float nlo = D.hbox[b * 6 + a];
  const double coef = D.hcoef[b * 3 + a];
  for (int64_t s = s0 + threadIdx.x; s < s1; s += blockDim.x) {
    float lo[3], hi[3];
    uint32_t kl[3], kh[3];
    for (int c = 0; c < 3; ++c) {
      lo[c] = D.box[s * 6 + c];
      hi[c] = D.box[s * 6 + 3 + c];
      kl[c] = isnan(lo[c]) ? 0xFFFFFFFFu : okey(lo[c]);
      kh[c] = isnan(hi[c]) ? 0u : okey(hi[c]);
    }
    const int lefts_begin = plane_of(__fsub_rn(hi[a], nlo), coef, tries);
    const int rights_end = plane_of(__fsub_rn(lo[a], nlo), coef, tries);
    if (rights_end > 0) bucket_add(sb + 7 * (2 * tries + rights_end - 1), kl, kh);
    if (lefts_begin < tries) bucket_add(sb + 7 * lefts_begin, kl, kh);
    for (int j = rights_end; j < lefts_begin; ++j) bucket_add(sb + 7 * (tries + j), kl, kh);
  }
  __syncthreads();
}

// One axis of one node's split search over its filled buckets
// (_DetermineBestSplit, :566-608), one warp: lane l takes a contiguous slice
// of the candidate planes.  The right buckets' suffix unions and the left
// buckets' prefix unions come from warp scans of the slices' unions and are
// stored back in place, decoded; then the costs: the float ones first, the
// double ones of the planes that could be the least.
__device__ __forceinline__ void store_box(uint32_t *r, const BoxN &b) {
  for (int c = 0; c < 3; ++c) {
    r[c] = __float_as_uint(b.lo[c]);
    r[3 + c] = __float_as_uint(b.hi[c]);
  }
  r[6] = b.n;
}
__device__ __forceinline__ BoxN load_box(const uint32_t *r) {
  BoxN b;
  for (int c = 0; c < 3; ++c) {
    b.lo[c] = __uint_as_float(r[c]);
    b.hi[c] = __uint_as_float(r[3 + c]);
  }
  b.n = r[6];
  return b;
}
__device__ __forceinline__ void score_axis(const Dev &D, int64_t s, int a, uint32_t *L) {
  const int lane = threadIdx.x & 31;
  const int tries = D.htries[s];
  uint32_t *M = L + (int64_t)tries * 7, *R = M + (int64_t)tries * 7;
  const int per = (tries + 31) / 32, i0 = min(tries, lane * per), i1 = min(tries, i0 + per);
  BoxN ls = box_empty(), rs = box_empty();
  for (int i = i0; i < i1; ++i) {
    box_unite(ls, box_keys(L + (int64_t)i * 7));
    box_unite(rs, box_keys(R + (int64_t)i * 7));
  }
  // inclusive prefix of the left slices, inclusive suffix of the right ones
  for (int o = 1; o < 32; o <<= 1) {
    const BoxN u = box_shfl_up(ls, o), d = box_shfl_down(rs, o);
    if (lane >= o) box_unite(ls, u);
    if (lane + o < 32) box_unite(rs, d);
  }
  BoxN lp = box_shfl_up(ls, 1), rp = box_shfl_down(rs, 1);  // exclusive
  if (lane == 0) lp = box_empty();
  if (lane == 31) rp = box_empty();
  for (int i = i1 - 1; i >= i0; --i) {
    uint32_t *r = R + (int64_t)i * 7;
    box_unite(rp, box_keys(r));
    store_box(r, rp);
  }
  const float *nlo = D.hbox + s * 6, *nhi = nlo + 3;
  const float area = area_f(nlo, nhi), inv_f = 1.0f / area;
  const double inv_area = __ddiv_rn(1.0, (double)area);
  float least = INFINITY;
  for (int i = i0; i < i1; ++i) {
    uint32_t *l = L + (int64_t)i * 7;
    box_unite(lp, box_keys(l));
    store_box(l, lp);
    float cl, ch;
    plane_cost_bounds(lp, box_keys(M + (int64_t)i * 7), load_box(R + (int64_t)i * 7), inv_f, cl, ch);
    least = fminf(least, ch);
  }
  least = warp_min(least);
  double best = INFINITY;
  int bi = 0x7FFFFFFF;
  for (int i = i0; i < i1; ++i) {
    const BoxN l = load_box(L + (int64_t)i * 7), m = box_keys(M + (int64_t)i * 7), r = load_box(R + (int64_t)i * 7);
    float cl, ch;
    plane_cost_bounds(l, m, r, inv_f, cl, ch);
    if (cl <= least) {
      const double cost = plane_cost(l, m, r, inv_area);
      if (cost < best) {
        best = cost;
        bi = i;
      }
    }
  }
  warp_least(best, bi);
  if (lane == 0) {
    D.bcost[3 * s + a] = best;
    D.bpos[3 * s + a] = plane_position(bi, nlo[a], nhi[a], tries);
  }
}

// A node of 33 to 4,096 triangles, one block per axis.
__global__ void __launch_bounds__(128) k_split_mid(Dev D) {
  __shared__ uint32_t sb[21 * kTries];
  const int64_t k = blockIdx.x / 3u;
  const int a = (int)(blockIdx.x % 3u);
  if (k >= D.count[1]) return;
  const int64_t b = D.mid[k];
  if (D.smask[b] & (1u << a)) {
    if (threadIdx.x == 0) {
      D.bcost[3 * b + a] = INFINITY;
      D.bpos[3 * b + a] = 0.0;
    }
    return;
  }
  fill_buckets(D, sb, b, b, D.seg[b].y, a, D.htries[b]);
  if (threadIdx.x < 32) score_axis(D, b, a, sb);
}

// Larger nodes: their buckets emptied, filled chunk by chunk (the chunk's own
// buckets merged into them) and searched.
__global__ void k_big_init(Dev D) {
  const int64_t total = (int64_t)D.count[2] * 9 * kTries * 7;
  for (int64_t i = (int64_t)blockIdx.x * kB + threadIdx.x; i < total; i += (int64_t)gridDim.x * kB)
    D.buckets[i] = i % 7 < 3 ? 0xFFFFFFFFu : 0u;
}
__global__ void __launch_bounds__(256) k_fill_big(Dev D) {
  __shared__ uint32_t sb[21 * kTries];
  const int64_t k = blockIdx.x / 3u;
  const int a = (int)(blockIdx.x % 3u);
  if (k >= D.count[3]) return;
  const int64_t b = D.chunks[k].x, s0 = b + (int64_t)D.chunks[k].y * kMid;
  if (D.smask[b] & (1u << a)) return;
  fill_buckets(D, sb, b, s0, min((int64_t)D.seg[b].y, s0 + kMid), a, kTries);
  uint32_t *g = D.buckets + ((int64_t)D.hbase[b] + (int64_t)a * 3 * kTries) * 7;
  for (int i = threadIdx.x; i < 3 * kTries; i += blockDim.x) {
    const uint32_t *r = sb + 7 * i;
    if (r[6] == 0u) continue;
    for (int c = 0; c < 3; ++c) {
      atomicMin(g + 7 * i + c, r[c]);
      atomicMax(g + 7 * i + 3 + c, r[3 + c]);
    }
    atomicAdd(g + 7 * i + 6, r[6]);
  }
}
__global__ void __launch_bounds__(32) k_score_big(Dev D) {
  const int64_t k = blockIdx.x / 3u;
  const int a = (int)(blockIdx.x % 3u);
  if (k >= D.count[2]) return;
  const int64_t s = D.big[k];
  if (D.smask[s] & (1u << a)) {
    if (threadIdx.x == 0) {
      D.bcost[3 * s + a] = INFINITY;
      D.bpos[3 * s + a] = 0.0;
    }
    return;
  }
  score_axis(D, s, a, D.buckets + ((int64_t)D.hbase[s] + (int64_t)a * 3 * kTries) * 7);
}

// The split axis of the mid and big nodes: the lowest of the axes with the
// least cost.
__global__ void k_choose(Dev D) {
  const int64_t k = (int64_t)blockIdx.x * kB + threadIdx.x;
  const int n_mid = D.count[1];
  if (k >= (int64_t)n_mid + D.count[2]) return;
  const int64_t s = k < n_mid ? D.mid[k] : D.big[k - n_mid];
  const double c0 = D.bcost[3 * s], c1 = D.bcost[3 * s + 1], c2 = D.bcost[3 * s + 2];
  int a;
  if (c0 <= c1 && c0 <= c2)
    a = 0;
  else if (c1 <= c0 && c1 <= c2)
    a = 1;
  else
    a = 2;
  D.haxis[s] = a;
  D.hsplit[s] = D.bpos[3 * s + a];
  D.rflags[D.hid[s]] = (uint8_t)(a + 1);
}

// Classes of the partition (Node::Node, :644-673): 0 entirely below the
// split, 2 entirely above, 1 straddling; packed counts of the right class
// (low word) and of the others (high word) for the scan.
__global__ void k_classify(Dev D) {
  const int64_t s = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (s > D.n) return;
  uint64_t v = 0;
  if (s < D.n) {
    const int b = D.seg[s].x;
    if (b >= 0 && !D.hleaf[b]) {
      const int a = D.haxis[b];
      const double split = D.hsplit[b];
      uint8_t c;
      if ((double)D.box[s * 6 + 3 + a] < split)
        c = 0;
      else if ((double)D.box[s * 6 + a] > split)
        c = 2;
      else
        c = 1;
      D.cls[s] = c;
      v = c == 2 ? 1ull : (1ull << 32);
    }
  }
  D.cnt[s] = v;
}

__device__ __forceinline__ uint32_t lo32(uint64_t v) { return (uint32_t)v; }
__device__ __forceinline__ uint32_t hi32(uint64_t v) { return (uint32_t)(v >> 32); }

// The back stream's runs (index u = e - 1 - slot): T[r] = u of its r-th
// element that is not right-class; J[r] = front index of the r-th
// right-class element of the front stream.
__global__ void k_runs(Dev D) {
  const int64_t s = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (s >= D.n) return;
  const int2 g = D.seg[s];
  if (g.x < 0 || D.hleaf[g.x]) return;
  const uint32_t b = (uint32_t)g.x, e = (uint32_t)g.y;
  if (D.cls[s] == 2) {
    const uint32_t r = lo32(D.cnt[s]) - lo32(D.cnt[b]);
    D.jarr[b + r] = (uint32_t)s - b;
  } else {
    const uint32_t r = hi32(D.cnt[e]) - hi32(D.cnt[s + 1]);
    D.tarr[b + r] = e - 1 - (uint32_t)s;
  }
}

// Processing step of every element: the front element j comes after j
// front elements and the runs of the right-class front elements before it;
// a back element comes after its run's trigger and its run's earlier
// elements.  ord[b + step] = slot.
__device__ __forceinline__ uint32_t front_step(const Dev &D, uint32_t b, uint32_t j, uint32_t a, uint32_t cnt_n,
                                               uint32_t nn) {
  if (a == 0) return j;
  if (a - 1 < cnt_n) return j + D.tarr[b + a - 1] + 1;
  return nn + 1;  // more triggers than runs: never reached
}
__global__ void k_steps(Dev D) {
  const int64_t s = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (s >= D.n) return;
  const int2 g = D.seg[s];
  if (g.x < 0 || D.hleaf[g.x]) return;
  const uint32_t b = (uint32_t)g.x, e = (uint32_t)g.y, nn = e - b, j = (uint32_t)s - b;
  const uint64_t cb = D.cnt[b], ce = D.cnt[e];
  const uint32_t cnt_n = hi32(ce) - hi32(cb), cnt_r = lo32(ce) - lo32(cb);
  uint32_t step = front_step(D, b, j, lo32(D.cnt[s]) - lo32(cb), cnt_n, nn);
  if (step >= nn) {
    const uint32_t u = e - 1 - (uint32_t)s;
    const uint32_t r = hi32(ce) - hi32(D.cnt[s + 1]);
    const uint32_t start = r == 0 ? 0u : D.tarr[b + r - 1] + 1;
    step = 0xFFFFFFFFu;
    if (r < cnt_r) {
      const uint32_t jr = D.jarr[b + r];
      const uint32_t sr = front_step(D, b, jr, r, cnt_n, nn);
      if (sr < nn) step = sr + 1 + (u - start);
    }
  }
  if (step >= nn) {
    atomicOr(D.err, 1);
    return;
  }
  D.ord[b + step] = (uint32_t)s;
}

// Every position of an internal node must have received an element.
__global__ void k_steps_check(Dev D) {
  const int64_t p = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (p >= D.n) return;
  const int b = D.seg[p].x;
  if (b >= 0 && !D.hleaf[b] && D.ord[p] == 0xFFFFFFFFu) atomicOr(D.err, 2);
}

// In processing order: packed counts (left, right) and (left or middle, 0).
__global__ void k_order_flags(Dev D) {
  const int64_t p = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (p > D.n) return;
  uint64_t v = 0, w = 0;
  if (p < D.n) {
    const int b = D.seg[p].x;
    const uint32_t s = b >= 0 && !D.hleaf[b] ? D.ord[p] : 0xFFFFFFFFu;
    if (s < (uint64_t)D.n) {  // (an unfilled position is already an error)
      const uint8_t c = D.cls[s];
      v = c == 0 ? 1ull : (c == 2 ? (1ull << 32) : 0ull);
      w = c != 2 ? 1ull : 0ull;
    }
  }
  D.cnt2[p] = v;
  D.cnt3[p] = w;
}

// Destinations: the r-th left element (in processing order) to b + r, the
// r-th right one to e - 1 - r; I[r] = elements of the left-or-middle
// classes processed before the r-th left one (the block's end when it
// moves the middle block's front); a middle element starts at the block
// position lm = left-or-middle elements before it.
__global__ void k_dest(Dev D) {
  const int64_t p = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (p >= D.n) return;
  const int2 g = D.seg[p];
  if (g.x < 0 || D.hleaf[g.x]) return;
  const uint32_t b = (uint32_t)g.x, e = (uint32_t)g.y;
  const uint64_t cb = D.cnt2[b], cp = D.cnt2[p];
  const uint32_t rl = lo32(cp) - lo32(cb), rr = hi32(cp) - hi32(cb);
  const uint32_t lm = (uint32_t)(D.cnt3[p] - D.cnt3[b]);
  const uint32_t s = D.ord[p];
  if (s >= (uint64_t)D.n) return;
  const uint8_t c = D.cls[s];
  if (c == 0) {
    D.dest[s] = b + rl;
    D.iarr[b + rl] = lm;
  } else if (c == 2) {
    D.dest[s] = e - 1 - rr;
  } else {
    D.lmb[p] = lm;
  }
  if (p == b) {
    const uint64_t ce = D.cnt2[e];
    D.hnl[b] = lo32(ce) - lo32(cb);
    D.hnr[b] = hi32(ce) - hi32(cb);
  }
}

// The middle block's moves as a function on block positions: a position
// below the number of left elements moves to I of it, the others stay.
__global__ void k_jump_init(Dev D) {
  const int64_t p = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (p >= D.n) return;
  const int b = D.seg[p].x;
  if (b < 0 || D.hleaf[b]) return;
  const uint32_t x = (uint32_t)p - (uint32_t)b;
  D.f0[p] = x < D.hnl[b] ? D.iarr[p] : x;
}
// Eight applications a round (253 rounds of two over a 1,098,576-triangle
// build took 2.2 ms).
constexpr int kJumps = 8;
__global__ void k_jump(Dev D, const uint32_t *__restrict__ fin, uint32_t *__restrict__ fout) {
  const int64_t p = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (p >= D.n) return;
  const int2 g = D.seg[p];
  if (g.x < 0 || D.hleaf[g.x]) return;
  uint32_t v = fin[p];
#pragma unroll
  for (int k = 1; k < kJumps; ++k) {
    if (v >= (uint32_t)(g.y - g.x)) {  // only after an inconsistent step map
      atomicOr(D.err, 4);
      break;
    }
    const uint32_t x = fin[(uint32_t)g.x + v];
    if (x == v) break;
    v = x;
  }
  fout[p] = v;
}
__global__ void k_dest_middle(Dev D, const uint32_t *__restrict__ f) {
  const int64_t p = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (p >= D.n) return;
  const int b = D.seg[p].x;
  if (b < 0 || D.hleaf[b]) return;
  const uint32_t s = D.ord[p];
  if (s >= (uint64_t)D.n || D.cls[s] != 1) return;
  const uint32_t x = D.lmb[p], nn = (uint32_t)(D.seg[p].y - b);
  const uint32_t d = x < nn ? f[(uint32_t)b + x] : 0xFFFFFFFFu;
  if (d >= nn) {
    atomicOr(D.err, 4);
    return;
  }
  D.dest[s] = (uint32_t)b + d;
}

__global__ void k_scatter(Dev D) {
  const int64_t s = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (s >= D.n) return;
  const int2 g = D.seg[s];
  const int64_t d = (g.x >= 0 && !D.hleaf[g.x]) ? (int64_t)D.dest[s] : s;
  if (d < g.x || (g.x >= 0 && d >= g.y) || d >= D.n) {  // unset: only after an inconsistent step map
    atomicOr(D.err, 8);
    return;
  }
  for (int c = 0; c < 6; ++c) D.box2[d * 6 + c] = D.box[s * 6 + c];
  D.perm2[d] = D.perm[s];
}

// Next level's node of every position (in the partitioned order): the
// left, middle or right child's range, its middle-split axes and parent.
__global__ void k_children(Dev D) {
  const int64_t p = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (p >= D.n) return;
  const int2 g = D.seg[p];
  if (g.x < 0) return;
  if (D.hleaf[g.x]) {
    D.seg[p] = make_int2(-1, -1);
    return;
  }
  const int b = g.x, e = g.y;
  const int l = b + (int)D.hnl[b], r = e - (int)D.hnr[b];
  D.spar[p] = D.hid[b];
  if ((int)p < l) {
    D.seg[p] = make_int2(b, l);
    D.sord[p] = 0;
  } else if ((int)p < r) {
    D.seg[p] = make_int2(l, r);
    D.sord[p] = 1;
    D.smask[p] = (uint8_t)(D.smask[p] | (1u << D.haxis[b]));
  } else {
    D.seg[p] = make_int2(r, e);
    D.sord[p] = 2;
  }
}

// Flattening: the tree in pre-order, a node's present children in
// consecutive places, so that a child's subtree starts where those of its
// left siblings end.  Levels bottom up give every subtree's size (the root
// left out), levels top down the places.  Bound by its launches (28 for 21
// levels): 0.15 ms for 1,098,576 triangles, and 0.02 for the slots, all of it
// in device memory.  On the host one walk over the records took 5.4 ms, the
// slots 4.2, their copies to the host and back 2.5.  A launch takes one level, or several of at most kNarrow nodes
// in one block (the first and last levels are narrow: a launch each costs
// more than their work).
constexpr int kNarrow = 1024;

__global__ void k_subtree(Dev D, const int64_t *__restrict__ level, int l0, int l1, uint32_t *sub) {
  for (int l = l1 - 1; l >= l0; --l) {
    for (int64_t id = level[l] + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; id < level[l + 1];
         id += (int64_t)gridDim.x * blockDim.x) {
      uint32_t n = 0;
      for (int c = 0; c < 3; ++c) {
        const int32_t ch = D.rchild[id * 3 + c];
        if (ch >= 0) n += 1 + sub[ch];
      }
      sub[id] = n;
    }
    __syncthreads();
  }
}

// place: a node's own place and its first child's.
__global__ void k_flatten(Dev D, const int64_t *__restrict__ level, int l0, int l1, const uint32_t *__restrict__ sub,
                          uint2 *place, int64_t n_nodes, DevNode *__restrict__ nodes) {
  for (int l = l0; l < l1; ++l) {
    for (int64_t id = level[l] + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; id < level[l + 1];
         id += (int64_t)gridDim.x * blockDim.x) {
      const uint2 at = id == 0 ? make_uint2(0, 1) : place[id];
      if (at.x >= n_nodes) {  // no parent: only after an inconsistent step map
        atomicOr(D.err, 16);
        continue;
      }
      DevNode dn;
      for (int k = 0; k < 3; ++k) {
        dn.lo[k] = D.rbox[id * 6 + k];
        dn.hi[k] = D.rbox[id * 6 + 3 + k];
      }
      const uint32_t flags = D.rflags[id];
      if (flags == 0) {
        dn.a = D.rtb[id];
        dn.b = (D.rte[id] - D.rtb[id]) << 8;
      } else {
        int32_t ch[3];
        uint32_t mask = 0;
        for (int c = 0; c < 3; ++c) {
          ch[c] = D.rchild[id * 3 + c];
          if (ch[c] >= 0) mask |= 1u << c;
        }
        uint32_t slot = at.y, first = at.y + __popc(mask);
        for (int c = 0; c < 3; ++c)
          if (ch[c] >= 0) {
            place[ch[c]] = make_uint2(slot++, first);
            first += sub[ch[c]];
          }
        dn.a = at.y;
        dn.b = flags | (mask << 2);
      }
      nodes[at.x] = dn;
    }
    __syncthreads();
  }
}

__global__ void k_tris(Dev D, const DevTri *__restrict__ src, DevTri *__restrict__ tris) {
  const int64_t i = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (i >= D.n) return;
  const float4 *r = (const float4 *)(src + D.perm[i]);
  float4 *w = (float4 *)(tris + i);
  const float4 c = r[2];
  w[0] = r[0];
  w[1] = r[1];
  w[2] = make_float4(c.x, c.y, c.z, __int_as_float((int32_t)i));
}

// A slot's primitive and mesh triangle.
__global__ void k_slot_ids(const DevTri *__restrict__ tris, int64_t n, int32_t *prim, int32_t *tri) {
  const int64_t i = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (i >= n) return;
  prim[i] = tris[i].prim;
  tri[i] = tris[i].tri;
}

// The leaf of every light triangle: each leaf looks its triangles up in the
// sorted keys.  A light triangle's record stays as it is if no leaf holds it.
__global__ void k_light_leaves(const DevNode *__restrict__ nodes, int64_t n_nodes, const LeafExt *__restrict__ ext,
                               const DevTri *__restrict__ tris, const int32_t *__restrict__ prim_first,
                               const LightKey *__restrict__ keys, int64_t n_keys, float *__restrict__ leaf) {
  const int64_t id = (int64_t)blockIdx.x * kB + threadIdx.x;
  if (id >= n_nodes) return;
  const DevNode nd = nodes[id];
  if ((nd.b & 3u) != 0u) return;
  const bool x = (nd.b & kLeafExt) != 0;
  const uint32_t first = x ? ext[nd.a].tri_first : nd.a, count = x ? ext[nd.a].tri_count : nd.b >> 8;
  for (uint32_t k = 0; k < count; ++k) {
    const DevTri &t = tris[first + k];
    if (t.prim < 0) continue;  // a shared mesh's slot belongs to no one primitive
    const int32_t key = prim_first[t.prim] + t.tri;
    int64_t lo = 0, hi = n_keys;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (keys[mid].tri < key) lo = mid + 1;
      else hi = mid;
    }
    for (; lo < n_keys && keys[lo].tri == key; ++lo) {
      float *o = leaf + 8 * (int64_t)keys[lo].light;
      for (int c = 0; c < 3; ++c) {
        o[c] = nd.lo[c];
        o[3 + c] = nd.hi[c];
      }
      o[6] = __uint_as_float(first);
      o[7] = __uint_as_float(count);
    }
  }
}

// Three vertices per triangle of a mesh; the triangles TriangleMesh drops
// (k_keep) get indices that it drops too.
void gather_vertices(const MeshIn &m, float *v, int32_t *ix) {
  for (int64_t t = 0; t < m.n_triangles; ++t, v += 9, ix += 3) {
    const int32_t *s = m.triangles + 3 * t;
    bool kept = s[0] != s[1] && s[0] != s[2] && s[1] != s[2];
    for (int k = 0; k < 3; ++k) kept = kept && s[k] >= 0 && s[k] < m.n_vertices;
    for (int k = 0; k < 3; ++k) {
      ix[k] = kept ? (int32_t)(3 * t + k) : -1;
      if (kept) std::memcpy(v + 3 * k, m.vertices + 3 * (int64_t)s[k], 12);
    }
  }
}

inline size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

cudaError_t build_accel_tree_gpu(const std::vector<MeshJob> &jobs, int64_t min_n, cudaStream_t st, DeviceTree &out) {
  out = DeviceTree();
  // The meshes' arrays: one copy for all the small ones, one each for the
  // others (a copy costs some microseconds, whatever it moves).
  constexpr size_t kOwnCopy = 1 << 16;
  // A mesh of more vertices than this per triangle -- the parts of a scene
  // often share one array -- gives only its triangles' own, so that a build
  // copies and holds at most 396 bytes a triangle (600,000 triangles in 300
  // parts of one array of 1.8M vertices: 54.8 ms with the array copied for
  // each part, 18.3 without; gathering takes what copying 56 vertices a
  // triangle does).
  constexpr int64_t kSpareVertices = 32;
  std::vector<std::vector<float>> own_v;
  std::vector<std::vector<int32_t>> own_ix;
  struct Part {
    const void *src;
    size_t bytes, at;
  };
  std::vector<Part> parts;
  std::vector<DevMesh> meshes;
  int64_t n = 0;
  for (const MeshJob &j : jobs) {
    if (j.m->n_triangles <= 0) continue;
    DevMesh d{};
    d.n_vertices = std::max<int64_t>(j.m->n_vertices, 0);
    d.t0 = n;
    d.prim = j.prim;
    d.has_m = j.xf ? 1 : 0;
    if (j.xf) std::memcpy(d.m, j.xf, sizeof(d.m));
    const float *v = j.m->vertices;
    const int32_t *ix = j.m->triangles;
    if (j.m->n_triangles <= INT32_MAX / 3 && d.n_vertices / kSpareVertices > j.m->n_triangles) {
      own_v.emplace_back((size_t)j.m->n_triangles * 9);
      own_ix.emplace_back((size_t)j.m->n_triangles * 3);
      gather_vertices(*j.m, own_v.back().data(), own_ix.back().data());
      v = own_v.back().data();
      ix = own_ix.back().data();
      d.n_vertices = 3 * j.m->n_triangles;
    }
    meshes.push_back(d);
    parts.push_back(Part{v, (size_t)d.n_vertices * 12, 0});
    parts.push_back(Part{ix, (size_t)j.m->n_triangles * 12, 0});
    n += j.m->n_triangles;
  }
  if (n <= 0 || n > (int64_t)INT32_MAX / 2) return cudaErrorInvalidValue;
  size_t staged = al256(meshes.size() * sizeof(DevMesh)), mesh_bytes = 0;
  for (Part &p : parts)
    if (p.bytes < kOwnCopy) {
      p.at = staged;
      staged += (p.bytes + 15) & ~(size_t)15;
    }
  mesh_bytes = al256(staged);
  for (Part &p : parts)
    if (p.bytes >= kOwnCopy) {
      p.at = mesh_bytes;
      mesh_bytes += al256(p.bytes);
    }
  Dev D{};
  size_t n1 = (size_t)n + 1;
  const size_t nb = (n1 + kB - 1) / kB;
  size_t total = 0;
  std::vector<std::pair<void **, size_t>> plan;
  auto want = [&](void *pp, size_t bytes) {
    plan.push_back({(void **)pp, bytes});
    total += al256(bytes);
  };
  size_t nn = (size_t)n;
  want(&D.box, nn * 24);
  want(&D.box2, nn * 24);
  want(&D.perm, nn * 4);
  want(&D.perm2, nn * 4);
  want(&D.seg, nn * 8);
  want(&D.smask, nn);
  want(&D.sord, nn);
  want(&D.spar, nn * 4);
  want(&D.hkeys, nn * 48);
  want(&D.hbox, nn * 24);
  want(&D.hcoef, nn * 24);
  want(&D.hsplit, nn * 8);
  want(&D.hid, nn * 4);
  want(&D.htries, nn * 4);
  want(&D.haxis, nn * 4);
  want(&D.hnl, nn * 4);
  want(&D.hnr, nn * 4);
  want(&D.hleaf, nn);
  want(&D.bcost, nn * 24);
  want(&D.bpos, nn * 24);
  want(&D.hbase, nn * 4);
  want(&D.small, (nn / (kLeafMax + 1) + 1) * 4);
  want(&D.mid, (nn / (kSmall + 1) + 1) * 4);
  want(&D.big, (nn / (kMid + 1) + 1) * 4);
  want(&D.chunks, (nn / kMid + nn / (kMid + 1) + 2) * 8);
  want(&D.buckets, (nn / (kMid + 1) + 1) * 9 * kTries * 28);
  want(&D.count, 256);
  want(&D.cls, nn);
  want(&D.cnt, n1 * 8);
  want(&D.cnt2, n1 * 8);
  want(&D.cnt3, n1 * 8);
  want(&D.sums, nb * 8);
  want(&D.tarr, nn * 4);
  want(&D.jarr, nn * 4);
  want(&D.ord, nn * 4);
  want(&D.iarr, nn * 4);
  want(&D.f0, nn * 4);
  want(&D.f1, nn * 4);
  want(&D.lmb, nn * 4);
  want(&D.dest, nn * 4);
  want(&D.err, 256);
  want(&D.maxseg, 256);
  want(&D.n_leaves, 256);
  char *mesh_mem = nullptr;
  DevTri *src = nullptr;
  want(&mesh_mem, mesh_bytes);
  want(&src, nn * sizeof(DevTri));
  char *arena = nullptr;
  cudaError_t e = cudaMalloc(&arena, total);
  if (e != cudaSuccess) return e;
  {
    char *w = arena;
    for (auto &pr : plan) {
      *pr.first = w;
      w += al256(pr.second);
    }
  }
  // node records, grown as levels add nodes
  int64_t cap = 0, n_nodes = 0;
  auto grow = [&](int64_t need) -> cudaError_t {
    if (need <= cap) return cudaSuccess;
    int64_t nc = std::max<int64_t>(need, cap + cap / 2 + (int64_t)1024);
    float *rbox = nullptr;
    uint32_t *rtb = nullptr, *rte = nullptr;
    uint8_t *rflags = nullptr;
    int32_t *rchild = nullptr;
    cudaError_t g;
    if ((g = cudaMalloc(&rbox, (size_t)nc * 24)) != cudaSuccess || (g = cudaMalloc(&rtb, (size_t)nc * 4)) != cudaSuccess ||
        (g = cudaMalloc(&rte, (size_t)nc * 4)) != cudaSuccess || (g = cudaMalloc(&rflags, (size_t)nc)) != cudaSuccess ||
        (g = cudaMalloc(&rchild, (size_t)nc * 12)) != cudaSuccess) {
      cudaFree(rbox);
      cudaFree(rtb);
      cudaFree(rte);
      cudaFree(rflags);
      cudaFree(rchild);
      return g;
    }
    if (n_nodes > 0) {
      cudaMemcpyAsync(rbox, D.rbox, (size_t)n_nodes * 24, cudaMemcpyDeviceToDevice, st);
      cudaMemcpyAsync(rtb, D.rtb, (size_t)n_nodes * 4, cudaMemcpyDeviceToDevice, st);
      cudaMemcpyAsync(rte, D.rte, (size_t)n_nodes * 4, cudaMemcpyDeviceToDevice, st);
      cudaMemcpyAsync(rflags, D.rflags, (size_t)n_nodes, cudaMemcpyDeviceToDevice, st);
      cudaMemcpyAsync(rchild, D.rchild, (size_t)n_nodes * 12, cudaMemcpyDeviceToDevice, st);
    }
    if ((g = cudaStreamSynchronize(st)) != cudaSuccess) return g;
    cudaFree(D.rbox);
    cudaFree(D.rtb);
    cudaFree(D.rte);
    cudaFree(D.rflags);
    cudaFree(D.rchild);
    D.rbox = rbox;
    D.rtb = rtb;
    D.rte = rte;
    D.rflags = rflags;
    D.rchild = rchild;
    cap = nc;
    return cudaSuccess;
  };
  auto release = [&]() {
    cudaFree(D.rbox);
    cudaFree(D.rtb);
    cudaFree(D.rte);
    cudaFree(D.rflags);
    cudaFree(D.rchild);
    cudaFree(arena);
  };
  uint64_t *h_count = nullptr;
  if ((e = cudaMallocHost(&h_count, 16)) != cudaSuccess) {
    release();
    return e;
  }
  const int n_meshes = (int)meshes.size();
  for (size_t k = 0; k < parts.size(); ++k) {
    const void *at = mesh_mem + parts[k].at;
    if (k & 1) meshes[k / 2].ix = (const int32_t *)at;
    else meshes[k / 2].v = (const float *)at;
  }
  std::vector<char> stage(staged);
  std::memcpy(stage.data(), meshes.data(), meshes.size() * sizeof(DevMesh));
  for (const Part &p : parts)
    if (p.bytes > 0 && p.bytes < kOwnCopy) std::memcpy(stage.data() + p.at, p.src, p.bytes);
  e = cudaMemcpyAsync(mesh_mem, stage.data(), staged, cudaMemcpyHostToDevice, st);
  for (const Part &p : parts)
    if (e == cudaSuccess && p.bytes >= kOwnCopy)
      e = cudaMemcpyAsync(mesh_mem + p.at, p.src, p.bytes, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(D.err, 0, 4, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(D.n_leaves, 0, 8, st);
  const DevMesh *d_meshes = (const DevMesh *)mesh_mem;
  const int64_t total_tris = n;
  if (e == cudaSuccess) {
    k_keep<<<grid_of(total_tris + 1), kB, 0, st>>>(d_meshes, n_meshes, total_tris, D.cnt);
    e = scan64(D.cnt, total_tris + 1, D.sums, st);
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(h_count, D.cnt + total_tris, 8, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) {
    n = (int64_t)h_count[0];
    if (n < std::max<int64_t>(min_n, 1)) {
      out.few = true;
      cudaFreeHost(h_count);
      release();
      return cudaSuccess;
    }
  }
  D.n = n;
  nn = (size_t)n;
  n1 = nn + 1;
  const unsigned gn = grid_of(n), gn1 = grid_of((int64_t)n1);
  if (e == cudaSuccess) e = grow(std::max<int64_t>(2 * n, 1024));
  if (e == cudaSuccess) {
    k_collect<<<grid_of(total_tris), kB, 0, st>>>(D, d_meshes, n_meshes, total_tris, src);
    e = cudaGetLastError();
  }
  std::vector<int64_t> level_base;  // first node of every level, and the end
  int depth = 0;
  for (; e == cudaSuccess; ++depth) {
    level_base.push_back(n_nodes);
    if ((e = cudaMemsetAsync(D.maxseg, 0, 4, st)) != cudaSuccess) break;
    k_heads<<<gn1, kB, 0, st>>>(D);
    if ((e = scan64(D.cnt, (int64_t)n1, D.sums, st)) != cudaSuccess) break;
    if ((e = cudaMemcpyAsync(h_count, D.cnt + n, 8, cudaMemcpyDeviceToHost, st)) != cudaSuccess) break;
    if ((e = cudaMemcpyAsync(h_count + 1, D.err, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess) break;
    if ((e = cudaMemcpyAsync((char *)(h_count + 1) + 4, D.maxseg, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess) break;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) break;
    const int64_t level_nodes = (int64_t)h_count[0];
    if (level_nodes == 0 || (uint32_t)h_count[1] != 0) break;
    // a middle element's chain stays inside its node: kJumps^rounds >= its size
    const int64_t maxseg = (int64_t)(h_count[1] >> 32);
    int rounds = 1;
    for (int64_t reach = kJumps; reach < maxseg; reach *= kJumps) ++rounds;
    if ((e = grow(n_nodes + level_nodes)) != cudaSuccess) break;
    k_node_box<<<gn, kB, 0, st>>>(D);
    if ((e = cudaMemsetAsync(D.count, 0, 16, st)) != cudaSuccess) break;
    k_head_setup<<<gn, kB, 0, st>>>(D, n_nodes, depth);
    n_nodes += level_nodes;
    // at most this many nodes of each size; the kernels' blocks past the
    // level's own numbers return at once
    const int64_t most_mid = std::min(level_nodes, n / (kSmall + 1)), most_big = std::min(level_nodes, n / (kMid + 1));
    const int64_t most_small = maxseg > kLeafMax ? std::min(level_nodes, n / (kLeafMax + 1)) : 0;
    if (maxseg > kMid) {
      k_big_init<<<512, kB, 0, st>>>(D);
      k_fill_big<<<(unsigned)(3 * (n / kMid + most_big + 1)), 256, 0, st>>>(D);
      k_score_big<<<(unsigned)(3 * most_big), 32, 0, st>>>(D);
    }
    if (maxseg > kSmall) {
      if (most_mid > 0) k_split_mid<<<(unsigned)(3 * most_mid), 128, 0, st>>>(D);
      if (most_mid + most_big > 0) k_choose<<<grid_of(most_mid + most_big), kB, 0, st>>>(D);
    }
    if (most_small > 0) k_split_small<<<(unsigned)((most_small + kSmallWarps - 1) / kSmallWarps), kSmallWarps * 32, 0, st>>>(D);
    k_classify<<<gn1, kB, 0, st>>>(D);
    if ((e = scan64(D.cnt, (int64_t)n1, D.sums, st)) != cudaSuccess) break;
    k_runs<<<gn, kB, 0, st>>>(D);
    if ((e = cudaMemsetAsync(D.ord, 0xFF, nn * 4, st)) != cudaSuccess) break;
    if ((e = cudaMemsetAsync(D.dest, 0xFF, nn * 4, st)) != cudaSuccess) break;
    k_steps<<<gn, kB, 0, st>>>(D);
    k_steps_check<<<gn, kB, 0, st>>>(D);
    k_order_flags<<<gn1, kB, 0, st>>>(D);
    if ((e = scan64(D.cnt2, (int64_t)n1, D.sums, st)) != cudaSuccess) break;
    if ((e = scan64(D.cnt3, (int64_t)n1, D.sums, st)) != cudaSuccess) break;
    k_dest<<<gn, kB, 0, st>>>(D);
    k_jump_init<<<gn, kB, 0, st>>>(D);
    uint32_t *fa = D.f0, *fb = D.f1;
    for (int r = 0; r < rounds; ++r) {
      k_jump<<<gn, kB, 0, st>>>(D, fa, fb);
      std::swap(fa, fb);
    }
    k_dest_middle<<<gn, kB, 0, st>>>(D, fa);
    k_scatter<<<gn, kB, 0, st>>>(D);
    std::swap(D.box, D.box2);
    std::swap(D.perm, D.perm2);
    k_children<<<gn, kB, 0, st>>>(D);
    e = cudaGetLastError();
  }
  int err_flag = 0;
  unsigned long long leaves = 0;
  char *flat_mem = nullptr;
  if (e == cudaSuccess && (uint32_t)h_count[1] != 0) {
    out.inconsistent = true;
  } else if (e == cudaSuccess) {
    // Level k is [level_base[k], level_base[k + 1]): the last one is empty.
    const int n_levels = (int)level_base.size() - 1;
    const size_t sub_at = al256(level_base.size() * 8), place_at = sub_at + al256((size_t)n_nodes * 4);
    std::vector<std::pair<int, int>> runs;
    for (int l = 0; l < n_levels; ++l) {
      const bool narrow = level_base[(size_t)l + 1] - level_base[(size_t)l] <= kNarrow;
      const bool joins = !runs.empty() && narrow &&
                         level_base[(size_t)l] - level_base[(size_t)l - 1] <= kNarrow;
      if (joins) runs.back().second = l + 1;
      else runs.push_back({l, l + 1});
    }
    auto grid = [&](const std::pair<int, int> &r) {
      const int64_t m = level_base[(size_t)r.first + 1] - level_base[(size_t)r.first];
      return m <= kNarrow ? 1u : grid_of(m);
    };
    auto block = [&](const std::pair<int, int> &r) { return grid(r) == 1u ? (unsigned)kNarrow : (unsigned)kB; };
    if ((e = cudaMalloc(&flat_mem, place_at + (size_t)n_nodes * 8)) == cudaSuccess &&
        (e = cudaMalloc(&out.nodes, (size_t)n_nodes * sizeof(DevNode))) == cudaSuccess &&
        (e = cudaMalloc(&out.tris, nn * sizeof(DevTri))) == cudaSuccess &&
        (e = cudaMemcpyAsync(flat_mem, level_base.data(), level_base.size() * 8, cudaMemcpyHostToDevice, st)) ==
            cudaSuccess &&
        (e = cudaMemsetAsync(flat_mem + place_at, 0xFF, (size_t)n_nodes * 8, st)) == cudaSuccess) {
      const int64_t *level = (const int64_t *)flat_mem;
      uint32_t *sub = (uint32_t *)(flat_mem + sub_at);
      uint2 *place = (uint2 *)(flat_mem + place_at);
      for (size_t r = runs.size(); r-- > 0;)
        k_subtree<<<grid(runs[r]), block(runs[r]), 0, st>>>(D, level, runs[r].first, runs[r].second, sub);
      for (const auto &r : runs)
        k_flatten<<<grid(r), block(r), 0, st>>>(D, level, r.first, r.second, sub, place, n_nodes,
                                                 out.nodes);
      k_tris<<<gn, kB, 0, st>>>(D, src, out.tris);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess &&
        (e = cudaMemcpyAsync(out.bounds, D.rbox, 24, cudaMemcpyDeviceToHost, st)) == cudaSuccess &&
        (e = cudaMemcpyAsync(&err_flag, D.err, 4, cudaMemcpyDeviceToHost, st)) == cudaSuccess &&
        (e = cudaMemcpyAsync(&leaves, D.n_leaves, 8, cudaMemcpyDeviceToHost, st)) == cudaSuccess)
      e = cudaStreamSynchronize(st);
  }
  out.n_nodes = n_nodes;
  out.n_tris = n;
  out.max_depth = depth - 1;
  out.n_leaves = (int64_t)leaves;
  out.inconsistent = out.inconsistent || err_flag != 0;
  if (e != cudaSuccess || out.inconsistent) out.release();
  cudaFree(flat_mem);
  cudaFreeHost(h_count);
  release();
  return e;
}

void DeviceTree::release() {
  cudaFree(nodes);
  cudaFree(tris);
  nodes = nullptr;
  tris = nullptr;
}

cudaError_t launch_slot_ids(const DevTri *tris, int64_t n, int32_t *prim, int32_t *tri, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_slot_ids<<<grid_of(n), kB, 0, st>>>(tris, n, prim, tri);
  return cudaGetLastError();
}

cudaError_t launch_light_leaves(const DevNode *nodes, int64_t n_nodes, const LeafExt *ext, const DevTri *tris,
                                const int32_t *prim_first, const LightKey *keys, int64_t n_keys, float *leaf,
                                cudaStream_t st) {
  if (n_nodes <= 0 || n_keys <= 0) return cudaSuccess;
  k_light_leaves<<<grid_of(n_nodes), kB, 0, st>>>(nodes, n_nodes, ext, tris, prim_first, keys, n_keys, leaf);
  return cudaGetLastError();
}

}  // namespace skw
