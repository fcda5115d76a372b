// Photon kd-tree lookups on sm_103a: filtered k-nearest neighbours
// (KDTree::GetNearestPoints with PhotonFilter) and the nearest point
// (KDTree::GetNearestPoint), one query per thread.
//
// Restated from Raytracer/Core/KDTree.h:
//   * _Lookup (:537-576): visit a node's own point, then the child on the
//     query's side of the split, then the other child if the squared plane
//     distance is below the current search radius -- tested after the near
//     subtree is done.  The recursion becomes an explicit stack whose entries
//     carry the plane distance, re-tested on pop against the radius of that
//     moment, which is exactly when the reference tests it.
//   * distances in double from float positions and a double query
//     (:547-550), compared with strict "<" against the radius;
//   * NearestPointsProc (:331-387): the filter runs first; the first k
//     accepted points fill an unordered array that becomes a max-heap
//     (ordered by squared distance, ties by array position = the reference's
//     pointer order); afterwards each accepted point replaces the heap top.
//     The heap routines below are the classic binary-heap algorithms in the
//     same form as the C++ library's make/pop/push_heap (sift the hole to the
//     bottom, then sift the value up), so that not only the index sets but
//     the output order match the reference.
//   * PhotonFilter (PhotonInternalTypes.h:113-137): the photon's normal (from
//     the 16-bit direction table) within the cosine threshold of the surface
//     normal, and the photon near the surface's tangent plane.
// Double products and sums use round-to-nearest intrinsics so that no fused
// multiply-add changes a result.
//
// Layout: 16-byte nodes (x, y, z, word) read with one vector load, or 32-byte
// records of a node and its photon's normal (struct Tree).  The walk stack
// lives in shared memory, and so does the heap for k <= 128 (one word per
// entry); larger k use a heap in a caller-provided global scratch buffer of k
// entries per query.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <type_traits>

#include "kernels.h"

// Scratch of the allocation-free k-NN entry point (skw_knn_noalloc): heaps
// of SKW_KNN_NOALLOC_ENTRIES 16-byte entries (16 MiB), allocated with the
// module on every GPU that loads this library and held until the process
// exits.  Host code must not pass this symbol to a kernel (in host code it
// is only a stand-in for the device address); knn_noalloc_scratch() looks
// the device address up.
#define SKW_KNN_NOALLOC_ENTRIES (1 << 20)
static __device__ __align__(256) unsigned char g_knn_noalloc_scratch[(size_t)SKW_KNN_NOALLOC_ENTRIES * 16];

namespace skw {
namespace {

// One warp per block: a block's slot frees as soon as its warp's slowest
// query ends (queries differ widely in cost), and small blocks let the
// walk stack's shared memory be sized to fit, leaving the rest of the SM's
// storage to L1 (measured on the k = 100 photon lookups, 2,971,920 queries:
// 128 threads 34.3 ms, 32 threads 32.7 ms).
#ifndef SKW_KNN_BLOCK
#define SKW_KNN_BLOCK 32
#endif
constexpr int kKnnBlock = SKW_KNN_BLOCK;  // threads per block of the lookup kernels
// Minimum resident blocks per SM of k_knn and k_nearest: 32 one-warp blocks
// bound the registers at 64, too few for heaps of up to 32 entries (28 blocks,
// 72 registers: 669,824 filtered queries of k = 32 2.04 -> 1.97 ms; 24 blocks
// are slower for k = 1); larger ones leave room for 16 or fewer.
#ifndef SKW_KNN_MINB
#define SKW_KNN_MINB (1024 / SKW_KNN_BLOCK)
#endif
constexpr int knn_min_blocks(int kmax) { return kmax == 128 ? 16 : kmax == 32 ? 28 : SKW_KNN_MINB; }

constexpr float kKe1 = 6.2e-7f;

// The doubles stay where the caller put them: only what float cannot decide
// reads them (16 registers less, which the walks need).
struct Query {
  const double *q, *n;  // n: where the filter is on
  double cos_t;
  bool filter;
  float qf[3];  // q rounded up to float
  float dq[3];  // q - qf in float
  float e0;     // max |q - qf| over the axes
  float eq;     // what a float difference may be off besides its relative roundings (dist2f)
  float nf[3];  // the normal in float (filter pre-test)
  float cos_f, sin_f;  // cos_t, sin_t in float (filter pre-test)
  float ke0;           // a float squared distance k is within ke0 + kKe1 k of the exact one
};

__device__ __forceinline__ double sin_of(double cos_t) { return __dsqrt_rn(__dsub_rn(1.0, __dmul_rn(cos_t, cos_t))); }

// Fills the float copy of the query point used by the pre-tests.
__device__ __forceinline__ void query_float(Query &Q) {
  float e = 0.0f;
  for (int k = 0; k < 3; ++k) {
    const double qk = __ldg(Q.q + k);
    Q.qf[k] = __double2float_ru(qk);
    Q.dq[k] = (float)(qk - (double)Q.qf[k]);
    e = fmaxf(e, fabsf(Q.dq[k]));
    Q.nf[k] = Q.filter ? (float)__ldg(Q.n + k) : 0.0f;
  }
  Q.e0 = e * 1.0001f;
  Q.eq = e * 1.2e-7f;  // 2u e, rounded up
  Q.ke0 = 1.76e7f * Q.eq * Q.eq + 1e-37f;
  Q.cos_f = (float)Q.cos_t;
  Q.sin_f = (float)sin_of(Q.cos_t);
}

// Coordinates of the query by a run-time axis, selected without indexing so
// that the query stays in registers.
__device__ __forceinline__ float qf_at(const Query &Q, uint32_t a) {
  return a == 0 ? Q.qf[0] : (a == 1 ? Q.qf[1] : Q.qf[2]);
}
__device__ __forceinline__ float dq_at(const Query &Q, uint32_t a) {
  return a == 0 ? Q.dq[0] : (a == 1 ? Q.dq[1] : Q.dq[2]);
}
__device__ __forceinline__ double q_at(const Query &Q, uint32_t a) {
  return __ldg(Q.q + a);
}

// A tree as the lookups read it: its 16-byte nodes, and its records of a node
// and its photon's normal (4 floats; kernels.h, nids_bytes).  A record is one
// load, of the sector that the node alone would take, so walks with the filter
// and registers to spare read those; the others read the nodes, of which twice
// as many fit into L1, and a normal once the distance is known.
struct NodeN {
  float4 p, m;
};
struct Tree {
  const float4 *nodes, *records;
  int n;
  __device__ __forceinline__ float4 at(int i) const { return __ldg(nodes + i); }
  __device__ __forceinline__ float4 normal(int i) const { return __ldg(records + 2 * (int64_t)i + 1); }
  __device__ __forceinline__ NodeN load(int i, bool with_normal) const {
    NodeN r;
    if (with_normal) {
      asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
          : "=f"(r.p.x), "=f"(r.p.y), "=f"(r.p.z), "=f"(r.p.w), "=f"(r.m.x), "=f"(r.m.y), "=f"(r.m.z), "=f"(r.m.w)
          : "l"(records + 2 * (int64_t)i));
    } else {
      r.p = __ldg(nodes + i);
      r.m = make_float4(0, 0, 0, 0);
    }
    return r;
  }
};

// PhotonFilter::operator() (PhotonInternalTypes.h:127-133), with float
// pre-tests: the normal's cosine and the in-plane test are decided in float
// when they clear their thresholds by more than the float error (unit
// vectors: a few 1e-7), else in double as the reference computes them.
__device__ __forceinline__ bool photon_filter_exact(const Query &Q, const float4 p, uint16_t nid,
                                                    const double *__restrict__ dirs);
__device__ __forceinline__ bool photon_filter(const Query &Q, const NodeN &node, int i,
                                              const uint16_t *__restrict__ nids, const double *__restrict__ dirs) {
  const float4 p = node.p, m = node.m;
  const float cf = m.x * Q.nf[0] + m.y * Q.nf[1] + m.z * Q.nf[2];
  const float ct = Q.cos_f;
  if (cf < ct - 2e-6f) return false;
  if (cf > ct + 2e-6f) {
    // |to . n| < sin_t |to|, compared as squares when both sides clearly differ
    const float tx = p.x - Q.qf[0], ty = p.y - Q.qf[1], tz = p.z - Q.qf[2];
    const float dn = tx * Q.nf[0] + ty * Q.nf[1] + tz * Q.nf[2];
    const float l2 = tx * tx + ty * ty + tz * tz;
    const float st = Q.sin_f;
    const float lhs = dn * dn, rhs = st * st * l2;
    // error: the float query's rounding e0 on each component plus relative rounding
    const float a = fabsf(tx) + fabsf(ty) + fabsf(tz);
    // |d(dn)| <= 3 e0 + 5e-7 a and |d(l2)| <= 2 a (e0 + 6e-8 a) (a = |tx| + |ty| + |tz|), so
    // the squares move by at most 2 a |d(dn)| + |d(dn)|^2 and st^2 |d(l2)|
    const float err = 12.0f * Q.e0 * (a + Q.e0) + 4e-6f * a * a + 2e-6f * (lhs + rhs) + 1e-37f;
    if (lhs + err < rhs) return true;
    if (lhs - err > rhs) return false;
  }
  return photon_filter_exact(Q, p, __ldg(nids + i), dirs);
}

__device__ __forceinline__ bool photon_filter_exact(const Query &Q, const float4 p, uint16_t nid,
                                                    const double *__restrict__ dirs) {
  const double nx = __ldg(dirs + 3 * nid), ny = __ldg(dirs + 3 * nid + 1), nz = __ldg(dirs + 3 * nid + 2);
  const double qx = __ldg(Q.q), qy = __ldg(Q.q + 1), qz = __ldg(Q.q + 2);
  const double mx = __ldg(Q.n), my = __ldg(Q.n + 1), mz = __ldg(Q.n + 2);
  const double cosn = __dadd_rn(__dadd_rn(__dmul_rn(nx, mx), __dmul_rn(ny, my)), __dmul_rn(nz, mz));
  if (!(cosn > Q.cos_t)) return false;
  const double tx = __dsub_rn((double)p.x, qx), ty = __dsub_rn((double)p.y, qy), tz = __dsub_rn((double)p.z, qz);
  const double dotn = __dadd_rn(__dadd_rn(__dmul_rn(tx, mx), __dmul_rn(ty, my)), __dmul_rn(tz, mz));
  const double len = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(tx, tx), __dmul_rn(ty, ty)), __dmul_rn(tz, tz)));
  return fabs(dotn) < __dmul_rn(sin_of(Q.cos_t), len);
}

__device__ __forceinline__ double point_d2(const float4 p, const double *__restrict__ q) {
  const double dx = __dsub_rn((double)p.x, __ldg(q)), dy = __dsub_rn((double)p.y, __ldg(q + 1)),
               dz = __dsub_rn((double)p.z, __ldg(q + 2));
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

__device__ __forceinline__ double point_d2(const float4 p, const Query &Q) { return point_d2(p, Q.q); }

// Float pre-tests.  A point's squared distance and a splitting plane's
// squared distance are first computed in float and compared with two
// thresholds derived from the current radius and a bound on the float
// value's distance from the reference's double value; only a value between
// the thresholds is decided in double.
// A difference from the query is (p - qf) - dq: with u = 2^-24 and e the
// largest |dq|, the two subtractions and dq's own rounding put it within
// 2u|d| + 2u e =: 2u|d| + eq of the exact difference d.  (Without dq the
// difference is off by e itself: near keys of a heap, a millionth of the
// coordinates apart, could then not be told apart in float, and the double
// comparisons of some lane held up nearly every heap operation of a warp.)
// The squared distance F from those differences, its fused sum's three
// roundings and the double result's own rounding give
//   |F - d2| <= 7u D + 2 eq sum|d| + 3 eq^2 (+ 2^-52 D),  D = sum d^2 <= F (1 + 5u),
// and sum|d| <= sqrt(3 D):  E(F) = 4.3e-7 F + 3.47 eq sqrt(F) + 3.01 eq^2,
// plus 1e-37 for roundings in the subnormal range.  A plane's squared
// distance (one axis, two roundings fewer) is within the same bound.
__device__ __forceinline__ float dist2f(const float4 p, const Query &Q) {
  const float dx = (p.x - Q.qf[0]) - Q.dq[0], dy = (p.y - Q.qf[1]) - Q.dq[1], dz = (p.z - Q.qf[2]) - Q.dq[2];
  return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}
__device__ __forceinline__ float d2_err(const Query &Q, float x) {
  // 1.0001: the roundings of this float evaluation (about 6u)
  return (4.3e-7f * x + 3.47f * Q.eq * __fsqrt_ru(x) + 3.01f * Q.eq * Q.eq + 1e-37f) * 1.0001f;
}
// Thresholds on a float squared distance F against a radius known to lie
// in [rlo, rhi]: F < tin => inside, F >= tout => outside (else decide in
// double).  tin = rlo - E(rlo): for F < tin, F + E(F) < rlo because E grows
// with F.  tout = rhi + E(2 rhi): for F in [tout, 2 rhi], F - E(F) >= rhi;
// above 2 rhi, E(F) <= F / 2 <= F - rhi once sqrt(rhi) >= 8 eq; below that
// (or for an infinite radius) nothing is decided outside in float.
__device__ __forceinline__ void radius_thresholds(const Query &Q, float rlo, float rhi, float &tin, float &tout) {
  tin = isinf(rlo) ? rlo : (rlo > 0.0f ? __fsub_rd(rlo, d2_err(Q, rlo)) : -1.0f);
  const float two = 2.0f * rhi;
  tout = (!isinf(two) && rhi >= fmaxf(64.0f * Q.eq * Q.eq, 1e-36f)) ? __fadd_ru(rhi, d2_err(Q, two)) : INFINITY;
}

// A node's children in the reference's visit order: near = the child on the
// query's side of the split (visited next), far = the other (postponed and
// visited only if its plane is within the radius when it is popped); -1
// where a child is absent or the node is a leaf.  q <= split is decided on
// the float query: it is q rounded up, and split is a float.  s2: the plane's
// squared distance in float (dist2f's bound holds for it).
__device__ __forceinline__ void node_children(const float4 p, int cur, int n, const Query &Q, int &near, int &far,
                                              float &s2) {
  const uint32_t w = __float_as_uint(p.w), axis = w & 3u;
  near = far = -1;
  s2 = 0.0f;
  if (axis == 3u) return;
  const float split = axis == 0 ? p.x : (axis == 1 ? p.y : p.z), q = qf_at(Q, axis), sd = (q - split) + dq_at(Q, axis);
  s2 = sd * sd;
  const uint32_t right = w >> 3;
  const int l = (w & 4u) != 0u ? cur + 1 : -1, r = right < (uint32_t)n ? (int)right : -1;
  const bool le = q <= split;
  near = le ? l : r;
  far = le ? r : l;
}

// The plane's test in double, as the reference's: (q - split)^2.
__device__ __forceinline__ double plane_d2(const float4 p, const Query &Q) {
  const uint32_t axis = __float_as_uint(p.w) & 3u;
  const double pd = __dsub_rn(q_at(Q, axis), (double)(axis == 0 ? p.x : (axis == 1 ? p.y : p.z)));
  return __dmul_rn(pd, pd);
}

// The node whose child `child` is: the tree lies in pre-order, so the descent
// from the root goes right where `child` is not before the right child.
__device__ __noinline__ int node_parent(Tree T, int child) {
  int cur = 0;
  for (int next = 0; cur < child; cur = next) {
    const uint32_t right = __float_as_uint(T.at(cur).w) >> 3;
    next = right < (uint32_t)T.n && child >= (int)right ? (int)right : cur + 1;
    if (next == child) break;
  }
  return cur;
}

// The search radius of a walk: max_dist^2 (KDTree::Lookup, KDTree.h:475-482)
// until set() makes it the exact squared distance of a photon, of which only
// a float bracket is kept; the exact double is computed when a decision needs
// it.  tin / tout: radius_thresholds of the bracket.
struct Radius {
  double exact;
  int idx;  // the photon (get's `ids`: its place there) at this distance; -1: `exact` holds it
  float tin, tout;

  __device__ __forceinline__ void start(const Query &Q, double max_dist) {
    exact = __dmul_rn(max_dist, max_dist);
    idx = -1;
    radius_thresholds(Q, __double2float_rd(exact), __double2float_ru(exact), tin, tout);
  }
  // cut: how far `key` may be from the photon's, relative to itself
  __device__ __forceinline__ void set(const Query &Q, int photon, float key, float cut) {
    const float e = 1.0001f * fmaf(kKe1 + cut, key, Q.ke0);
    idx = photon;
    radius_thresholds(Q, __fsub_rd(key, e), __fadd_ru(key, e), tin, tout);
  }
  __device__ __forceinline__ double get(const Tree &T, const Query &Q, const int32_t *ids = nullptr) {
    if (idx >= 0) {
      exact = point_d2(T.at(ids ? ids[idx] : idx), Q);
      idx = -1;
    }
    return exact;
  }
};

// The walk stack lives in shared memory ([entry][thread], so lanes never
// share a bank).  k_knn's entry is the parent of a postponed far child: on pop
// the parent is read again (a recently visited node, usually still in L1) and
// its split gives both the far child and the plane distance to re-test.  Shared
// memory and L1 share the SM's storage, and the walk's reads want the L1, so
// the stack is sized by the tree's depth: the median-split tree of n points is
// floor(log2 n) + 1 levels deep and the walk holds at most one entry per level,
// so S = 20 serves n < 2^20 and S = 32 any n < 2^31.  k_knn_gang and the nearest
// points' walks, whose L1 holds little or whose pops are most of the work, keep
// the far child and its plane's float distance instead, and look the parent up
// (node_parent) when that does not decide.

// ------------------------------------------------------------ k_knn --
// The heap holds float squared distances: an entry's key is the float
// distance of its point (dist2f), within ke0 + kKe1 key of the reference's
// double value: that bounds the error derived above, 7u D + 2 sqrt(3) eq
// sqrt(D) + 3 eq^2, the square-root term by
// 2 sqrt(3) eq sqrt(D) <= sqrt(3) (1e7 eq^2 + 1e-7 D).
// Heap comparisons are decided on the keys and their bounds, and only when
// two keys' intervals overlap are the exact doubles of both points computed
// (GB300 runs a double operation at ~1/64 of the float rate, and divergent
// double work in the former exact-keyed heap kept its FP64 pipe half busy);
// ties of exact distances go to the lower tree position, as the reference's
// NearestPoint comparison (KDTree.h:331-387) decides them.  So the heap
// takes the same branches as the reference's and its order is the
// reference's.  The search radius is max_dist^2 until the heap is full and
// then the top's exact distance, represented by a float bracket [rlo, rhi]
// and computed exactly on demand.  The exact distances of the output are
// computed at the end, four independent chains at a time.

// A heap entry: float squared distance and tree position.
struct FCand {
  float key;
  int32_t idx;
};

// Entries per query of a global heap: k + 1 rounded up to even.
__host__ __device__ __forceinline__ int64_t knn_heap_stride(int k) { return ((int64_t)k + 2) & ~(int64_t)1; }

// (d2, idx) lexicographic on the exact distances, decided on the keys when
// their bounds do not overlap.
__device__ __forceinline__ bool fcand_less(const Tree &T, const Query &Q, const FCand &a,
                                           const FCand &b) {
  // decided when |a - b| exceeds both bounds (with a margin for this float arithmetic)
  const float d = a.key - b.key, tol = 1.0001f * fmaf(kKe1, a.key + b.key, 2.0f * Q.ke0);
  if (d < -tol) return true;
  if (d > tol) return false;
  const double da = point_d2(T.at(a.idx), Q), db = point_d2(T.at(b.idx), Q);
  return da == db ? a.idx < b.idx : da < db;
}

__device__ __forceinline__ void fheap_push_up(const Tree &T, const Query &Q, FCand *h, int hole, int top, FCand value) {
  int parent = (hole - 1) / 2;
  while (hole > top && fcand_less(T, Q, h[parent], value)) {
    h[hole] = h[parent];
    hole = parent;
    parent = (hole - 1) / 2;
  }
  h[hole] = value;
}

// PAIR: h[1] is 16-byte aligned, so that the children 2j+1, 2j+2 of every
// entry j share one 16-byte load.
template <bool PAIR = false>
__device__ __forceinline__ void fheap_adjust(const Tree &T, const Query &Q, FCand *h, int hole, int len, FCand value) {
  const int top = hole;
  int second = hole;
  while (second < (len - 1) / 2) {
    second = 2 * (second + 1);
    if (PAIR) {
      const uint4 two = *reinterpret_cast<const uint4 *>(h + second - 1);
      const FCand a{__uint_as_float(two.x), (int32_t)two.y}, b{__uint_as_float(two.z), (int32_t)two.w};
      const bool left = fcand_less(T, Q, b, a);
      second -= left ? 1 : 0;
      h[hole] = left ? a : b;
    } else {
      if (fcand_less(T, Q, h[second], h[second - 1])) second--;
      h[hole] = h[second];
    }
    hole = second;
  }
  if ((len & 1) == 0 && second == (len - 2) / 2) {
    second = 2 * (second + 1);
    h[hole] = h[second - 1];
    hole = second - 1;
  }
  fheap_push_up(T, Q, h, hole, top, value);
}

__device__ __forceinline__ void fheap_make(const Tree &T, const Query &Q, FCand *h, int len) {
  if (len < 2) return;
  for (int parent = (len - 2) / 2;; --parent) {
    fheap_adjust(T, Q, h, parent, len, h[parent]);
    if (parent == 0) return;
  }
}

__device__ __forceinline__ void load_query(Query &Q, const double *__restrict__ q, const double *__restrict__ qn,
                                           int64_t i, double cos_t) {
  Q.q = q + 3 * i;
  Q.filter = cos_t >= 0.0;
  Q.n = Q.filter ? qn + 3 * i : nullptr;
  Q.cos_t = cos_t;
  query_float(Q);
}

// The two heaps of k_knn.  Until a heap is full its entries are the accepted
// points in visit order (the reference's array holds them unordered); at k
// entries it becomes a heap.  add(): the i-th point of those; make(): the heap
// of the first k; replace(): pop_heap (the top goes to the back, the back's
// old value is re-placed), then the point pushed up from the back; top(): the
// top as the search radius.

// Heaps in a global scratch buffer (k > 128, and skw_knn_noalloc): query i's
// entries from scratch[i * stride + 1], stride even (16-byte aligned sibling
// pairs, fheap_adjust<true>).
struct GlobalHeap {
  FCand *h;
  __device__ __forceinline__ void add(int i, float key, int32_t photon) { h[i] = FCand{key, photon}; }
  __device__ __forceinline__ void make(const Tree &T, const Query &Q, int k) {
    fheap_make(T, Q, h, k);
  }
  __device__ __forceinline__ void replace(const Tree &T, const Query &Q, int k, float key,
                                          int32_t photon) {
    const FCand back = h[k - 1];
    h[k - 1] = h[0];
    fheap_adjust<true>(T, Q, h, 0, k - 1, back);
    fheap_push_up(T, Q, h, k - 1, 0, FCand{key, photon});
  }
  __device__ __forceinline__ int32_t photon(int i) const { return h[i].idx; }
  __device__ __forceinline__ void top(const Query &Q, Radius &r) const { r.set(Q, h[0].idx, h[0].key, 0.0f); }
};

// Heaps in shared memory (k <= 128), one word per entry: the key with its low
// 7 bits replaced by the entry's slot, the place in `ids` that holds its tree
// position.  A heap operation moves words only, one load and a store per level
// ([row][thread], so that lanes never share a bank), and a photon's position is
// written once, into local memory.  As a float the word is within 2^-16 of the
// photon's key, which joins the error bounds; two words that close are compared
// by their photons' distances in double, out of line.  What bounds the lookup is
// the latency of its chains of moves and node reads at 12 to 14 warps per SM
// (ncu: issue 36 %).  The k = 100 lookups of 669,824 queries took 9.91 ms with
// 8-byte entries in local memory (1 KB per query, which L1 cannot hold), 9.17 ms
// with words here, 7.64 ms with far children dropped at the push when their
// plane is outside by then, 7.29 ms with the normals read in one load, 6.48 ms
// with records, words compared as integers and lanes that wait for one another
// (k_knn_gang), 6.12 ms with the heaps made together.
struct SharedHeap {
  static constexpr uint32_t kSlot = 127u;
  static constexpr float kCut = 1.5262e-5f;  // 128 units in the last place: 2^-16, rounded up
  char *h;  // this thread's 8 bytes of row 0
  int32_t *ids;
  // Entries 2r - 1 and 2r share the 8 bytes of row r, so that the children of
  // entry i are one load, of row i + 1 (the root is the second word of row 0).
  static constexpr int kRow = kKnnBlock * 8;
  __host__ __device__ static __forceinline__ size_t bytes(int k) { return (size_t)(k / 2 + 1) * kRow; }
  __device__ __forceinline__ uint32_t *slot(int i) const {
    return reinterpret_cast<uint32_t *>(h + ((i + 1) >> 1) * kRow + ((i + 1) & 1) * 4);
  }
  __device__ __forceinline__ uint2 children(int i) const { return *reinterpret_cast<const uint2 *>(h + (i + 1) * kRow); }
  __device__ __forceinline__ uint32_t at(int i) const { return *slot(i); }
  static __device__ __forceinline__ uint32_t entry(float key, uint32_t slot) {
    return (__float_as_uint(key) & ~kSlot) | slot;
  }
  // (d2, position) lexicographic, as fcand_less.  Words that differ by more
  // than kApart are in the order of their photons' exact distances if the
  // smaller is not below `tiny`: floats a > b that are n words apart have
  // a - b >= n 2^-24 b, and what must be exceeded is 2 (kKe1 + kCut) of their
  // mean and 2 ke0, 4.18e-5 b for b >= tiny = 2e5 ke0 -- 702 words.  Infinite
  // keys and NaN (all of a query's, then) lie within kApart of each other.
  static constexpr uint32_t kApart = 720u;
  uint32_t tiny;
  static __device__ __noinline__ bool less_exact(Tree T, const double *q, int32_t ia, int32_t ib) {
    const double da = point_d2(T.at(ia), q), db = point_d2(T.at(ib), q);
    return da == db ? ia < ib : da < db;
  }
  __device__ __forceinline__ bool less(const Tree &T, const Query &Q, uint32_t a, uint32_t b) const {
    if (a - b + kApart > 2u * kApart && min(a, b) >= tiny) return a < b;
    return less_exact(T, Q.q, ids[a & kSlot], ids[b & kSlot]);
  }
  // to: the slot of `hole`
  __device__ __forceinline__ void push_up(const Tree &T, const Query &Q, int hole, uint32_t *to,
                                          int top, uint32_t value) {
    while (hole > top) {
      const int parent = (hole - 1) >> 1;
      uint32_t *from = slot(parent);
      const uint32_t p = *from;
      if (!less(T, Q, p, value)) break;
      *to = p;
      hole = parent;
      to = from;
    }
    *to = value;
  }
  __device__ __forceinline__ void adjust(const Tree &T, const Query &Q, int hole, int len,
                                         uint32_t value) {
    const int top = hole, two = (len - 1) / 2;
    uint32_t *to = slot(hole);
    while (hole < two) {
      const uint2 c = children(hole);
      const bool left = less(T, Q, c.y, c.x);
      *to = left ? c.x : c.y;
      to = reinterpret_cast<uint32_t *>(h + (hole + 1) * kRow + (left ? 0 : 4));
      hole = 2 * hole + (left ? 1 : 2);
    }
    if ((len & 1) == 0 && hole == (len - 2) / 2) {
      *to = children(hole).x;
      to = reinterpret_cast<uint32_t *>(h + (hole + 1) * kRow);
      hole = 2 * hole + 1;
    }
    push_up(T, Q, hole, to, top, value);
  }
  __device__ __forceinline__ void add(int i, float key, int32_t photon) {
    ids[i] = photon;
    *slot(i) = entry(key, (uint32_t)i);
  }
  __device__ __forceinline__ void make(const Tree &T, const Query &Q, int k) {
    for (int parent = (k - 2) / 2; parent >= 0 && k >= 2; --parent) adjust(T, Q, parent, k, at(parent));
  }
  __device__ __forceinline__ void replace(const Tree &T, const Query &Q, int k, float key,
                                          int32_t photon) {
    const uint32_t back = at(k - 1), top = at(0);
    adjust(T, Q, 0, k - 1, back);
    ids[top & kSlot] = photon;
    push_up(T, Q, k - 1, slot(k - 1), 0, entry(key, top & kSlot));
  }
  __device__ __forceinline__ int32_t photon(int i) const { return ids[at(i) & kSlot]; }
  __device__ __forceinline__ void top(const Query &Q, Radius &r) const {
    const uint32_t t = at(0);
    r.set(Q, (int)(t & kSlot), __uint_as_float(t), kCut);
  }
};

// A query's output: its heap's photons and their exact squared distances, four
// independent chains at a time.
template <class Heap>
__device__ __forceinline__ void write_found(const Tree &T, const Query &Q, const Heap &heap, int64_t i, int size, int k,
                                            int32_t *__restrict__ out_idx, double *__restrict__ out_d2) {
  int j = 0;
  for (; j + 4 <= size; j += 4) {
    const int32_t a0 = heap.photon(j), a1 = heap.photon(j + 1), a2 = heap.photon(j + 2), a3 = heap.photon(j + 3);
    const double d0 = point_d2(T.at(a0), Q), d1 = point_d2(T.at(a1), Q),
                 d2 = point_d2(T.at(a2), Q), d3 = point_d2(T.at(a3), Q);
    out_idx[i * k + j] = a0;
    out_idx[i * k + j + 1] = a1;
    out_idx[i * k + j + 2] = a2;
    out_idx[i * k + j + 3] = a3;
    out_d2[i * k + j] = d0;
    out_d2[i * k + j + 1] = d1;
    out_d2[i * k + j + 2] = d2;
    out_d2[i * k + j + 3] = d3;
  }
  for (; j < size; ++j) {
    const int32_t a = heap.photon(j);
    out_idx[i * k + j] = a;
    out_d2[i * k + j] = point_d2(T.at(a), Q);
  }
  for (; j < k; ++j) {
    out_idx[i * k + j] = -1;
    out_d2[i * k + j] = 0.0;
  }
}

// KMAX > 0: heaps of k <= KMAX entries in shared memory; KMAX == 0: global
// heaps.
template <int KMAX, int S>
__global__ void __launch_bounds__(kKnnBlock, knn_min_blocks(KMAX)) k_knn(
    Tree T, const uint16_t *__restrict__ nids, const double *__restrict__ dirs, const double *__restrict__ q,
    const double *__restrict__ qn, int64_t nq, int k, double max_dist, double cos_t, int32_t *__restrict__ out_idx,
    double *__restrict__ out_d2, int32_t *__restrict__ out_count, int32_t *__restrict__ out_visited,
    FCand *__restrict__ scratch, unsigned *__restrict__ status, const int *__restrict__ nq_dev,
    const int32_t *__restrict__ order, int per_warp) {
  __shared__ uint32_t stk[S][kKnnBlock];
  const int lane = threadIdx.x & 31;
  if (lane >= per_warp) return;
  int64_t i = ((int64_t)blockIdx.x * (kKnnBlock / 32) + (threadIdx.x >> 5)) * per_warp + lane;
  if (nq_dev && *nq_dev < nq) nq = *nq_dev;
  if (i >= nq) return;
  if (order) i = order[i];
  Query Q;
  load_query(Q, q, qn, i, cos_t);
  int32_t ids[KMAX > 0 ? KMAX : 1];
  extern __shared__ __align__(16) char s_mem[];
  typename std::conditional<(KMAX > 0), SharedHeap, GlobalHeap>::type heap = [&]() {
    if constexpr (KMAX > 0) return SharedHeap{s_mem + threadIdx.x * 8, ids, __float_as_uint(2.0e5f * Q.ke0)};
    else return GlobalHeap{scratch + i * (int64_t)knn_heap_stride(k) + 1};
  }();
  int size = 0, visited = 0;
  if (k > 0 && T.n > 0) {
    Radius rad;  // max_dist until the heap is full, then its top
    rad.start(Q, max_dist);
    int sp = 0, cur = 0;
    bool overflow = false;
    float4 p = T.at(0);
    for (;;) {
      ++visited;
      int near, far;
      float s2;
      node_children(p, cur, T.n, Q, near, far, s2);
      {
        const float d2f = dist2f(p, Q);
        if ((d2f < rad.tin || (!(d2f >= rad.tout) && point_d2(p, Q) < rad.get(T, Q, KMAX > 0 ? ids : nullptr))) &&
            (!Q.filter || photon_filter(Q, NodeN{p, T.normal(cur)}, cur, nids, dirs))) {
          if (size < k) {
            heap.add(size++, d2f, cur);
            if (size == k) {
              heap.make(T, Q, k);
              heap.top(Q, rad);
            }
          } else {
            heap.replace(T, Q, k, d2f, cur);
            heap.top(Q, rad);
          }
        }
      }
      // The far child waits on the stack, unless its plane is certainly outside
      // already (the radius only shrinks, so it would be when popped).
      if (far >= 0 && !(s2 >= rad.tout)) {
        if (sp >= S) {
          overflow = true;
          break;
        }
        stk[sp][threadIdx.x] = (uint32_t)cur;
        ++sp;
      }
      if (near >= 0) {
        cur = near;
        p = T.at(near);
        continue;
      }
      int next = -1;
      while (sp > 0) {
        --sp;
        // the reference's pop test: (qa - split)^2 < radius, in double
        const uint32_t par = stk[sp][threadIdx.x];
        int pnear, pfar;
        float ps2;
        const float4 pp = T.at((int)par);
        node_children(pp, (int)par, T.n, Q, pnear, pfar, ps2);
        if (ps2 < rad.tin || (!(ps2 >= rad.tout) && plane_d2(pp, Q) < rad.get(T, Q, KMAX > 0 ? ids : nullptr))) {
          next = pfar;
          break;
        }
      }
      if (next < 0) break;
      cur = next;
      p = T.at(cur);
    }
    if (overflow) atomicOr(status, 2u);
  }
  out_count[i] = size;
  write_found(T, Q, heap, i, size, k, out_idx, out_d2);
  if (out_visited) out_visited[i] = visited;
}

// A heap operation is a chain of some 15 levels (the make_heap of a full heap,
// of 100), which a warp walks for whichever of its lanes are at one.  So in
// full warps a lane that has a point for its heap waits with it until a third
// of the lanes with full heaps do (kReplaceShare / 3), and one whose heap is
// full for the first time until seven eighths of those still filling are
// (kMakeShare / 8); what the lookups visit and find is the same, as a lane
// takes no step with a radius that is not up to date.  k = 100, 669,824
// queries: at once 6.98 ms, a third 6.53, half 6.48, two thirds 7.23; with the
// heaps made at three quarters 6.28, seven eighths 6.19, all 6.08 (but queries
// that never fill theirs would then hold up the others).  A waiting walk's
// stack keeps a far child with its plane's distance, which spares the parent's
// load at a pop.  Heaps of 32 entries are too short for it (gather lookups 2.82
// -> 3.50 ms), at 33 to 40 it depends on the number of queries (669,824: 2.19
// -> 2.37 ms, 100,000: 0.54 -> 0.50), from 50 on both gain (3.21 -> 2.92 ms,
// 0.84 -> 0.59); and in warps with few queries (irradiance estimates 3.51 ->
// 4.25 ms) no lane waits either.
constexpr int kReplaceShare = 1, kMakeShare = 7, kGangEntries = 48;
constexpr int kGangBlocks = 24;  // resident per SM with heaps in global memory

template <int KMAX>
__global__ void __launch_bounds__(kKnnBlock, KMAX == 128 ? 16 : kGangBlocks) k_knn_gang(
    Tree T, const uint16_t *__restrict__ nids, const double *__restrict__ dirs, const double *__restrict__ q,
    const double *__restrict__ qn, int64_t nq, int k, double max_dist, double cos_t, int32_t *__restrict__ out_idx,
    double *__restrict__ out_d2, int32_t *__restrict__ out_count, int32_t *__restrict__ out_visited,
    FCand *__restrict__ scratch, unsigned *__restrict__ status, const int *__restrict__ nq_dev,
    const int32_t *__restrict__ order, int depth) {
  static_assert(kKnnBlock == 32, "one warp per block");
  // the heaps' rows, then the walk stacks: `depth` entries each
  extern __shared__ __align__(16) char s_mem[];
  uint2 *stk = reinterpret_cast<uint2 *>(s_mem + (KMAX > 0 ? SharedHeap::bytes(k) : 0)) + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int64_t i = ((int64_t)blockIdx.x * (kKnnBlock / 32) + (threadIdx.x >> 5)) * 32 + lane;
  if (nq_dev && *nq_dev < nq) nq = *nq_dev;
  const bool mine = i < nq;
  if (mine && order) i = order[i];
  Query Q{};
  if (mine) load_query(Q, q, qn, i, cos_t);
  int32_t ids[KMAX > 0 ? KMAX : 1];
  typename std::conditional<(KMAX > 0), SharedHeap, GlobalHeap>::type heap = [&]() {
    if constexpr (KMAX > 0) return SharedHeap{s_mem + threadIdx.x * 8, ids, __float_as_uint(2.0e5f * Q.ke0)};
    else return GlobalHeap{scratch + i * (int64_t)knn_heap_stride(k) + 1};
  }();
  int size = 0, visited = 0;
  Radius rad;  // max_dist until the heap is full, then its top
  if (mine) rad.start(Q, max_dist);
  // A point for the heap waits in (key, photon), and its lane with it, until
  // enough lanes have one.
  bool walks = mine && k > 0 && T.n > 0, waits = false, made = false;
  float key = 0.0f;
  int photon = 0, sp = 0, cur = 0;  // cur < 0: the next node comes from the stack
  NodeN p{};
  if (walks) p = T.load(0, Q.filter);
  for (;;) {
    if (walks && !waits) {
      while (cur < 0 && sp > 0) {
        --sp;
        // the reference's pop test: (qa - split)^2 < radius, in double
        const uint2 top = stk[sp * kKnnBlock];
        const float s2 = __uint_as_float(top.y);
        if (s2 < rad.tin || (!(s2 >= rad.tout) && plane_d2(T.at(node_parent(T, (int)top.x)), Q) <
                                                      rad.get(T, Q, KMAX > 0 ? ids : nullptr))) {
          cur = (int)top.x;
          p = T.load(cur, Q.filter);
        }
      }
      walks = cur >= 0;
      if (walks) {
        ++visited;
        int near, far;
        float s2;
        node_children(p.p, cur, T.n, Q, near, far, s2);
        const float d2f = dist2f(p.p, Q);
        if ((d2f < rad.tin || (!(d2f >= rad.tout) && point_d2(p.p, Q) < rad.get(T, Q, KMAX > 0 ? ids : nullptr))) &&
            (!Q.filter || photon_filter(Q, p, cur, nids, dirs))) {
          key = d2f;
          photon = cur;
          waits = size >= k - 1;
          if (size < k) heap.add(size++, d2f, cur);
        }
        // The far child waits on the stack, unless its plane is certainly outside
        // already (the radius only shrinks, so it would be when popped).
        if (far >= 0 && !(s2 >= rad.tout)) {
          if (sp >= depth) {
            atomicOr(status, 2u);
            walks = waits = false;
          } else {
            stk[sp * kKnnBlock] = make_uint2((uint32_t)far, __float_as_uint(s2));
            ++sp;
          }
        }
        cur = near;
        if (near >= 0) p = T.load(near, Q.filter);
      }
    }
    if (!__any_sync(0xffffffffu, walks)) break;
    const int filling = __popc(__ballot_sync(0xffffffffu, walks && !made)),
              full = __popc(__ballot_sync(0xffffffffu, walks && made)),
              to_make = __popc(__ballot_sync(0xffffffffu, waits && !made)),
              to_replace = __popc(__ballot_sync(0xffffffffu, waits && made));
    if (waits && (made ? 3 * to_replace >= kReplaceShare * full : 8 * to_make >= kMakeShare * filling)) {
      if (made) heap.replace(T, Q, k, key, photon);
      else heap.make(T, Q, k);
      heap.top(Q, rad);
      made = true;
      waits = false;
    }
  }
  if (!mine) return;
  out_count[i] = size;
  write_found(T, Q, heap, i, size, k, out_idx, out_d2);
  if (out_visited) out_visited[i] = visited;
}

// GetNearestPoint (KDTree.h:495-503) with NearestPointProc (:293-323):
// every accepted point becomes the nearest and shrinks the radius.  BOUNDED:
// a walk that has not ended after `budget` nodes is given up (kUnfinished).
constexpr int kUnfinished = -2;
template <int S, bool BOUNDED>
__device__ __forceinline__ int nearest_walk(Tree T, const uint16_t *__restrict__ nids,
                                            const double *__restrict__ dirs, const Query &Q, double max_dist, uint2 (*stk)[kKnnBlock],
                                            unsigned *__restrict__ status, int budget) {
  int best = -1;
  if (T.n <= 0) return best;
  Radius rad;
  rad.start(Q, max_dist);
  int sp = 0, cur = 0;
  NodeN p = T.load(0, Q.filter);
  for (;;) {
    if (BOUNDED && budget-- == 0) return kUnfinished;
    int near, far;
    float s2;
    node_children(p.p, cur, T.n, Q, near, far, s2);
    const float d2f = dist2f(p.p, Q);
    if ((d2f < rad.tin || (!(d2f >= rad.tout) && point_d2(p.p, Q) < rad.get(T, Q))) &&
        (!Q.filter || photon_filter(Q, p, cur, nids, dirs))) {
      best = cur;
      rad.set(Q, cur, d2f, 0.0f);
    }
    // The far child waits on the stack, unless its plane is certainly outside
    // already (the radius only shrinks, so it would be when popped).
    if (far >= 0 && !(s2 >= rad.tout)) {
      if (sp >= S) {
        atomicOr(status, 2u);
        return best;
      }
      stk[sp][threadIdx.x] = make_uint2((uint32_t)far, __float_as_uint(s2));
      ++sp;
    }
    if (near >= 0) {
      cur = near;
      p = T.load(near, Q.filter);
      continue;
    }
    int next = -1;
    while (sp > 0) {
      --sp;
      // the reference's pop test: (qa - split)^2 < radius, in double
      const uint2 top = stk[sp][threadIdx.x];
      const float s2 = __uint_as_float(top.y);
      if (s2 < rad.tin || (!(s2 >= rad.tout) &&
                           plane_d2(T.at(node_parent(T, (int)top.x)), Q) < rad.get(T, Q))) {
        next = (int)top.x;
        break;
      }
    }
    if (next < 0) break;
    cur = next;
    p = T.load(cur, Q.filter);
  }
  return best;
}

template <int S>
__global__ void __launch_bounds__(kKnnBlock, SKW_KNN_MINB) k_nearest(Tree T, const uint16_t *__restrict__ nids,
                                                 const double *__restrict__ dirs,
                                                 const double *__restrict__ q, const double *__restrict__ qn,
                                                 int64_t nq, double max_dist, double cos_t,
                                                 int32_t *__restrict__ out_idx, unsigned *__restrict__ status,
                                                 const int *__restrict__ nq_dev, const int32_t *__restrict__ order,
                                                 int per_warp) {
  __shared__ uint2 stk[S][kKnnBlock];
  const int lane = threadIdx.x & 31;
  if (lane >= per_warp) return;
  int64_t i = ((int64_t)blockIdx.x * (kKnnBlock / 32) + (threadIdx.x >> 5)) * per_warp + lane;
  if (nq_dev && *nq_dev < nq) nq = *nq_dev;
  if (i >= nq) return;
  if (order) i = order[i];
  Query Q;
  load_query(Q, q, qn, i, cos_t);
  out_idx[i] = nearest_walk<S, false>(T, nids, dirs, Q, max_dist, stk, status, 0);
}

// The walk of lane 0 where a scan met equal distances.
template <int S>
__device__ __noinline__ int nearest_walk_alone(Tree T, const uint16_t *nids, const double *dirs, const double *q,
                                               const double *qn, int64_t i, double max_dist, double cos_t,
                                               uint2 (*stk)[kKnnBlock], unsigned *status) {
  Query Q;
  load_query(Q, q, qn, i, cos_t);
  return nearest_walk<S, false>(T, nids, dirs, Q, max_dist, stk, status, 0);
}

// The nearest point of query i by looking at every point, one warp.  Equal
// exact distances are settled by the walk (the first visited stays), and so
// is the answer wherever one is met.
template <int S>
__device__ __forceinline__ void nearest_scan(Tree T, const uint16_t *__restrict__ nids,
                                             const double *__restrict__ dirs, const double *__restrict__ q,
                                             const double *__restrict__ qn, int64_t i, double max_dist, double cos_t,
                                             int32_t *__restrict__ out_idx, uint2 (*stk)[kKnnBlock],
                                             unsigned *__restrict__ status) {
  const int lane = threadIdx.x;
  Query Q;
  load_query(Q, q, qn, i, cos_t);
  Radius rad;
  rad.start(Q, max_dist);
  int best = -1;
  bool tie = false;
  for (int t0 = lane; t0 < T.n; t0 += 128) {
    float4 ps[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) ps[u] = T.at(min(t0 + 32 * u, T.n - 1));
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = t0 + 32 * u;
      const float4 p = ps[u];
      const float d2f = dist2f(p, Q);
      if (t >= T.n || d2f >= rad.tout) continue;
      bool equal = false;
      if (!(d2f < rad.tin)) {
        const double d = point_d2(p, Q), r = rad.get(T, Q);
        if (!(d <= r)) continue;
        equal = d == r;
      }
      if (Q.filter && !photon_filter(Q, NodeN{p, T.normal(t)}, t, nids, dirs)) continue;
      if (equal) {
        tie = true;
      } else {
        best = t;
        tie = false;
        rad.set(Q, t, d2f, 0.0f);
      }
    }
  }
  const double mine = best >= 0 ? point_d2(T.at(best), Q) : INFINITY;
  double least = mine;
  for (int o = 16; o > 0; o >>= 1) least = fmin(least, __shfl_xor_sync(0xffffffffu, least, o));
  const unsigned who = __ballot_sync(0xffffffffu, best >= 0 && mine == least);
  const bool ties = __ballot_sync(0xffffffffu, tie) != 0u || __popc(who) > 1;
  if (ties) {
    if (lane == 0) out_idx[i] = nearest_walk_alone<S>(T, nids, dirs, q, qn, i, max_dist, cos_t, stk, status);
  } else if (who == 0u) {
    if (lane == 0) out_idx[i] = -1;
  } else if (lane == __ffs(who) - 1) {
    out_idx[i] = best;
  }
}

// Launches of few queries over few points: their time is their longest walk,
// and a query whose filter takes no point near it walks the whole tree, one
// node after the other.  A walk is given up after `budget` nodes, and its warp
// looks at every point instead.
template <int S>
__global__ void __launch_bounds__(kKnnBlock, 16) k_nearest_few(
    Tree T, const uint16_t *__restrict__ nids, const double *__restrict__ dirs,
    const double *__restrict__ q, const double *__restrict__ qn, int64_t nq, double max_dist, double cos_t,
    int32_t *__restrict__ out_idx, unsigned *__restrict__ status, int per_warp, int budget) {
  static_assert(kKnnBlock == 32, "one warp per block");
  __shared__ uint2 stk[S][kKnnBlock];
  const int lane = threadIdx.x;
  const int64_t first = (int64_t)blockIdx.x * per_warp, i = first + lane;
  int found = -1;
  if (lane < per_warp && i < nq) {
    Query Q;
    load_query(Q, q, qn, i, cos_t);
    found = nearest_walk<S, true>(T, nids, dirs, Q, max_dist, stk, status, budget);
    if (found != kUnfinished) out_idx[i] = found;
  }
  for (unsigned left = __ballot_sync(0xffffffffu, found == kUnfinished); left != 0u; left &= left - 1u)
    nearest_scan<S>(T, nids, dirs, q, qn, first + __ffs(left) - 1, max_dist, cos_t, out_idx, stk, status);
}

// Walk stack entries for a tree of n points (see walk).
constexpr int kShallowStack = 20;
inline bool shallow_tree(int n) { return n < (1 << kShallowStack); }

// Queries per warp.  A warp's time is the sum of its lanes' divergent walks,
// so a launch with fewer queries than kSpreadWarps full warps -- about what is
// resident at k = 100 -- spreads them (the photon maps' 6,427 irradiance
// estimates: 3.90 -> 1.94 ms in 4s; 2s and 1s measure the same).
constexpr int64_t kSpreadWarps = 2048;
inline int queries_per_warp(int64_t nq, int64_t warps = kSpreadWarps) {
  const int64_t per = (nq + warps - 1) / warps;
  return (int)(per < 32 ? per : 32);
}
// Of heaps of more than 100 entries fewer fit into the SMs' shared memory
// (k = 128: 11 a SM), and a launch of a few warps more than that takes a second
// round of blocks (50,000 unfiltered queries of k = 128 with some 40 points
// each: 337 us in 2,000 warps, 213 in 1,667).
inline int64_t spread_warps(size_t smem) {
  constexpr size_t kSms = 152, kPerSm = 228 << 10, kStack = kShallowStack * kKnnBlock * 4, kReserved = 1024;
  const int64_t fit = (int64_t)(kSms * (kPerSm / (smem + kStack + kReserved)));
  return fit < kSpreadWarps ? fit : kSpreadWarps;
}
inline unsigned knn_grid(int64_t nq, int per_warp) {
  const int64_t per_block = (int64_t)per_warp * (kKnnBlock / 32);
  return (unsigned)((nq + per_block - 1) / per_block);
}

// Nearest points of few queries over few points: k_nearest_few, or with no
// walk at all (budget 0) where looking at every point takes no longer than a
// short walk.  Else a walk is given up after half as many nodes as its warp
// would take rounds of 128 points to look at all of them for each of its
// queries (a round takes about a node's time), so that a launch is never far
// from the less of walking and looking.  16,384 queries over 8,000 points, us,
// by full warps' walks / by looking alone / so: all points pass 76 / 84 / 38,
// the normals alike 86 / 272 / 41, radii of a point or two 30 / 122 / 19, a
// filter that no near point passes 6,850 / 286 / 665; 64 queries over 2,000
// points, the same: 59 / 22 / 22, 65 / 28 / 28, 17 / 16 / 16, 1,600 / 33 / 33.
constexpr int64_t kScanPoints = 8192, kScanQueries = 16384, kLookPoints = 2048, kLookQueries = 2048, kLookFrom = 16;
inline int nearest_budget(int64_t nq, int n, int per_warp) {
  if (n <= kLookPoints && nq >= kLookFrom && nq <= kLookQueries) return 0;
  return n * per_warp / 256 + 24;
}

// Levels of the median-split tree of n points: as many entries as a walk's
// stack can hold.
inline int tree_levels(int n) {
  int levels = 1;
  for (int64_t m = n; m > 1; m >>= 1) ++levels;
  return levels;
}

// Whether lanes wait for one another at heaps in global memory.  Beyond two
// rounds of blocks the walks' number counts more than the waits (heaps and
// nodes share L2).  k_knn_gang / k_knn, k = 200 over 270,000 points, radii of
// 300 and of 600: 110,000 queries 3.71 / 5.65 and 5.47 / 6.91 ms, 130,000 5.41 /
// 5.98 and 8.07 / 7.62, 200,000 7.75 / 10.42 and 11.34 / 12.57, 300,000 14.36 /
// 13.77 and 21.62 / 19.86, 600,000 34.42 / 29.23 and 53.66 / 49.00.
inline bool gang_in_global(int64_t nq) { return nq <= (int64_t)2 * 152 * kGangBlocks * kKnnBlock; }

// Full warps with heaps of more than kGangEntries entries: k_knn_gang.  The others:
// k_knn<KMAX, S> with S chosen by the tree's depth.
template <int KMAX>
void knn_kernel(cudaStream_t stream, const Tree &T, const uint16_t *nids, const double *dirs, const double *q,
                const double *qn, int64_t nq, int k, double max_dist, double cos_t, int32_t *out_idx, double *out_d2,
                int32_t *out_count, int32_t *out_visited, FCand *scratch, unsigned *status, const int *nq_dev,
                const int32_t *order) {
  const size_t smem = KMAX > 0 ? SharedHeap::bytes(k) : 0;
  const int per_warp = queries_per_warp(nq, spread_warps(smem));
  const unsigned grid = knn_grid(nq, per_warp);
  if constexpr (KMAX != 32) {
    if (per_warp == 32 && k > kGangEntries && (KMAX > 0 || gang_in_global(nq))) {
      const int depth = tree_levels(T.n);
      k_knn_gang<KMAX><<<grid, kKnnBlock, smem + (size_t)depth * kKnnBlock * sizeof(uint2), stream>>>(
          T, nids, dirs, q, qn, nq, k, max_dist, cos_t, out_idx, out_d2, out_count, out_visited, scratch, status, nq_dev,
          order, depth);
      return;
    }
  }
  if (shallow_tree(T.n))
    k_knn<KMAX, kShallowStack><<<grid, kKnnBlock, smem, stream>>>(T, nids, dirs, q, qn, nq, k, max_dist, cos_t, out_idx,
                                                               out_d2, out_count, out_visited, scratch, status, nq_dev,
                                                               order, per_warp);
  else
    k_knn<KMAX, 32><<<grid, kKnnBlock, smem, stream>>>(T, nids, dirs, q, qn, nq, k, max_dist, cos_t, out_idx, out_d2,
                                                    out_count, out_visited, scratch, status, nq_dev, order, per_warp);
}

inline Tree tree_of(const void *nodes, const uint16_t *nids, int n) {
  return Tree{(const float4 *)nodes,
              reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(nids) + nids_offset(n)), n};
}

// Spatial bins of queries: a box cut into 64^3 cells, each query's cell as
// an 18-bit Morton code; a counting sort by cell (count, one exclusive scan,
// scatter) gives the order in which the lookup kernels take the queries, so
// that a warp's walks start near each other.  The order inside a cell
// follows the atomics; every query's answer is the same whichever thread
// computes it, and it is written at the query's own index.
constexpr int kBinBits = 6, kBins = 1 << (3 * kBinBits);
#ifndef SKW_KNN_SORT_BITS
#define SKW_KNN_SORT_BITS 6  // cell bits per axis of the sorted order (1..10)
#endif
constexpr int kSortCellBits = SKW_KNN_SORT_BITS;
static_assert(kSortCellBits >= 1 && kSortCellBits <= 10, "sorted cells: 1 to 10 bits per axis");

__device__ __forceinline__ uint32_t spread3(uint32_t v) {  // bit b of v (v < 2^10) to bit 3b
  uint32_t r = 0;
#pragma unroll
  for (int b = 0; b < 10; ++b) r |= ((v >> b) & 1u) << (3 * b);
  return r;
}

template <int BITS>
__global__ void k_bin_keys(const double *__restrict__ q, int64_t n, const int *__restrict__ count, float3 lo,
                           float3 scale, uint32_t *__restrict__ key, int *__restrict__ bins) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || (count && i >= *count)) return;
  const float c[3] = {((float)q[3 * i] - lo.x) * scale.x, ((float)q[3 * i + 1] - lo.y) * scale.y,
                      ((float)q[3 * i + 2] - lo.z) * scale.z};
  uint32_t k = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float f = fminf(fmaxf(c[a], 0.0f), (float)((1 << BITS) - 1));  // NaN -> 0
    k |= spread3((uint32_t)f) << a;
  }
  key[i] = k;
  if (bins) atomicAdd(bins + k, 1);
}

// Exclusive scan of the kBins counts in place, one block of 1024 threads.
__global__ void __launch_bounds__(1024) k_bin_scan(int *__restrict__ bins) {
  constexpr int per = kBins / 1024;
  __shared__ int part[1024];
  int local[per];
  int sum = 0;
  for (int j = 0; j < per; ++j) {
    local[j] = sum;
    sum += bins[threadIdx.x * per + j];
  }
  part[threadIdx.x] = sum;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {  // inclusive Hillis-Steele scan of the parts
    const int v = threadIdx.x >= (unsigned)off ? part[threadIdx.x - off] : 0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  const int base = part[threadIdx.x] - sum;
  for (int j = 0; j < per; ++j) bins[threadIdx.x * per + j] = base + local[j];
}

__global__ void k_bin_scatter(const uint32_t *__restrict__ key, int64_t n, const int *__restrict__ count,
                              int *__restrict__ bins, int32_t *__restrict__ order) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || (count && i >= *count)) return;
  // the lanes of one cell take consecutive slots in lane order (one atomic
  // per cell and warp), so runs of neighbouring queries stay in order
  const uint32_t k = key[i];
  const unsigned grp = __match_any_sync(__activemask(), k);
  const int lane = threadIdx.x & 31, leader = __ffs(grp) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(bins + k, __popc(grp));
  base = __shfl_sync(grp, base, leader);
  order[base + __popc(grp & ((1u << lane) - 1u))] = (int32_t)i;
}

// A stable LSD radix sort of the cell keys (3 × SKW_KNN_SORT_BITS bits, 6-bit
// digits, one pass per digit) carrying the query indices: per block of 256 keys, each digit's
// count (lanes of a warp grouped by digit with __match_any_sync), one
// exclusive scan of the counts digit-major (all blocks of digit 0, then
// digit 1, ...), and a scatter that ranks a key after the block's earlier
// warps and the warp's earlier lanes with the same digit.  Stable, so the
// queries of a cell keep their image order.
constexpr int kSortBlock = 256, kDigitBits = 6, kDigits = 1 << kDigitBits;

__device__ __forceinline__ void digit_counts(uint32_t d, bool valid, unsigned &grp, int (*wcnt)[kDigits]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  grp = __match_any_sync(0xffffffffu, valid ? d : 0xFFFFFFFFu);
  if (valid && lane == __ffs(grp) - 1) wcnt[w][d] = __popc(grp);
}

__global__ void __launch_bounds__(kSortBlock) k_sort_hist(const uint32_t *__restrict__ key, int64_t n, int shift,
                                                          uint64_t *__restrict__ hist, int64_t nblocks) {
  __shared__ int wcnt[kSortBlock / 32][kDigits];
  for (int j = threadIdx.x; j < (kSortBlock / 32) * kDigits; j += kSortBlock) (&wcnt[0][0])[j] = 0;
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * kSortBlock + threadIdx.x;
  const bool valid = i < n;
  const uint32_t d = valid ? (key[i] >> shift) & (kDigits - 1) : 0u;
  unsigned grp;
  digit_counts(d, valid, grp, wcnt);
  __syncthreads();
  if (threadIdx.x < kDigits) {
    int c = 0;
    for (int w = 0; w < kSortBlock / 32; ++w) c += wcnt[w][threadIdx.x];
    hist[(int64_t)threadIdx.x * nblocks + blockIdx.x] = (uint64_t)c;
  }
}

__global__ void __launch_bounds__(kSortBlock) k_sort_scatter(const uint32_t *__restrict__ key,
                                                             const int32_t *__restrict__ val, int64_t n, int shift,
                                                             const uint64_t *__restrict__ offs, int64_t nblocks,
                                                             uint32_t *__restrict__ key2, int32_t *__restrict__ val2) {
  __shared__ int wcnt[kSortBlock / 32][kDigits];
  for (int j = threadIdx.x; j < (kSortBlock / 32) * kDigits; j += kSortBlock) (&wcnt[0][0])[j] = 0;
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * kSortBlock + threadIdx.x;
  const bool valid = i < n;
  const uint32_t k = valid ? key[i] : 0u, d = (k >> shift) & (kDigits - 1);
  unsigned grp;
  digit_counts(d, valid, grp, wcnt);
  __syncthreads();
  if (!valid) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int before = 0;
  for (int v = 0; v < w; ++v) before += wcnt[v][d];
  const int64_t dst = (int64_t)offs[(int64_t)d * nblocks + blockIdx.x] + before + __popc(grp & ((1u << lane) - 1u));
  key2[dst] = k;
  val2[dst] = val ? val[i] : (int32_t)i;
}

__global__ void k_node_records(const float4 *__restrict__ nodes, const uint16_t *__restrict__ nids, int64_t n,
                               const float *__restrict__ dirs_f, float4 *__restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float *d = dirs_f + 3 * (int)nids[i];
  out[2 * i] = nodes[i];
  out[2 * i + 1] = make_float4(d[0], d[1], d[2], 0.0f);
}

}  // namespace

cudaError_t launch_node_records(const void *nodes, uint16_t *nids, int64_t n, const double *dirs, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_node_records<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
      (const float4 *)nodes, nids, n, reinterpret_cast<const float *>(dirs + (3 << 16)),
      reinterpret_cast<float4 *>(reinterpret_cast<char *>(nids) + nids_offset(n)));
  return cudaGetLastError();
}

int64_t bin_order_bins() { return kBins; }

size_t sort_order_bytes(int64_t n) {
  const int64_t nb = (n + kSortBlock - 1) / kSortBlock, m = nb * kDigits;
  auto al = [](int64_t x) { return (size_t)((x + 255) & ~(int64_t)255); };
  return 3 * al(n * 4) + al(m * 8) + al(((m + 255) / 256) * 8);
}

cudaError_t launch_sort_order(const double *q, int64_t n, const float lo[3], const float hi[3], void *scratch,
                              int32_t *order, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int64_t nb = (n + kSortBlock - 1) / kSortBlock, m = nb * kDigits;
  auto al = [](int64_t x) { return (size_t)((x + 255) & ~(int64_t)255); };
  char *w = (char *)scratch;
  uint32_t *ka = (uint32_t *)w, *kb = (uint32_t *)(w + al(n * 4));
  int32_t *va = (int32_t *)(w + 2 * al(n * 4)), *vb = order;
  uint64_t *hist = (uint64_t *)(w + 3 * al(n * 4));
  uint64_t *sums = (uint64_t *)((char *)hist + al(m * 8));
  float sc[3];
  for (int a = 0; a < 3; ++a) {
    const float ext = hi[a] - lo[a];
    sc[a] = ext > 0.0f && ext < INFINITY ? (float)(1 << kSortCellBits) / ext : 0.0f;
  }
  k_bin_keys<kSortCellBits><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
      q, n, nullptr, make_float3(lo[0], lo[1], lo[2]), make_float3(sc[0], sc[1], sc[2]), ka, nullptr);
  // passes alternate ka/kb for the keys and va/vb for the indices, the
  // indices' parity chosen so that the last pass lands in order (vb)
  constexpr int passes = (3 * kSortCellBits + kDigitBits - 1) / kDigitBits;
  const int32_t *vin = nullptr;
  for (int pass = 0; pass < passes; ++pass) {
    const int shift = pass * kDigitBits;
    uint32_t *kin = pass % 2 ? kb : ka, *kout = pass % 2 ? ka : kb;
    int32_t *vout = (passes - 1 - pass) % 2 ? va : vb;
    k_sort_hist<<<(unsigned)nb, kSortBlock, 0, st>>>(kin, n, shift, hist, nb);
    cudaError_t e = scan64(hist, m, sums, st);
    if (e != cudaSuccess) return e;
    k_sort_scatter<<<(unsigned)nb, kSortBlock, 0, st>>>(kin, vin, n, shift, hist, nb, kout, vout);
    vin = vout;
  }
  return cudaGetLastError();
}

cudaError_t launch_bin_order(const double *q, int64_t n, const int *count_dev, const float lo[3], const float hi[3],
                             uint32_t *keys, int *bins, int32_t *order, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  float sc[3];
  for (int a = 0; a < 3; ++a) {
    const float ext = hi[a] - lo[a];
    sc[a] = ext > 0.0f && ext < INFINITY ? (float)(1 << kBinBits) / ext : 0.0f;
  }
  const unsigned grid = (unsigned)((n + 255) / 256);
  cudaError_t e = cudaMemsetAsync(bins, 0, (size_t)kBins * 4, st);
  if (e != cudaSuccess) return e;
  k_bin_keys<kBinBits><<<grid, 256, 0, st>>>(q, n, count_dev, make_float3(lo[0], lo[1], lo[2]),
                                   make_float3(sc[0], sc[1], sc[2]), keys, bins);
  k_bin_scan<<<1, 1024, 0, st>>>(bins);
  k_bin_scatter<<<grid, 256, 0, st>>>(keys, n, count_dev, bins, order);
  return cudaGetLastError();
}

#ifndef SKW_KNN_GHEAP
#define SKW_KNN_GHEAP 129  // smallest k whose heaps live in global scratch
#endif
size_t knn_scratch_bytes(int64_t nq, int k) {
  return k >= SKW_KNN_GHEAP ? (size_t)nq * (size_t)knn_heap_stride(k) * sizeof(FCand) : 0;
}

cudaError_t launch_knn(const void *nodes, const uint16_t *nids, const double *dirs, int n, const double *q,
                       const double *qn, int64_t nq, int k, double max_dist, double cos_t, int32_t *out_idx,
                       double *out_d2, int32_t *out_count, int32_t *out_visited, void *scratch, unsigned *status,
                       cudaStream_t stream, const int *nq_dev, const int32_t *order) {
  if (nq <= 0) return cudaSuccess;
  const Tree T = tree_of(nodes, nids, n);
  if (scratch && k >= SKW_KNN_GHEAP) {
    knn_kernel<0>(stream, T, nids, dirs, q, qn, nq, k, max_dist, cos_t, out_idx, out_d2, out_count,
                  out_visited, (FCand *)scratch, status, nq_dev, order);
  } else if (k <= 32) {
    knn_kernel<32>(stream, T, nids, dirs, q, qn, nq, k, max_dist, cos_t, out_idx, out_d2, out_count,
                   out_visited, nullptr, status, nq_dev, order);
  } else if (k <= 128) {
    knn_kernel<128>(stream, T, nids, dirs, q, qn, nq, k, max_dist, cos_t, out_idx, out_d2, out_count,
                    out_visited, nullptr, status, nq_dev, order);
  } else {
    if (!scratch) return cudaErrorInvalidValue;
    knn_kernel<0>(stream, T, nids, dirs, q, qn, nq, k, max_dist, cos_t, out_idx, out_d2, out_count,
                  out_visited, (FCand *)scratch, status, nq_dev, order);
  }
  return cudaGetLastError();
}

int64_t knn_noalloc_capacity() { return SKW_KNN_NOALLOC_ENTRIES; }

// The calling thread's current CUDA context (the driver's cuCtxGetCurrent,
// reached through the runtime so that the library needs no link against the
// driver library); null where the driver does not offer it.
static void *current_context() {
  using Fn = CUresult (*)(CUcontext *);
  static const Fn fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return (Fn)p;
  }();
  CUcontext c = nullptr;
  if (!fn || fn(&c) != CUDA_SUCCESS) return nullptr;
  return (void *)c;
}

// Device address of the static scratch for the current device, looked up
// once per device (cudaGetSymbolAddress with that device current; the first
// lookup may load this module on the device) and again whenever the
// device's current context has changed since (a device reset destroys the
// context and the module with it; the next context loads the module anew).
static cudaError_t knn_noalloc_scratch(void **out) {
  static std::mutex mu;
  static void *addr[64] = {nullptr};
  static void *owner[64] = {nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  // make the device's primary context current (a no-op when it already is)
  if ((e = cudaFree(nullptr)) != cudaSuccess) return e;
  void *ctx = current_context();
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev] || owner[dev] != ctx) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_knn_noalloc_scratch);
    if (e != cudaSuccess) return e;
    addr[dev] = p;
    owner[dev] = ctx;
  }
  *out = addr[dev];
  return cudaSuccess;
}

cudaError_t launch_knn_noalloc(const void *nodes, const uint16_t *nids, const double *dirs, int n, const double *q,
                               const double *qn, int64_t nq, int k, double max_dist, double cos_t,
                               int32_t *out_idx, double *out_d2, int32_t *out_count, unsigned *status,
                               cudaStream_t stream) {
  if (nq <= 0) return cudaSuccess;
  if (nq * (int64_t)k > SKW_KNN_NOALLOC_ENTRIES) return cudaErrorInvalidValue;
  void *scratch = nullptr;
  cudaError_t e = knn_noalloc_scratch(&scratch);
  if (e != cudaSuccess) return e;
  // Every heap slot is written before it is read, so the array needs no
  // clearing between calls.
  knn_kernel<0>(stream, tree_of(nodes, nids, n), nids, dirs, q, qn, nq, k, max_dist, cos_t, out_idx, out_d2,
                out_count, nullptr, (FCand *)scratch, status, nullptr, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_nearest(const void *nodes, const uint16_t *nids, const double *dirs, int n, const double *q,
                           const double *qn, int64_t nq, double max_dist, double cos_t, int32_t *out_idx,
                           unsigned *status, cudaStream_t stream, const int *nq_dev, const int32_t *order) {
  if (nq <= 0) return cudaSuccess;
  const Tree T = tree_of(nodes, nids, n);
  const int per_warp = queries_per_warp(nq);
  const unsigned grid = knn_grid(nq, per_warp);
  if (!nq_dev && !order && n <= kScanPoints && nq <= kScanQueries)
    k_nearest_few<kShallowStack><<<grid, kKnnBlock, 0, stream>>>(T, nids, dirs, q, qn, nq, max_dist, cos_t, out_idx,
                                                                 status, per_warp, nearest_budget(nq, n, per_warp));
  else if (shallow_tree(n))
    k_nearest<kShallowStack><<<grid, kKnnBlock, 0, stream>>>(T, nids, dirs, q, qn, nq, max_dist,
                                                         cos_t, out_idx, status, nq_dev, order, per_warp);
  else
    k_nearest<32><<<grid, kKnnBlock, 0, stream>>>(T, nids, dirs, q, qn, nq, max_dist, cos_t,
                                              out_idx, status, nq_dev, order, per_warp);
  return cudaGetLastError();
}

}  // namespace skw
