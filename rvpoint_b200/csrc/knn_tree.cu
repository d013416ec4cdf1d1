// Exact k nearest neighbours in one cloud (k <= 64) over a 32-wide box tree.
//
// Build: the points sorted by the Hilbert code of their quantised position
// (32 bits, one power-of-two cell for all axes), every 32 consecutive points
// a leaf with its bounding box, every 32 leaves a node, and so on, four levels
// in all. No cell size is chosen and nothing depends on the
// density: a leaf is small where the points are dense.
//
// Search: one warp answers 32 queries that lie close together (the points of
// a leaf, or 32 consecutive queries of a sorted query set). The lanes test
// the boxes of 32 children at once against the box of the queries and go down
// into those nearer than the largest K-th distance so far, nearest first; a
// leaf's points are staged in shared memory and every lane tests all of them
// against its own query. The distances that pass wait in a buffer per lane;
// when one fills, every lane sorts its own in registers and merges them into
// its sorted list, all lanes in step. With the K-th distance known, the leaves
// scanned are gone over again, the points within it collected and each put at
// its rank. Queries that do not fit this (far from their packet, equal
// distances) are listed and answered one per warp by a second kernel.
//
// Pruning needs no slack: every operation of the distance (subtract, square,
// add) is monotone under rounding, so the distance to a box computed with the
// same operations is never above the computed distance to a point inside it.
// Equal distances are ordered by index: the second kernel works on packed
// (distance, index) keys.
//
// Bound by issue (distance tests, list networks, box tests); small clouds by
// the latency of one packet. The grid search it replaces for single clouds ran
// one warp per query on cells sized from a sample of queries: 105k LiDAR
// points, k 16: 3818 us, now 171 us; 89k room points, mean of 30: 863 and
// 254 us; normals of a 2M-point map, k 32: 15.9 ms and 4.0 ms.
#include <float.h>
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "grid_device.cuh"
#include "internal.cuh"
#include "normals_device.cuh"
#include "tree_device.cuh"

namespace rvp {
using namespace gd;
using namespace td;

namespace {
inline size_t al(size_t b) { return (b + 255) & ~(size_t)255; }

constexpr int kTreeKeyBits = 32;

// ---------------------------------------------------------------------------
// build
// ---------------------------------------------------------------------------
struct TreeFrame {  // the quantisation of the cloud's box
  float lo[3];
  float inv;    // cells per unit (a power of two)
  int bits[3];  // of each axis, kTreeKeyBits together at most
};

__global__ void k_tree_init(float *bb) {
  if (threadIdx.x < 3) bb[threadIdx.x] = INFINITY;
  else if (threadIdx.x < 6) bb[threadIdx.x] = -INFINITY;
}

// the finest power-of-two cell whose codes fit the key
__device__ void tree_frame(const float *bb, TreeFrame &F) {
  float ext[3], emax = 0.0f;
  for (int a = 0; a < 3; ++a) {
    const float lo = bb[a], hi = bb[3 + a];
    F.lo[a] = lo < INFINITY && lo > -INFINITY ? lo : 0.0f;
    float e = fsub(hi, lo);
    e = e > 0.0f ? fminf(e, 1e30f) : 0.0f;  // (NaN and empty axes: one cell)
    ext[a] = e;
    emax = fmaxf(emax, e);
  }
  int k = emax > 0.0f ? ilogbf(emax) - kTreeKeyBits : -60;
  k = max(k, -100);
  for (;; ++k) {
    int sum = 0;
    for (int a = 0; a < 3; ++a) {
      const float q = ldexpf(ext[a], -k);  // cells along the axis
      F.bits[a] = q < 1.0f ? 0 : ilogbf(q) + 1;
      sum += F.bits[a];
    }
    if (sum <= kTreeKeyBits) break;
  }
  F.inv = ldexpf(1.0f, -k);
}

__device__ __forceinline__ u32 tree_key(const TreeFrame &F, float x, float y, float z) {
  const float v[3] = {x, y, z};
  u32 q[3];
  int top = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float t = fmul(fsub(v[a], F.lo[a]), F.inv);
    const u32 last = F.bits[a] >= 32 ? 0xFFFFFFFFu : (1u << F.bits[a]) - 1u;
    q[a] = t > 0.0f ? (t < 4.0e9f ? min((u32)t, last) : last) : 0u;
    top = max(top, F.bits[a]);
  }
  // Compact Hilbert index (C. Hamilton, A. Rau-Chaplin, "Compact Hilbert
  // indices", 2008): per level the Gray code rank of the point's octant in the
  // frame of the entry e and direction d, over the axes that have this bit.
  // Consecutive codes are neighbouring cells (but for a few jumps where an
  // axis has run out of bits), so a leaf's box is small: with Morton codes
  // packets tested 19 to 41 leaves, one that spans a jump all of a large box.
  constexpr u32 kGray = 0x54672310u, kEntry = 0x56633000u, kDir = 0x01122110u;
  auto rotr = [](u32 v, u32 k) { return ((v >> k) | (v << (3 - k))) & 7u; };
  u32 key = 0, e = 0, d = 0;
  for (int b = top - 1; b >= 0; --b) {
    const u32 mask = (b < F.bits[0] ? 1u : 0u) | (b < F.bits[1] ? 2u : 0u) |
                     (b < F.bits[2] ? 4u : 0u);
    const u32 l = ((q[0] >> b) & 1u) | (((q[1] >> b) & 1u) << 1) | (((q[2] >> b) & 1u) << 2);
    const u32 k = d == 2 ? 0 : d + 1;
    const u32 w = (kGray >> (4 * rotr(l ^ e, k))) & 7u;
    const u32 mu = rotr(mask, k);
    if (mu & 4u) key = (key << 1) | (w >> 2);
    if (mu & 2u) key = (key << 1) | ((w >> 1) & 1u);
    if (mu & 1u) key = (key << 1) | (w & 1u);
    e ^= rotr((kEntry >> (4 * w)) & 7u, 3 - k);
    d += ((kDir >> (4 * w)) & 7u) + 1;
    d = d >= 3 ? d - 3 : d;
  }
  return key;
}

__global__ __launch_bounds__(256) void k_tree_keys(const float *__restrict__ x,
                                                   const float *__restrict__ y,
                                                   const float *__restrict__ z, size_t n_max,
                                                   const u64 *n_dev, const float *bb, u64 *keys,
                                                   u32 *vals) {
  __shared__ TreeFrame F;
  const size_t n = n_dev ? *n_dev : n_max;
  if (threadIdx.x == 0) tree_frame(bb, F);
  __syncthreads();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    keys[i] = tree_key(F, x[i], y[i], z[i]);
    vals[i] = (u32)i;
  }
}

// box reduction over a warp; lane 0 writes node `c` of a level
__device__ __forceinline__ void box_out(float (&m)[6], float *box, u32 stride, u32 c) {
#pragma unroll
  for (int k = 0; k < 6; ++k) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const float t = __shfl_xor_sync(0xffffffffu, m[k], o);
      m[k] = k < 3 ? fminf(m[k], t) : fmaxf(m[k], t);
    }
  }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int k = 0; k < 6; ++k) box[(size_t)k * stride + c] = m[k];
  }
}

// one warp per leaf: its records in tree order and its box
__global__ __launch_bounds__(256) void k_tree_leaves(const float *__restrict__ x,
                                                     const float *__restrict__ y,
                                                     const float *__restrict__ z,
                                                     const u32 *__restrict__ vals, u32 n,
                                                     float4 *pts, u32 *pos_of, float *box,
                                                     u32 stride) {
  const u32 c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, i = c * 32 + (threadIdx.x & 31);
  if (c * 32 >= n) return;
  float m[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  if (i < n) {
    const u32 v = vals[i];
    const float p[3] = {x[v], y[v], z[v]};
    pts[i] = make_float4(p[0], p[1], p[2], __uint_as_float(v));
    pos_of[v] = i;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      m[a] = fminf(m[a], p[a]);
      m[3 + a] = fmaxf(m[3 + a], p[a]);
    }
  }
  box_out(m, box, stride, c);
}

// one warp per node of the next level: the box of up to 32 children
__device__ __forceinline__ void parent_box(const float *kid, u32 kid_stride, u32 kids, float *box,
                                           u32 stride, u32 c) {
  const u32 i = c * 32 + (threadIdx.x & 31);
  float m[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  if (i < kids) {
#pragma unroll
    for (int k = 0; k < 6; ++k) m[k] = kid[(size_t)k * kid_stride + i];
  }
  box_out(m, box, stride, c);
}

__global__ __launch_bounds__(256) void k_tree_parents(TreeView t, int level) {
  const u32 c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= t.count[level]) return;
  parent_box(t.box[level - 1], t.stride[level - 1], t.count[level - 1], t.box[level],
             t.stride[level], c);
}

// the levels from `level` on, by one block
__global__ __launch_bounds__(1024) void k_tree_top(TreeView t, int level) {
  for (; level < kTreeLevels; ++level) {
    for (u32 c = threadIdx.x >> 5; c < t.count[level]; c += 32)
      parent_box(t.box[level - 1], t.stride[level - 1], t.count[level - 1], t.box[level],
                 t.stride[level], c);
    __syncthreads();
  }
}

// 0 in *n_sort if the queries are the cloud itself, value by value, else nq:
// the sort of the queries then has nothing to do
__global__ void k_tree_same(const float *qx, const float *qy, const float *qz, const float *x,
                            const float *y, const float *z, size_t n, u64 *n_sort) {
  bool differs = false;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    differs = differs || __float_as_uint(qx[i]) != __float_as_uint(x[i]) ||
              __float_as_uint(qy[i]) != __float_as_uint(y[i]) ||
              __float_as_uint(qz[i]) != __float_as_uint(z[i]);
  if (__any_sync(0xffffffffu, differs) && (threadIdx.x & 31) == 0) *n_sort = n;
}
__global__ void k_tree_count(u64 *n_sort, u64 v) { *n_sort = v; }

__global__ void k_tree_queries(const float *__restrict__ x, const float *__restrict__ y,
                               const float *__restrict__ z, const u32 *__restrict__ vals,
                               const u64 *n_sort, float4 *q) {
  const size_t n = *n_sort;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const u32 v = vals[i];
    q[i] = make_float4(x[v], y[v], z[v], __uint_as_float(v));
  }
}

// ---------------------------------------------------------------------------
// search
// ---------------------------------------------------------------------------
// Walks every leaf within limit() of the box q, nearest child first. All
// lanes take part; limit() is uniform and may shrink on the way.
template <int LV, class Limit, class Leaf>
__device__ __forceinline__ void tree_walk(const TreeView &t, const Box &q, u32 first, Limit &limit,
                                          Leaf &leaf) {
  const int lane = threadIdx.x & 31;
  const u32 c = first + lane;
  const float lb = c < t.count[LV] ? box_d2(q, t.box[LV], t.stride[LV], c) : 0.0f;
  bool open = c < t.count[LV] && lb <= limit();
  while (true) {
    // (the low bits of the distance give way to the lane)
    const u32 key = open ? (__float_as_uint(lb) & ~31u) | lane : 0xFFFFFFFFu;
    const u32 best = __reduce_min_sync(0xffffffffu, key);
    if (best == 0xFFFFFFFFu) break;
    const int s = best & 31;
    if (lane == s) open = false;
    if (__uint_as_float(best & ~31u) > limit()) break;  // and so are all that are left
    if (__shfl_sync(0xffffffffu, lb, s) > limit()) continue;
    if constexpr (LV == 0) leaf(first + s);
    else tree_walk<LV - 1>(t, q, (first + s) * 32, limit, leaf);
  }
}
// (at most 32 nodes are left at the top up to 33.5M points; more than that go
// 32 at a time)
template <class Limit, class Leaf>
__device__ __forceinline__ void tree_walk_all(const TreeView &t, const Box &q, Limit &limit,
                                              Leaf &leaf) {
  for (u32 f = 0; f < t.count[kTreeLevels - 1]; f += 32)
    tree_walk<kTreeLevels - 1>(t, q, f, limit, leaf);
}

// The same walk leaf by leaf, for a caller whose leaf code is too long to be
// inlined more than once (it would not fit the instruction cache).
template <class T>
__device__ __forceinline__ T by_level(const T (&v)[kTreeLevels], int l) {
  static_assert(kTreeLevels == 4, "four levels");
  return l < 2 ? (l == 0 ? v[0] : v[1]) : (l == 2 ? v[2] : v[3]);  // (stays in registers)
}
template <class T>
__device__ __forceinline__ void set_level(T (&v)[kTreeLevels], int l, T x) {
#pragma unroll
  for (int i = 0; i < kTreeLevels; ++i) v[i] = i == l ? x : v[i];
}

struct TreeWalk {
  float lb[kTreeLevels];   // per level: the lane's child's distance
  u32 open[kTreeLevels];   // children left (a mask, uniform)
  u32 first[kTreeLevels];  // their numbers start here
  int level;               // where the walk stands
  u32 top;                 // next group of top nodes
  __device__ __forceinline__ void begin() {
    level = kTreeLevels;
    top = 0;
#pragma unroll
    for (int l = 0; l < kTreeLevels; ++l) {
      lb[l] = 0.0f;
      open[l] = first[l] = 0;
    }
  }
  // the next leaf within `limit` of q; false at the end
  __device__ __forceinline__ bool next(const TreeView &t, const Box &q, float limit, u32 &leaf) {
    const int lane = threadIdx.x & 31;
    while (true) {
      u32 f = top;
      int to = kTreeLevels - 1;
      if (level == kTreeLevels) {
        if (top >= t.count[kTreeLevels - 1]) return false;
        top += 32;
      } else {
        const u32 mask = by_level(open, level);
        const float v = by_level(lb, level);
        // (the low bits of the distance give way to the lane)
        const u32 best = __reduce_min_sync(
            0xffffffffu,
            (mask >> lane) & 1u ? (__float_as_uint(v) & ~31u) | lane : 0xFFFFFFFFu);
        if (best == 0xFFFFFFFFu || __uint_as_float(best & ~31u) > limit) {  // none near enough
          ++level;
          continue;
        }
        const int s = best & 31;
        set_level(open, level, mask & ~(1u << s));
        if (__shfl_sync(0xffffffffu, v, s) > limit) continue;
        f = by_level(first, level) + s;
        if (level == 0) {
          leaf = f;
          return true;
        }
        f *= 32;
        to = level - 1;
      }
      const u32 c = f + lane, n = by_level(t.count, to);
      const float d = c < n ? box_d2(q, by_level(t.box, to), by_level(t.stride, to), c) : 0.0f;
      set_level(lb, to, d);
      set_level(open, to, __ballot_sync(0xffffffffu, c < n && d <= limit));
      set_level(first, to, f);
      level = to;
    }
  }
};

constexpr int kTreeBuf = 64;   // buffered distances per lane, flushed above 32
constexpr int kTreeExtra = 3;  // collected points past the list, for equal distances
// a query joins its packet's walk if its limit (a squared distance) is within
// this factor of the median one
constexpr float kLoner = 16.0f;
// leaves a packet tests before it gives up: one with points far apart has every
// leaf of a large box to test (milliseconds, with no other work left to hide
// them), most test 20 to 40
constexpr int kLeafBudget = 128;

// shared memory of a packet: the staged leaf, the leaves scanned, the buffered
// distances and later (in the same place) the collected points, and the
// positions in order where a normal follows
constexpr int kTreeLeaves = (kLeafBudget + 3 + 3) & ~3;
template <int KCAP, int MODE>
constexpr size_t tree_buffer() {
  constexpr size_t dist = (size_t)kTreeBuf * 32 * 4;
  constexpr size_t near = (size_t)(KCAP + kTreeExtra) * 32 * 8;
  return MODE != TREE_MEAN && near > dist ? near : dist;
}
template <int KCAP, int MODE>
constexpr size_t tree_smem() {
  return 3 * 32 * 4 + kTreeLeaves * 4 + tree_buffer<KCAP, MODE>() +
         (MODE == TREE_NORMALS || MODE == TREE_PRECISE ? (size_t)(KCAP + 1) * 32 * 4 : 0);
}

// Compare-exchange networks over registers. They are straight code: batches of
// 32 took fewer steps than 16, but the kernel then waited for instructions
// (4.7 of 9 cycles per issue).
__device__ __forceinline__ void order2(float &a, float &b) {
  const float l = fminf(a, b), h = fmaxf(a, b);
  a = l;
  b = h;
}
template <int N>
__device__ __forceinline__ void bitonic_merge(float (&v)[N]) {
#pragma unroll
  for (int j = N / 2; j > 0; j >>= 1) {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if ((i ^ j) > i) order2(v[i], v[i ^ j]);
  }
}
template <int N>
__device__ __forceinline__ void bitonic_sort(float (&v)[N]) {
#pragma unroll
  for (int k = 2; k <= N; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int l = i ^ j;
        if (l > i) {
          if ((i & k) == 0) order2(v[i], v[l]);
          else order2(v[l], v[i]);
        }
      }
    }
  }
}

// sor_sc's mean (statistical_outlier_removal.cpp:36-40): the ascending sum of
// sqrtf(d2_j), j = 1 .. k, over k; within a radius over those found, and the
// radius itself for a point without neighbours (:246-270)
__device__ __forceinline__ void tree_mean_out(float sum, int have, const float4 &q, u32 qidx,
                                              const TreeOut &o) {
  float m = have > 1 ? fdiv(sum, (float)(have - 1)) : 0.0f;
  if (o.radius_mode && have <= 1) m = o.fallback;
  const float none = dist2(q.x, q.y, q.z, q.x, q.y, q.z);  // NaN without a position
  o.mean[qidx] = none == 0.0f ? m : none;
}

// the normal of a query from its sorted neighbours nbr(0 .. have - 1)
template <int MODE, class Nbr>
__device__ __forceinline__ void tree_normal_out(Nbr nbr, int have, const float4 &q, u32 qidx,
                                                const TreeOut &o) {
  float nx = 0.0f, ny = 0.0f, nz = 0.0f;
  if constexpr (MODE == TREE_NORMALS) {
    if (have >= 3)
      nd::normal_from_points(nbr, have, true, o.iters, q.x, q.y, q.z, o.vpx, o.vpy, o.vpz, nx, ny,
                             nz);
  } else {
    float cond;
    bool wide;
    nd::precise_normal(nbr, have, q.x, q.y, q.z, o.vpx, o.vpy, o.vpz, o.cond_fp64, nx, ny, nz,
                       cond, wide);
    if (o.cond) o.cond[qidx] = cond;
    if (o.used64) o.used64[qidx] = wide ? 1 : 0;
  }
  o.nx[qidx] = nx;
  o.ny[qidx] = ny;
  o.nz[qidx] = nz;
}

// One warp (block) per packet of 32 queries. The list holds the K nearest, or
// for the cloud's own points the K - 1 nearest others (the point itself, at
// distance 0, is the first of its row); KCAP is at least that, a power of two.
template <int KCAP, int MODE>
__global__ __launch_bounds__(32, KCAP > 32 ? 10 : 16) void k_knn_tree(TreeView t, TreeQueries qs, int K,
                                                     float bound, TreeOut o) {
  extern __shared__ __align__(16) unsigned char tree_sm[];
  constexpr bool MEAN = MODE == TREE_MEAN;
  constexpr int PCAP = KCAP + kTreeExtra;
  constexpr int BATCH = KCAP < 16 ? KCAP : 16;  // distances sorted at once
  float(*stage)[32] = reinterpret_cast<float(*)[32]>(tree_sm);  // x, y, z
  u32 *leaves = reinterpret_cast<u32 *>(tree_sm + 384);
  unsigned char *buf = tree_sm + 384 + kTreeLeaves * 4;
  float(*fbuf)[32] = reinterpret_cast<float(*)[32]>(buf);
  uint2(*pbuf)[32] = reinterpret_cast<uint2(*)[32]>(buf);
  u32(*sorted)[32] = reinterpret_cast<u32(*)[32]>(buf + tree_buffer<KCAP, MODE>());
  const int lane = threadIdx.x;
  const u32 packet = blockIdx.x;
  // the cloud's own points (leaf `packet`), or 32 of the sorted queries
  const bool self = qs.n_sort == nullptr || *qs.n_sort == 0;
  const float4 *src = self ? t.pts : qs.q;
  const u32 qi = packet * 32 + lane;
  const bool active = qi < qs.n;
  const float4 q = src[active ? qi : packet * 32];
  const u32 qidx = __float_as_uint(q.w);
  u32 start = packet;
  if (!self) start = leaf_of_key(t, qs.keys[min(packet * 32 + 16, qs.n - 1)]);
  const Box own{{q.x, q.y, q.z}, {q.x, q.y, q.z}};

  // ---- the sorted distances: slots 0 .. pad - 1 hold -1 and never move
  const bool drop = self && K > 1;  // the point itself is not in the list
  const int KL = drop ? K - 1 : K, pad = KCAP - KL;
  float L[KCAP];
#pragma unroll
  for (int j = 0; j < KCAP; ++j) L[j] = j < pad ? -1.0f : INFINITY;
  bool mine = active;  // answered with the packet
  int cnt = 0;         // buffered distances
  float lim = -1.0f, pmax = -1.0f;  // what the buffer takes: d2 <= lim; its largest
  auto limits = [&]() {
    lim = mine ? fminf(fminf(L[KCAP - 1], bound), FLT_MAX) : -1.0f;
    pmax = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(lim)));
  };
  limits();
  auto flush = [&]() {
    const int most = __reduce_max_sync(0xffffffffu, cnt);
    int i = 0;
    // a sorted batch merged at once; the last few one by one
    for (; i + BATCH / 4 < most; i += BATCH) {
      float S[BATCH];
#pragma unroll
      for (int j = 0; j < BATCH; ++j) S[j] = i + j < cnt ? fbuf[i + j][lane] : INFINITY;
      bitonic_sort<BATCH>(S);
#pragma unroll
      for (int j = 0; j < BATCH; ++j)
        L[KCAP - BATCH + j] = fminf(L[KCAP - BATCH + j], S[BATCH - 1 - j]);
      bitonic_merge<KCAP>(L);
    }
    for (; i < most; ++i) {
      const float key = i < cnt ? fbuf[i][lane] : INFINITY;
#pragma unroll
      for (int j = KCAP - 1; j > 0; --j) L[j] = fmaxf(L[j - 1], fminf(L[j], key));
      L[0] = fminf(L[0], key);
    }
    cnt = 0;
    limits();
  };
  int scanned = 0, budget = kLeafBudget;
  auto stage_leaf = [&](u32 l, float at, const float4 &mate) {
    if (!__any_sync(0xffffffffu, at >= 0.0f)) return false;
    __syncwarp();
    stage[0][lane] = mate.x;
    stage[1][lane] = mate.y;
    stage[2][lane] = mate.z;
    __syncwarp();
    return true;
  };
  const u64 nqx = pack2(-q.x, -q.x), nqy = pack2(-q.y, -q.y), nqz = pack2(-q.z, -q.z);
  // hit(c, d2) for the staged points c within `at`, except `skip`
  auto test_staged = [&](float at, int skip, auto &&hit) {
#pragma unroll 2
    for (int c = 0; c < 32; c += 4) {
      const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(&stage[0][c]);
      const ulonglong2 y = *reinterpret_cast<const ulonglong2 *>(&stage[1][c]);
      const ulonglong2 z = *reinterpret_cast<const ulonglong2 *>(&stage[2][c]);
      const u64 a = dist2x2(x.x, y.x, z.x, nqx, nqy, nqz, qs.minus_zero);
      const u64 b = dist2x2(x.y, y.y, z.y, nqx, nqy, nqz, qs.minus_zero);
      const float d[4] = {half2f(a, 0), half2f(a, 1), half2f(b, 0), half2f(b, 1)};
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (d[u] <= at && c + u != skip) hit(c + u, d[u]);
    }
  };
  auto mate_of = [&](u32 l) {  // the lane's point of leaf l
    const u32 i = l * 32 + lane;
    return i < t.n ? __ldg(&t.pts[i]) : make_float4(INFINITY, INFINITY, INFINITY, 0.0f);
  };
  auto scan_leaf = [&](u32 l) {
    if (--budget < 0) {  // (uniform) nothing is left open: the walk ends
      mine = false;
      pmax = -1.0f;
      return;
    }
    const float4 mate = mate_of(l);
    const float at = box_d2(own, t.box[0], t.stride[0], l) <= lim ? lim : -1.0f;
    if (!stage_leaf(l, at, mate)) return;
    leaves[scanned++] = l;
    const int skip = drop && l == packet ? lane : -1;  // the point itself
    float *to = &fbuf[cnt][lane];
    test_staged(at, skip, [&](int, float d) {
      *to = d;
      to += 32;
    });
    cnt = (int)(to - &fbuf[0][lane]) >> 5;
  };
  // the leaves around the packet's place first (they set the limits), then
  // the walk
  const u32 s0 = start > 0 ? start - 1 : 0, s1 = min(start + 1, t.count[0] - 1);
  const int near = (int)(s1 - s0) + 1;
  Box pk{};  // the box of the packet
  TreeWalk walk;
  walk.begin();
  for (int step = 0;; ++step) {
    bool more = true;
    u32 l = step == 0 ? start : (step == 1 && s0 < start ? s0 : s1);
    if (step >= near) more = walk.next(t, pk, pmax, l);
    if (more && (step < near || l < s0 || l > s1)) scan_leaf(l);
    if (!more || step == 0 || step == near - 1 || __any_sync(0xffffffffu, cnt > kTreeBuf - 32))
      flush();
    if (!more) break;
    if (step != near - 1) continue;
    // A query whose limit is far above the others' (four times the median
    // radius) would take the packet through all the leaves around it
    int rank = 0;
    for (int i = 0; i < 32; ++i) {
      const float other = __shfl_sync(0xffffffffu, mine ? lim : INFINITY, i);
      rank += other < lim || (other == lim && i < lane) ? 1 : 0;
    }
    const unsigned mid = __ballot_sync(0xffffffffu, mine && rank == 16);
    if (mid) {
      const float ref = __shfl_sync(0xffffffffu, lim, __ffs(mid) - 1);
      mine = mine && lim <= kLoner * ref;
      limits();
    }
    pk = warp_box(q, mine);
  }

  // ---- results of the packet
  bool exact = mine;
  int have = 0;  // distances in the list
  if constexpr (MEAN) {
    // (without a radius they are all there, some infinitely far perhaps)
    float sum = 0.0f;
    bool first = !drop;  // the nearest of all does not count
#pragma unroll
    for (int j = 0; j < KCAP; ++j) {
      if (j >= pad && (!o.radius_mode || L[j] < INFINITY)) {
        if (!first) sum = fadd(sum, __fsqrt_rn(L[j]));
        first = false;
        ++have;
      }
    }
    if (exact) tree_mean_out(sum, have + (drop ? 1 : 0), q, qidx, o);
  } else {
    bool tied = false;
#pragma unroll
    for (int j = 0; j < KCAP; ++j) {
      if (j >= pad && L[j] < INFINITY) ++have;
      if (j > pad && L[j] < INFINITY && L[j] == L[j - (j > 0)]) tied = true;
      if (drop && j == pad && L[j] == 0.0f) tied = true;  // another point in its place
    }
    // the points within the K-th distance, from the leaves scanned
    const float tau = mine ? fminf(fminf(L[KCAP - 1], bound), FLT_MAX) : -1.0f;
    for (int i = 0; i < scanned; ++i) {
      const u32 l = leaves[i];
      const float4 mate = mate_of(l);
      const float at = box_d2(own, t.box[0], t.stride[0], l) <= tau ? tau : -1.0f;
      if (!stage_leaf(l, at, mate)) continue;
      test_staged(at, drop && l == packet ? lane : -1, [&](int c, float d) {
        if (cnt < PCAP) pbuf[cnt][lane] = make_uint2(__float_as_uint(d), l * 32 + c);
        ++cnt;
      });
    }
    // exactly these are within the K-th distance, no two equal (and what is
    // missing is not there: points infinitely far would be)
    exact = mine && cnt == have && !tied &&
            (have == KL || bound < INFINITY || (u32)(have + (drop ? 1 : 0)) == t.n);
    // each to its rank among the sorted distances, behind the point itself
    const int r0 = drop ? 1 : 0;
    if (exact) {
      if (drop) {
        if constexpr (MODE == TREE_PAIRS) {
          if (o.idx) o.idx[(size_t)qidx * K] = (int32_t)qidx;
          if (o.d2) o.d2[(size_t)qidx * K] = 0.0f;
        } else {
          sorted[0][lane] = qi;
        }
      }
      for (int i = 0; i < have; ++i) {
        const uint2 b = pbuf[i][lane];
        const float d = __uint_as_float(b.x);
        int r = r0 - pad;
#pragma unroll
        for (int j = 0; j < KCAP; ++j) r += L[j] < d ? 1 : 0;
        if constexpr (MODE == TREE_PAIRS) {
          const size_t at = (size_t)qidx * K + r;
          if (o.idx) o.idx[at] = (int32_t)__float_as_uint(__ldg(&t.pts[b.y]).w);
          if (o.d2) o.d2[at] = d;
        } else {
          sorted[r][lane] = b.y;
        }
      }
    }
    have += r0;
  }
  // the others are listed for the second kernel
  const unsigned again = __ballot_sync(0xffffffffu, active && !exact);
  if (again) {
    u32 at = 0;
    if (lane == 0) at = atomicAdd(qs.hard_count, (u32)__popc(again));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (active && !exact) qs.hard[at + __popc(again & ((1u << lane) - 1))] = qi;
  }
  if (!exact) return;
  if constexpr (MODE == TREE_PAIRS) {
    for (int j = have; j < K; ++j) {
      if (o.idx) o.idx[(size_t)qidx * K + j] = -1;
      if (o.d2) o.d2[(size_t)qidx * K + j] = INFINITY;
    }
    if (o.counts) o.counts[qidx] = have;
  } else if constexpr (!MEAN) {
    tree_normal_out<MODE>([&](int j) { return __ldg(&t.pts[sorted[j][lane]]); }, have, q, qidx, o);
  }
}

// one warp per listed query, lanes over a leaf's points, a list of packed
// (distance, index) keys over the lanes
template <int P, int MODE>
__global__ __launch_bounds__(128) void k_knn_tree_hard(TreeView t, TreeQueries qs, int K,
                                                       float bound, TreeOut o) {
  __shared__ float4 near[4][32 * P];  // the neighbours in order
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const u32 n = *qs.hard_count;
  const bool self = qs.n_sort == nullptr || *qs.n_sort == 0;
  for (u32 w = blockIdx.x * 4 + wib; w < n; w += gridDim.x * 4) {
    const u32 qi = qs.hard[w];
    const float4 q = self ? t.pts[qi] : qs.q[qi];
    const u32 qidx = __float_as_uint(q.w);
    u32 start = qi / 32;
    if (!self) start = leaf_of_key(t, qs.keys[qi]);
    WarpList<P> W;
    W.init();
    u64 key_thr = ~0ull;
    u32 found = 0;
    const Box own{{q.x, q.y, q.z}, {q.x, q.y, q.z}};
    auto limit = [&]() {
      return key_thr == ~0ull ? bound : fminf(nbr_d2(key_thr), bound);
    };
    auto scan = [&](u32 l) {
      const u32 i = l * 32 + lane;
      u64 key = ~0ull;
      if (i < t.n) {
        const float4 p = __ldg(&t.pts[i]);
        const float d = dist2(p.x, p.y, p.z, q.x, q.y, q.z);
        if (d <= bound) key = pack_nbr(d, (int)__float_as_uint(p.w));
      }
      found += __popc(__ballot_sync(0xffffffffu, key != ~0ull));
      unsigned m = __ballot_sync(0xffffffffu, key < key_thr);
      if constexpr (P == 1) {
        if (__popc(m) > 4) {  // many at once: one merge instead of serial inserts
          W.merge_lanes((m >> lane) & 1u ? key : ~0ull);
          key_thr = W.get(K - 1);
          m = 0;
        }
      }
      while (m) {
        const int b = __ffs(m) - 1;
        m &= m - 1;
        const u64 k = __shfl_sync(0xffffffffu, key, b);
        if (k < key_thr) {
          W.insert(k);
          key_thr = W.get(K - 1);
        }
      }
    };
    const u32 s0 = start > 0 ? start - 1 : 0, s1 = min(start + 1, t.count[0] - 1);
    for (u32 l = s0; l <= s1; ++l) scan(l);
    auto leaf = [&](u32 l) {
      if (l < s0 || l > s1) scan(l);
    };
    tree_walk_all(t, own, limit, leaf);
    const int have = min((int)found, K);
    if constexpr (MODE == TREE_MEAN) {
      float sum = 0.0f;
      for (int j = 1; j < have; ++j) sum = fadd(sum, __fsqrt_rn(nbr_d2(W.get(j))));
      if (lane == 0) tree_mean_out(sum, have, q, qidx, o);
    } else {
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const int j = p * 32 + lane;
        if constexpr (MODE == TREE_PAIRS) {
          if (j < K) {
            const size_t at = (size_t)qidx * K + j;
            if (o.idx) o.idx[at] = j < have ? nbr_idx(W.e[p]) : -1;
            if (o.d2) o.d2[at] = j < have ? nbr_d2(W.e[p]) : INFINITY;
          }
        } else {
          if (j < have) near[wib][j] = __ldg(&t.pts[t.pos_of[nbr_idx(W.e[p])]]);
        }
      }
      if constexpr (MODE == TREE_PAIRS) {
        if (lane == 0 && o.counts) o.counts[qidx] = have;
      } else {
        __syncwarp();
        if (lane == 0)
          tree_normal_out<MODE>([&](int j) { return near[wib][j]; }, have, q, qidx, o);
        __syncwarp();
      }
    }
  }
}

template <int KCAP, int MODE>
void launch_tree(rvp_context *ctx, const TreeView &t, const TreeQueries &q, int K, float bound,
                 const TreeOut &o) {
  constexpr size_t smem = tree_smem<KCAP, MODE>();
  static_assert(smem <= 48 * 1024, "no opt-in to larger shared memory here");
  k_knn_tree<KCAP, MODE><<<(q.n + 31) / 32, 32, smem, ctx->stream>>>(t, q, K, bound, o);
  RVP_LAUNCH_CHECK(ctx);
  const unsigned blocks = grid_for(q.n, 4, ctx->num_sms * 8);
  if (K <= 32)
    k_knn_tree_hard<1, MODE><<<blocks, 128, 0, ctx->stream>>>(t, q, K, bound, o);
  else
    k_knn_tree_hard<2, MODE><<<blocks, 128, 0, ctx->stream>>>(t, q, K, bound, o);
  RVP_LAUNCH_CHECK(ctx);
}

template <int MODE>
void launch_tree_k(rvp_context *ctx, const TreeView &t, const TreeQueries &q, int K, float bound,
                   const TreeOut &o) {
  // the list leaves the point itself out where the host knows that the
  // queries are the cloud (n_sort: the device finds out)
  const int KL = q.n_sort || K == 1 ? K : K - 1;
  if (KL <= 8) launch_tree<8, MODE>(ctx, t, q, K, bound, o);
  else if (KL <= 16) launch_tree<16, MODE>(ctx, t, q, K, bound, o);
  else if (KL <= 32) launch_tree<32, MODE>(ctx, t, q, K, bound, o);
  else launch_tree<64, MODE>(ctx, t, q, K, bound, o);
}
}  // namespace

void KnnTree::release() {
  keys.release(); vals.release(); sort.release(); pts.release(); pos.release(); boxes.release();
  misc.release(); qkeys.release(); qvals.release(); qpts.release(); hard.release();
}

TreeView tree_build(rvp_context *ctx, KnnTree &w, const float *x, const float *y, const float *z,
                    size_t n) {
  w.keys.reserve(n * 8);
  w.vals.reserve(n * 4);
  w.sort.reserve(sort_temp_bytes(n));
  w.pts.reserve(n * 16);
  w.pos.reserve(n * 4);
  w.misc.reserve(256);
  TreeView t{};
  t.n = (u32)n;
  size_t total = 0;
  u32 c = (u32)((n + 31) / 32);
  for (int l = 0; l < kTreeLevels; ++l, c = (c + 31) / 32) {
    t.count[l] = c;
    t.stride[l] = (c + 31) & ~31u;
    total += (size_t)t.stride[l] * 6 * 4;
  }
  w.boxes.reserve(total);
  float *b = w.boxes.as<float>();
  for (int l = 0; l < kTreeLevels; ++l) {
    t.box[l] = b;
    b += (size_t)t.stride[l] * 6;
  }
  t.pts = w.pts.as<float4>();
  t.pos_of = w.pos.as<u32>();
  t.keys = w.keys.as<u64>();
  t.bb = w.misc.as<float>();
  cudaStream_t st = ctx->stream;
  const int sms = ctx->num_sms;
  k_tree_init<<<1, 32, 0, st>>>(w.misc.as<float>());
  RVP_LAUNCH_CHECK(ctx);
  cloud_bbox(ctx, x, y, z, n, w.misc.as<float>());
  k_tree_keys<<<grid_for(n, 256, sms * 8), 256, 0, st>>>(x, y, z, n, nullptr, t.bb,
                                                         w.keys.as<u64>(), w.vals.as<u32>());
  RVP_LAUNCH_CHECK(ctx);
  SortTemp tmp;
  sort_temp_carve(tmp, w.sort.ptr, n);
  radix_sort_pairs(ctx, w.keys.as<u64>(), w.vals.as<u32>(), n, nullptr, tmp);
  k_tree_leaves<<<(unsigned)((t.count[0] + 7) / 8), 256, 0, st>>>(
      x, y, z, w.vals.as<u32>(), t.n, w.pts.as<float4>(), w.pos.as<u32>(), t.box[0], t.stride[0]);
  RVP_LAUNCH_CHECK(ctx);
  int level = 1;
  if (t.count[1] > 32) {  // past one block's reach
    k_tree_parents<<<(t.count[1] + 7) / 8, 256, 0, st>>>(t, 1);
    RVP_LAUNCH_CHECK(ctx);
    level = 2;
  }
  k_tree_top<<<1, 1024, 0, st>>>(t, level);
  RVP_LAUNCH_CHECK(ctx);
  return t;
}

TreeQueries tree_queries_as_given(rvp_context *ctx, KnnTree &w, size_t nq) {
  TreeQueries q{};
  q.n = (u32)nq;
  w.hard.reserve(nq * 8 + 256);
  q.hard_count = w.hard.as<u32>();
  q.hard = q.hard_count + 64;
  q.longer = q.hard + nq;
  RVP_CUDA_TRY(cudaMemsetAsync(q.hard_count, 0, 4, ctx->stream));
  return q;
}

TreeQueries tree_queries(rvp_context *ctx, KnnTree &w, const TreeView &t, const float *x,
                         const float *y, const float *z, const float *qx, const float *qy,
                         const float *qz, size_t nq) {
  TreeQueries q = tree_queries_as_given(ctx, w, nq);
  if (qx == x && qy == y && qz == z && nq == t.n) return q;
  w.qkeys.reserve(nq * 8);
  w.qvals.reserve(nq * 4);
  w.qpts.reserve(nq * 16);
  w.sort.reserve(sort_temp_bytes(std::max<size_t>(nq, t.n)));
  u64 *n_sort = w.misc.as<u64>() + 4;
  cudaStream_t st = ctx->stream;
  const unsigned gb = grid_for(nq, 256, ctx->num_sms * 8);
  k_tree_count<<<1, 1, 0, st>>>(n_sort, nq == t.n ? 0 : (u64)nq);
  RVP_LAUNCH_CHECK(ctx);
  if (nq == t.n) {
    k_tree_same<<<gb, 256, 0, st>>>(qx, qy, qz, x, y, z, nq, n_sort);
    RVP_LAUNCH_CHECK(ctx);
  }
  k_tree_keys<<<gb, 256, 0, st>>>(qx, qy, qz, nq, n_sort, t.bb, w.qkeys.as<u64>(),
                                  w.qvals.as<u32>());
  RVP_LAUNCH_CHECK(ctx);
  SortTemp tmp;
  sort_temp_carve(tmp, w.sort.ptr, nq);
  radix_sort_pairs(ctx, w.qkeys.as<u64>(), w.qvals.as<u32>(), nq, n_sort, tmp);
  k_tree_queries<<<gb, 256, 0, st>>>(qx, qy, qz, w.qvals.as<u32>(), n_sort, w.qpts.as<float4>());
  RVP_LAUNCH_CHECK(ctx);
  q.q = w.qpts.as<float4>();
  q.keys = w.qkeys.as<u64>();
  q.n_sort = n_sort;
  return q;
}

void tree_knn(rvp_context *ctx, const TreeView &t, const TreeQueries &q, int k, float radius,
              int mode, const TreeOut &o) {
  // the radius search's bound: d2 <= radius * radius in float
  volatile float r = radius;
  const float bound = radius > 0.0f ? r * r : INFINITY;
  switch (mode) {
    case TREE_MEAN: launch_tree_k<TREE_MEAN>(ctx, t, q, k, bound, o); break;
    case TREE_PAIRS: launch_tree_k<TREE_PAIRS>(ctx, t, q, k, bound, o); break;
    case TREE_NORMALS: launch_tree_k<TREE_NORMALS>(ctx, t, q, k, bound, o); break;
    default: launch_tree_k<TREE_PRECISE>(ctx, t, q, k, bound, o);
  }
}

}  // namespace rvp
