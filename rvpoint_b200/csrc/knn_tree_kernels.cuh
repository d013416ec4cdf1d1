// Kernels of the box tree (knn_tree.cu, knn_tree_frames.cu): keys, boxes and
// the search for the k nearest.
#pragma once

#include <float.h>
#include <math.h>

#include "grid_device.cuh"
#include "internal.cuh"
#include "normals_device.cuh"
#include "tree_device.cuh"

namespace rvp {
using namespace gd;
using namespace td;

namespace {
// Bits of a Hilbert code at least; each digit of eight is a pass of the sort.
// Outliers stretch the box, so the cells are far finer than the leaves: 24 bits
// for 87,000 points of a room with outliers make leaves that cost its normals
// 250 us more than the pass saves (9 us).
constexpr int kTreeKeyBits = 32;
__host__ __device__ inline int tree_key_bits(size_t n) {
  return n <= 4096 ? 24 : kTreeKeyBits;
}

struct TreeFrame {  // the quantisation of the cloud's box
  float lo[3];
  float inv;    // cells per unit (a power of two)
  int bits[3];  // of each axis
};

// the bits of a code with cells of 2^k
__device__ __forceinline__ int tree_code_bits(const float (&ext)[3], int k, TreeFrame &F) {
  int sum = 0;
  for (int a = 0; a < 3; ++a) {
    const float q = ldexpf(ext[a], -k);  // cells along the axis
    F.bits[a] = q < 1.0f ? 0 : min(ilogbf(q), 126) + 1;
    sum += F.bits[a];
  }
  F.inv = ldexpf(1.0f, -k);
  return sum;
}

// the finest power-of-two cell, 2^k, whose codes fit `key_bits`; returns k
__device__ __forceinline__ int tree_frame(const float *bb, int key_bits, TreeFrame &F,
                                          float (&ext)[3]) {
  float emax = 0.0f;
  for (int a = 0; a < 3; ++a) {
    // (points infinitely far: in the last cells)
    const float lo = fmaxf(bb[a], -1e30f), hi = fminf(bb[3 + a], 1e30f);
    const float e = fsub(hi, lo);
    F.lo[a] = lo < INFINITY ? lo : 0.0f;
    ext[a] = e > 0.0f ? e : 0.0f;  // (NaN and empty axes: one cell)
    emax = fmaxf(emax, ext[a]);
  }
  int k = emax > 0.0f ? ilogbf(emax) - key_bits : -60;
  k = max(k, -100);
  for (;; ++k) {
    const int sum = tree_code_bits(ext, k, F);
    if (sum <= key_bits) return k;
    k += (sum - key_bits) / 3 > 1 ? (sum - key_bits) / 3 - 1 : 0;  // three bits go per step
  }
}
__device__ __forceinline__ void tree_frame(const float *bb, int key_bits, TreeFrame &F) {
  float ext[3];
  tree_frame(bb, key_bits, F, ext);
}

// A few of a cloud's points: the median of the distances to the nearest other
// one among them (squared; 0: none), and the median of each coordinate. By a
// block's first 128 threads (all of it calls).
constexpr int kSample = 32;
struct TreeSample {
  float nearest, median[3];
};
__device__ __forceinline__ void tree_sample(const float *x, const float *y, const float *z,
                                            size_t n, TreeSample *out) {
  __shared__ float v[4][kSample];  // nearest distances, x, y, z
  const int i = threadIdx.x / 4, part = threadIdx.x % 4;
  const bool in = i < kSample;
  if (in && part < 3)
    v[1 + part][i] = (part == 0 ? x : part == 1 ? y : z)[n * (2 * i + 1) / (2 * kSample)];
  if (threadIdx.x < 4) (&out->nearest)[threadIdx.x] = 0.0f;
  __syncthreads();
  if (!in) return;  // (whole warps)
  float best = INFINITY;  // (points in one place say nothing)
#pragma unroll
  for (int j = part; j < kSample; j += 4) {
    const float d = dist2(v[1][j], v[2][j], v[3][j], v[1][i], v[2][i], v[3][i]);
    if (d > 0.0f && d < best) best = d;
  }
  best = fminf(best, __shfl_xor_sync(0xffffffffu, best, 1));
  best = fminf(best, __shfl_xor_sync(0xffffffffu, best, 2));
  if (part == 0) v[0][i] = best;
  asm volatile("bar.sync 1, %0;" ::"n"(4 * kSample) : "memory");
  // the one in the middle of those with a value writes it
  const float mine = v[part][i];
  int rank = 0, all = 0;
#pragma unroll 8
  for (int j = 0; j < kSample; ++j) {
    const float w = v[part][j];
    const bool finite = fabsf(w) < INFINITY;
    all += finite;
    rank += finite && (w < mine || (w == mine && j < i));
  }
  if (fabsf(mine) < INFINITY && rank == all / 2) (&out->nearest)[part] = mine;
}

// The quantisation of a cloud of n points, with longer codes (each digit of
// eight bits is another pass of the sort) where the cells would else be too coarse: far
// points stretch the box, or the points are dense in a few places. The spacing
// is estimated from the sample as on a surface; cells of up to four spacings
// are fine enough. Where even 63 bits do not reach, the cells lie around the
// sample's medians and points further out share the last ones. 105,000 LiDAR
// points in any order and one at 1e6 m, all neighbours within 0.3 m: 38.7 ms
// with 32 bits, 0.26 here; 700,000 points in 20 dense clusters, k 16: 6.3 and
// 1.1 ms; clouds that 32 bits suit have the same codes as before.
constexpr int kFineBits = 63;
__device__ __forceinline__ void tree_frame_fine(size_t n, const float *bb, const TreeSample &S,
                                                int key_bits, TreeFrame &F) {
  float ext[3];
  const int k = tree_frame(bb, key_bits, F, ext);
  if (!(S.nearest > 0.0f) || n <= 1024) return;
  const float spacing = sqrtf(S.nearest * ((float)kSample / (float)n));
  const int fine = max(ilogbf(4.0f * spacing), -100);
  if (fine >= k) return;
  if (tree_code_bits(ext, fine, F) <= kFineBits) return;
  const float half = ldexpf((float)((1 << (kFineBits / 3 - 1)) - 1), fine);
  for (int a = 0; a < 3; ++a) {
    const float hi = F.lo[a] + ext[a];
    F.lo[a] = fmaxf(F.lo[a], S.median[a] - half);
    ext[a] = fminf(hi, S.median[a] + half) - F.lo[a];
  }
  tree_code_bits(ext, fine, F);
}

// (Key: u32 where 32 bits are enough)
template <class Key>
__device__ __forceinline__ Key tree_key(const TreeFrame &F, const unsigned short *table, float x,
                                        float y, float z) {
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
  // (the levels that all axes have take a table: code, next e, next d)
  const int all = min(min(F.bits[0], F.bits[1]), F.bits[2]);
  auto rotr = [](u32 v, u32 k) { return ((v >> k) | (v << (3 - k))) & 7u; };
  Key key = 0;
  u32 e = 0, d = 0;
  for (int b = top - 1; b >= all; --b) {
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
  u32 state = (d * 8 + e) * 8;
  for (int b = all - 1; b >= 0; --b) {
    const u32 l = ((q[0] >> b) & 1u) | (((q[1] >> b) & 1u) << 1) | (((q[2] >> b) & 1u) << 2);
    const u32 v = table[state + l];
    key = (key << 3) | (v & 7u);
    state = v & ~7u;
  }
  return key;
}

// the 192 entries of tree_key's table, by the first threads of a block
__device__ __forceinline__ void tree_key_table(unsigned short *table) {
  constexpr u32 kGray = 0x54672310u, kEntry = 0x56633000u, kDir = 0x01122110u;
  auto rotr = [](u32 v, u32 k) { return ((v >> k) | (v << (3 - k))) & 7u; };
  const u32 i = threadIdx.x;
  if (i >= 192) return;
  const u32 d = i >> 6, e = (i >> 3) & 7u, l = i & 7u, k = d == 2 ? 0 : d + 1;
  const u32 w = (kGray >> (4 * rotr(l ^ e, k))) & 7u;
  const u32 e2 = e ^ rotr((kEntry >> (4 * w)) & 7u, 3 - k);
  const u32 d2 = (d + ((kDir >> (4 * w)) & 7u) + 1) % 3;
  table[i] = (unsigned short)(((d2 * 8 + e2) * 8) | w);
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

// ---------------------------------------------------------------------------
// search
// ---------------------------------------------------------------------------
// The nodes a search starts from: one cloud's top level (at most 32 nodes up to
// 33.5M points), or a frame's level-1 nodes; 32 at a time.
struct Roots {
  u32 first, end;
};
template <bool FRAMES>
constexpr int tree_top() { return FRAMES ? 1 : kTreeLevels - 1; }

// The leaves nearest first, one by one, for a caller whose leaf code is too long
// to be inlined more than once (it would not fit the instruction cache).
// element l of v without an index (v stays in registers)
template <int N, class A>
__device__ __forceinline__ auto by_level(const A &v, int l) {
  auto r = v[0];
#pragma unroll
  for (int i = 1; i < N; ++i) r = i == l ? v[i] : r;
  return r;
}
template <int N, class T>
__device__ __forceinline__ void set_level(T (&v)[N], int l, T x) {
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = i == l ? x : v[i];
}

template <int TOP>
struct TreeWalk {
  static constexpr int N = TOP + 1;
  float lb[N];   // per level: the lane's child's distance
  u32 open[N];   // children left (a mask, uniform)
  u32 first[N];  // their numbers start here
  int level;     // where the walk stands
  u32 top, end;  // the next group of top nodes, and their end
  __device__ __forceinline__ void begin(const Roots &r) {
    level = N;
    top = r.first;
    end = r.end;
#pragma unroll
    for (int l = 0; l < N; ++l) {
      lb[l] = 0.0f;
      open[l] = first[l] = 0;
    }
  }
  // the next leaf within `limit` of q; false at the end
  __device__ __forceinline__ bool next(const TreeView &t, const Box &q, float limit, u32 &leaf) {
    const int lane = threadIdx.x & 31;
    while (true) {
      u32 f = top;
      int to = TOP;
      if (level == N) {
        if (top >= end) return false;
        top += 32;
      } else {
        const u32 mask = by_level<N>(open, level);
        const float v = by_level<N>(lb, level);
        // (the low bits of the distance give way to the lane)
        const u32 best = __reduce_min_sync(
            0xffffffffu,
            (mask >> lane) & 1u ? (__float_as_uint(v) & ~31u) | lane : 0xFFFFFFFFu);
        if (best == 0xFFFFFFFFu || __uint_as_float(best & ~31u) > limit) {  // none near enough
          ++level;
          continue;
        }
        const int s = best & 31;
        set_level<N>(open, level, mask & ~(1u << s));
        if (__shfl_sync(0xffffffffu, v, s) > limit) continue;
        f = by_level<N>(first, level) + s;
        if (level == 0) {
          leaf = f;
          return true;
        }
        f *= 32;
        to = level - 1;
      }
      const u32 c = f + lane, n = to == TOP ? end : by_level<N>(t.count, to);
      const float d =
          c < n ? box_d2(q, by_level<N>(t.box, to), by_level<N>(t.stride, to), c) : 0.0f;
      set_level<N>(lb, to, d);
      set_level<N>(open, to, __ballot_sync(0xffffffffu, c < n && d <= limit));
      set_level<N>(first, to, f);
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
// leaves whose hits are noted before they are collected (with lists of up to
// 16 the notes fit behind them in the buffer)
constexpr int kTreeNotes = 24;
// the buffer: distances; then the collected points and, behind them, the notes
// and after these the sorted positions (each lane in its own column)
template <int KCAP>
constexpr size_t tree_near() { return (size_t)(KCAP + kTreeExtra) * 32 * 8; }
template <int KCAP, int MODE>
constexpr size_t tree_smem() {
  constexpr size_t dist = (size_t)kTreeBuf * 32 * 4;
  constexpr bool normals = MODE == TREE_NORMALS || MODE == TREE_PRECISE;
  constexpr size_t behind = (normals && KCAP + 1 > kTreeNotes ? KCAP + 1 : kTreeNotes) * 32 * 4;
  constexpr size_t list = tree_near<KCAP>() + behind;
  return 3 * 32 * 4 + kTreeLeaves * 4 + (MODE != TREE_MEAN && list > dist ? list : dist);
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
// sqrtf(d2_j), j = 1 .. k, over k, NaN for a point without a position (its
// distances are); within a radius over those found, and the radius itself for a
// point without neighbours (:246-270), one without a position among them
__device__ __forceinline__ void tree_mean_out(float sum, int have, const float4 &q, u32 qidx,
                                              const TreeOut &o) {
  const float self = dist2(q.x, q.y, q.z, q.x, q.y, q.z);
  float m = have > 1 ? fdiv(sum, (float)(have - 1)) : 0.0f;
  if (o.radius_mode) m = have > 1 ? m : o.fallback;
  else if (!(self == 0.0f)) m = self;
  o.mean[qidx] = m;
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
  const size_t at = o.out_pos ? (size_t)o.out_pos[qidx] : (size_t)qidx;
  o.nx[at] = nx;
  o.ny[at] = ny;
  o.nz[at] = nz;
}

// The ranks by (distance, index) of the points in a lane's column, five bits
// each. (Not inlined: the search's own code is as long as it may be.)
__device__ __noinline__ ulonglong2 tie_ranks(const float4 *pts, const uint2 *near, u32 *idx,
                                             int cnt) {
  for (int i = 0; i < cnt; ++i) idx[i * 32] = __float_as_uint(__ldg(&pts[near[i * 32].y]).w);
  ulonglong2 ranks{0, 0};
#pragma unroll 1
  for (int i = 0; i < cnt; ++i) {
    const u32 d = near[i * 32].x, own = idx[i * 32];
    u64 r = 0;
    for (int j = 0; j < cnt; ++j) {
      const u32 e = near[j * 32].x;  // (distances are not negative: ordered as bits)
      r += e < d || (e == d && idx[j * 32] < own) ? 1 : 0;
    }
    if (i < 12) ranks.x |= r << (5 * i);
    else ranks.y |= r << (5 * (i - 12));
  }
  return ranks;
}

// One warp (block) per packet of 32 queries. The list holds the K nearest, or
// for the cloud's own points the K - 1 nearest others (the point itself, at
// distance 0, is the first of its row); KCAP is at least that, a power of two.
// FRAMES: a tree of many frames (tree_build_frames), whose own points, all or
// those listed, are the queries.
template <int KCAP, int MODE, bool FRAMES>
__global__ __launch_bounds__(32, KCAP > 32 ? 10 : 16) void k_knn_tree(TreeView t, TreeQueries qs,
                                                                      int K, float bound,
                                                                      TreeOut o) {
  extern __shared__ __align__(16) unsigned char tree_sm[];
  constexpr bool MEAN = MODE == TREE_MEAN;  // distances only
  constexpr int PCAP = KCAP + kTreeExtra;
  constexpr int SORTED = KCAP < 16 ? KCAP : 16;  // distances sorted at once
  float(*stage)[32] = reinterpret_cast<float(*)[32]>(tree_sm);  // x, y, z
  u32 *leaves = reinterpret_cast<u32 *>(tree_sm + 384);
  unsigned char *buf = tree_sm + 384 + kTreeLeaves * 4;
  float(*fbuf)[32] = reinterpret_cast<float(*)[32]>(buf);
  uint2(*pbuf)[32] = reinterpret_cast<uint2(*)[32]>(buf);
  u32(*notes)[32] = reinterpret_cast<u32(*)[32]>(buf + tree_near<KCAP>());
  u32(*sorted)[32] = notes;
  const int lane = threadIdx.x;
  const u32 packet = blockIdx.x + (MODE == TREE_PRECISE ? o.packet0 : 0u);
  // the cloud's own points (leaf `packet`), or 32 of the sorted queries
  const bool self = FRAMES || qs.n_sort == nullptr || *qs.n_sort == 0;
  const float4 *src = self ? t.pts : qs.q;
  u32 qi = packet * 32 + lane, start = packet;
  bool active = qi < qs.n, mine = active;  // (mine: answered with the packet)
  Roots roots{0, t.count[kTreeLevels - 1]};
  u32 leaf0 = 0, leaf1 = t.count[0] - 1;  // the leaves there are
  if constexpr (FRAMES) {
    if (qs.list) {
      const u64 n = *qs.n_list;
      if (packet * 32 >= n) return;
      active = qi < n;
      qi = qs.list[active ? qi : packet * 32];
      start = __shfl_sync(0xffffffffu, qi, 0) / 32;
    }
    const u32 frame = t.node_frame[start / 32];
    if (frame == 0xFFFFFFFFu) return;
    active = active && !(__float_as_uint(src[qi].w) & kRemovedBit);  // (or no point at all)
    if (!__any_sync(0xffffffffu, active)) return;
    mine = active && t.node_frame[qi / 1024] == frame;
    const uint2 nodes = t.frame_nodes[frame];
    roots = Roots{nodes.x, nodes.y};
    leaf0 = nodes.x * 32;
    leaf1 = nodes.y * 32 - 1;
  } else if (!self) {
    start = leaf_of_key(t, qs.keys[min(packet * 32 + 16, qs.n - 1)]);
  }
  const float4 q = src[FRAMES || active ? qi : packet * 32];
  const u32 qidx = __float_as_uint(q.w) & (FRAMES ? 0x7FFFFFFFu : 0xFFFFFFFFu);
  const Box own{{q.x, q.y, q.z}, {q.x, q.y, q.z}};
  // (a point without a position, NaN or infinite, is not at distance 0 from
  // itself, as the packet takes for granted: the second kernel answers it)
  mine = mine && dist2(q.x, q.y, q.z, q.x, q.y, q.z) == 0.0f;

  // ---- the sorted distances: slots 0 .. pad - 1 hold -1 and never move
  const bool drop = self && K > 1;  // the point itself is not in the list
  const int KL = drop ? K - 1 : K, pad = KCAP - KL;
  float L[KCAP];
#pragma unroll
  for (int j = 0; j < KCAP; ++j) L[j] = j < pad ? -1.0f : INFINITY;
  int cnt = 0;  // buffered distances
  float lim = -1.0f, pmax = -1.0f;  // what the buffer takes: d2 <= lim; its largest
  bool idle = false;                // nothing can be nearer than what it has
  auto limits = [&]() {
    lim = mine && !idle ? fminf(fminf(L[KCAP - 1], bound), FLT_MAX) : -1.0f;
    pmax = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(lim)));
  };
  limits();
  auto flush = [&]() {
    const int most = __reduce_max_sync(0xffffffffu, cnt);
    int i = 0;
    // a sorted batch merged at once; the last few one by one
    for (; i + SORTED / 4 < most; i += SORTED) {
      float S[SORTED];
#pragma unroll
      for (int j = 0; j < SORTED; ++j) S[j] = i + j < cnt ? fbuf[i + j][lane] : INFINITY;
      bitonic_sort<SORTED>(S);
#pragma unroll
      for (int j = 0; j < SORTED; ++j)
        L[KCAP - SORTED + j] = fminf(L[KCAP - SORTED + j], S[SORTED - 1 - j]);
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
  // hit(c, d2) for the staged points c within `at`
  auto test_staged = [&](float at, auto &&hit) {
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
        if (d[u] <= at) hit(c + u, d[u]);
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
    const int skip = drop && l == qi / 32 ? (int)(qi & 31) : -1;  // the point itself
    float *to = &fbuf[cnt][lane];
    // (mostly the first leaf only; larger kernels wait for instructions: 2.88 ms
    // with and 2.72 without the second loop for 2 M lists of 30; 5.68 and 5.76 ms
    // for 14.5 M lists of 16)
    if (KCAP > 16 || __any_sync(0xffffffffu, skip >= 0)) {
      test_staged(at, [&](int c, float d) {
        if (c == skip) return;
        *to = d;
        to += 32;
      });
    } else {
      test_staged(at, [&](int, float d) {
        *to = d;
        to += 32;
      });
    }
    const int now = (int)(to - &fbuf[0][lane]) >> 5;
    // (without hits now it has none later)
    if (MEAN || __any_sync(0xffffffffu, now != cnt)) leaves[scanned++] = l;
    cnt = now;
  };
  // the leaves around the packet's place first (they set the limits), then
  // the walk
  const u32 s0 = start > leaf0 ? start - 1 : leaf0, s1 = min(start + 1, leaf1);
  const int near = (int)(s1 - s0) + 1;
  Box pk{};  // the box of the packet
  TreeWalk<tree_top<FRAMES>()> walk;
  walk.begin(roots);
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
    // (one of many points in one place has its distances, all 0; for the
    // indices it is left, and its packet need not test all of them: 150,000
    // points, 3000 of them in one place, k 16 within a radius: 684 us,
    // now 207)
    if (lim == 0.0f && KL > 1) {
      if constexpr (MEAN) idle = true;
      else mine = false;
    }
    int rank = 0;
    for (int i = 0; i < 32; ++i) {
      const float other = __shfl_sync(0xffffffffu, mine ? lim : INFINITY, i);
      rank += other < lim || (other == lim && i < lane) ? 1 : 0;
    }
    const unsigned mid = __ballot_sync(0xffffffffu, mine && rank == 16);
    if (mid) {
      const float ref = __shfl_sync(0xffffffffu, lim, __ffs(mid) - 1);
      mine = mine && lim <= kLoner * ref;
    }
    limits();
    pk = warp_box(q, mine && !idle);
  }

  // ---- results of the packet
  bool exact = mine;
  int have = 0;  // distances in the list
  float sum = 0.0f;
  if constexpr (MEAN || MODE == TREE_LIST) {
    // (without a bound, a list that is not full is of a frame of few points, or
    // some are infinitely far: the second kernel tells)
    if (MEAN) exact = exact && (bound < INFINITY || L[KCAP - 1] < INFINITY);
    bool first = !drop;  // the nearest of all does not count
#pragma unroll
    for (int j = 0; j < KCAP; ++j) {
      if (j >= pad && (!o.radius_mode || L[j] < INFINITY)) {
        if (!first) sum = fadd(sum, __fsqrt_rn(L[j]));
        first = false;
        ++have;
      }
    }
    if (MEAN && exact) tree_mean_out(sum, have + (drop ? 1 : 0), q, qidx, o);
  }
  if constexpr (!MEAN) {
    have = 0;
    bool tied = false, twin = false;
#pragma unroll
    for (int j = 0; j < KCAP; ++j) {
      if (j >= pad && L[j] < INFINITY) ++have;
      if (j > pad && L[j] < INFINITY && L[j] == L[j - (j > 0)]) tied = true;
      if (drop && j == pad && L[j] == 0.0f) twin = true;  // another point in its place
    }
    // the points within the K-th distance, from the leaves scanned
    const float tau = mine ? fminf(fminf(L[KCAP - 1], bound), FLT_MAX) : -1.0f;
    // (a leaf's hits are few and uneven over the lanes: they are noted for some
    // leaves, then each lane collects its own, about as many as any other; leaf
    // by leaf this was 36% of the kernel, 14.5 M lists of 16 in 5.94 ms, now 5.68)
    for (int i0 = 0; i0 < scanned; i0 += kTreeNotes) {
      u32 some = 0;  // leaves with hits of this lane
      for (int i = 0; i < min(kTreeNotes, scanned - i0); ++i) {
        const u32 l = leaves[i0 + i];
        const float4 mate = mate_of(l);
        const float at = box_d2(own, t.box[0], t.stride[0], l) <= tau ? tau : -1.0f;
        if (!stage_leaf(l, at, mate)) continue;
        u32 m = 0;
        test_staged(at, [&](int c, float) { m |= 1u << c; });
        if (drop && l == qi / 32) m &= ~(1u << (qi & 31));
        notes[i][lane] = m;
        some |= m ? 1u << i : 0u;
      }
      u32 m = 0, p0 = 0;
      while (some | m) {
        if (m == 0) {
          const int i = __ffs(some) - 1;
          some &= some - 1;
          m = notes[i][lane];
          p0 = leaves[i0 + i] * 32;
        }
        const u32 p = p0 + __ffs(m) - 1;
        m &= m - 1;
        const float4 v = __ldg(&t.pts[p]);
        const float d = dist2(v.x, v.y, v.z, q.x, q.y, q.z);
        if (cnt < PCAP) pbuf[cnt][lane] = make_uint2(__float_as_uint(d), p);
        ++cnt;
      }
    }
    // exactly these are within the K-th distance (and what is missing is not
    // there: points infinitely far would be)
    const bool whole =
        have == KL || bound < INFINITY || (!FRAMES && (u32)(have + (drop ? 1 : 0)) == t.n);
    exact = mine && cnt == have && !tied && !twin && whole;
    const int r0 = drop ? 1 : 0;
    auto put = [&](int r, u32 p, float d) {  // the r-th neighbour
      if constexpr (MODE == TREE_PAIRS) {
        const size_t at = (size_t)qidx * K + r;
        if (o.idx) o.idx[at] = (int32_t)__float_as_uint(__ldg(&t.pts[p]).w);
        if (o.d2) o.d2[at] = d;
      } else if constexpr (MODE == TREE_LIST) {
        o.rows[(size_t)qi * K + r] = p;
      } else {
        sorted[r][lane] = p;
      }
    };
    // each to its rank among the sorted distances, behind the point itself
    if (exact) {
      if (drop) put(0, qi, 0.0f);
      for (int i = 0; i < have; ++i) {
        const uint2 b = pbuf[i][lane];
        const float d = __uint_as_float(b.x);
        int r = r0 - pad;
#pragma unroll
        for (int j = 0; j < KCAP; ++j) r += L[j] < d ? 1 : 0;
        put(r, b.y, d);
      }
    }
    // Equal distances, and points past the list at the K-th: ranked by index as
    // well. (In short lists: of 31 or 63 the comparisons take longer than the
    // second kernel. Normals of a lattice of 700,000 points, k 16: 2.1 ms on the
    // grid, 3.0 with all its queries in the second kernel, 1.2 here.)
    if constexpr (KCAP <= 16) {
      const bool ties =
          mine && !twin && whole && cnt >= have && cnt <= PCAP && (tied || cnt > have);
      if (ties) {
        static_assert(PCAP <= kTreeNotes && PCAP <= 24, "an index, and five bits of rank, each");
        const ulonglong2 ranks = tie_ranks(t.pts, &pbuf[0][lane], &notes[0][lane], cnt);
        if (drop) put(0, qi, 0.0f);  // (over the notes)
#pragma unroll 1
        for (int i = 0; i < cnt; ++i) {
          const int r = (int)((i < 12 ? ranks.x : ranks.y) >> (5 * (i < 12 ? i : i - 12))) & 31;
          const uint2 b = pbuf[i][lane];
          if (r < KL) put(r0 + r, b.y, __uint_as_float(b.x));
        }
        exact = true;
      }
    }
    have += r0;
    if (MODE == TREE_LIST && exact) tree_mean_out(sum, have, q, qidx, o);
    if constexpr (MODE == TREE_PRECISE) {  // for k_tree_precise
      u32 *row = o.rows + (size_t)blockIdx.x * K * 32 + lane;
      for (int j = 0; j < K; ++j, row += 32)
        *row = exact && j < have ? sorted[j][lane] : 0xFFFFFFFFu;
    }
  }
  // the others are listed for the second kernel
  const unsigned again = __ballot_sync(0xffffffffu, active && !exact);
  if (again) {
    u32 at = 0;
    if (lane == 0) at = atomicAdd(qs.hard_count, (u32)__popc(again));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (active && !exact) qs.hard[at + __popc(again & ((1u << lane) - 1))] = qi;
  }
  if (o.n_packets) {
    const unsigned b = __ballot_sync(0xffffffffu, exact);
    if (lane == 0) atomicAdd(o.n_packets, (u32)__popc(b));
  }
  if (!exact) return;
  if constexpr (MODE == TREE_PAIRS) {
    for (int j = have; j < K; ++j) {
      if (o.idx) o.idx[(size_t)qidx * K + j] = -1;
      if (o.d2) o.d2[(size_t)qidx * K + j] = INFINITY;
    }
    if (o.counts) o.counts[qidx] = have;
  } else if constexpr (MODE == TREE_NORMALS) {
    tree_normal_out<MODE>([&](int j) { return __ldg(&t.pts[sorted[j][lane]]); }, have, q, qidx, o);
  }
}

// ---------------------------------------------------------------------------
// one query per warp: those the packets leave (qs.hard), or few of their own
// (qs.each), in any order
// ---------------------------------------------------------------------------
// The leaves nearest first, two loaded at a time, a lane per point, a sorted
// list of packed (distance, index) keys over the lanes: equal distances need no
// care. Normals are left for the end: a warp takes up to 32 queries, keeps their
// neighbours in columns of shared memory, and then every lane has one.
// Bound by issue where there are many (about 1100 instructions per query of 16
// within a few leaves, 65% of the issue slots), by the chain of one query, four
// levels of boxes and then leaves, where there are few: 700 queries among
// 150,000 LiDAR points, k 16, 45 us of a call, as packets 203. Keys collected in
// shared memory and ranked all at once, or merged 16 at a time, took up to twice
// the time of this (normals of a 700,000-point lattice 5.4 and 3.8 ms, 3.1 here;
// 4.0 with a lane of the warp making each normal).
constexpr int EK_WARPS = 4;
constexpr int EK_MERGE = 8;  // keys of a leaf that are merged at once
template <int MODE>
constexpr size_t each_smem(int K) {
  constexpr bool normals = MODE == TREE_NORMALS || MODE == TREE_PRECISE;
  return normals ? (size_t)EK_WARPS * K * 128 : 0;
}

// Visits the leaves within limit() of the box q, nearest child first: leaf(l, p)
// with the lane's point of a leaf, from load(l).
template <int LV, class Limit, class Load, class Leaf>
__device__ __forceinline__ void each_walk(const TreeView &t, const Box &q, u32 first, u32 end,
                                          Limit &limit, Load &load, Leaf &leaf) {
  const int lane = threadIdx.x & 31;
  const u32 c = first + lane;
  const float lb = c < end ? box_d2(q, t.box[LV], t.stride[LV], c) : 0.0f;
  bool open = c < end && lb <= limit();
  // the nearest open child, no longer open; -1: none (near enough)
  auto nearest = [&]() {
    // (the low bits of the distance give way to the lane)
    const u32 best = __reduce_min_sync(
        0xffffffffu, open ? (__float_as_uint(lb) & ~31u) | lane : 0xFFFFFFFFu);
    if (best == 0xFFFFFFFFu || __uint_as_float(best & ~31u) > limit()) return -1;
    if (lane == (int)(best & 31)) open = false;
    return (int)(best & 31);
  };
  auto near = [&](int s) { return __shfl_sync(0xffffffffu, lb, s) <= limit(); };
  while (true) {
    const int s = nearest();
    if (s < 0) break;
    if constexpr (LV > 0) {
      if (near(s))
        each_walk<LV - 1>(t, q, (first + s) * 32, t.count[LV - 1], limit, load, leaf);
    } else {
      const int s2 = nearest();
      const float4 p = load(first + s);
      const float4 p2 = s2 >= 0 ? load(first + s2) : p;
      if (near(s)) leaf(first + s, p);
      if (s2 < 0) break;
      if (near(s2)) leaf(first + s2, p2);
    }
  }
}

template <int P, int MODE, bool FRAMES>
__global__ __launch_bounds__(EK_WARPS * 32, 6) void k_knn_tree_each(TreeView t, TreeQueries qs,
                                                                    int K, float bound,
                                                                    TreeOut o) {
  extern __shared__ __align__(16) unsigned char tree_sm[];
  constexpr bool NORMALS = MODE == TREE_NORMALS || MODE == TREE_PRECISE;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  u32(*columns)[32] = reinterpret_cast<u32(*)[32]>(tree_sm) + wib * K;
  const bool each = qs.each[0] != nullptr;
  const u32 n = each ? qs.n : *qs.hard_count, warps = gridDim.x * EK_WARPS;
  const bool self = FRAMES || qs.n_sort == nullptr || *qs.n_sort == 0;
  auto query = [&](u32 w) {
    if (each) return make_float4(qs.each[0][w], qs.each[1][w], qs.each[2][w], __uint_as_float(w));
    return self ? t.pts[qs.hard[w]] : qs.q[qs.hard[w]];
  };
  auto index_of = [](const float4 &q) {
    return __float_as_uint(q.w) & (FRAMES ? 0x7FFFFFFFu : 0xFFFFFFFFu);
  };
  const u32 chunk = NORMALS ? min(32u, (n + warps - 1) / warps) : 1u;  // queries per turn
  for (u32 w0 = (blockIdx.x * EK_WARPS + wib) * chunk; w0 < n; w0 += warps * chunk) {
    const u32 m = min(chunk, n - w0);
    int mine = 0;  // the lane's query's neighbours
    for (u32 c = 0; c < m; ++c) {
      const float4 q = query(w0 + c);
      const u32 qidx = index_of(q);
      Roots roots{0, t.count[kTreeLevels - 1]};
      u32 s0 = 1, s1 = 0;  // leaves tested before the walk: around the cloud's own point
      if constexpr (FRAMES) {
        const u32 qi = qs.hard[w0 + c];
        const uint2 nodes = t.frame_nodes[t.node_frame[qi / 1024]];
        roots = Roots{nodes.x, nodes.y};
        s0 = max(qi / 32, nodes.x * 32 + 1) - 1;
        s1 = min(qi / 32 + 1, nodes.y * 32 - 1);
      } else if (!each && self) {
        const u32 leaf = qs.hard[w0 + c] / 32;
        s0 = max(leaf, 1u) - 1;
        s1 = min(leaf + 1, t.count[0] - 1);
      }
      WarpList<P> W;
      W.init();
      u32 found = 0;
      u64 thr = ~0ull;  // the K-th key, once there are K
      auto limit = [&]() { return thr == ~0ull ? bound : fminf(nbr_d2(thr), bound); };
      auto load = [&](u32 l) {
        const u32 i = l * 32 + lane;
        return i < t.n ? __ldg(&t.pts[i]) : make_float4(NAN, NAN, NAN, 0.0f);
      };
      auto take = [&](const float4 &p) {
        const float d = dist2(p.x, p.y, p.z, q.x, q.y, q.z);
        const u64 key = d <= bound ? pack_nbr(d, (int)__float_as_uint(p.w)) : ~0ull;
        unsigned m = __ballot_sync(0xffffffffu, key < thr);
        found += __popc(m);  // (more than there are, past the K-th)
        if constexpr (P == 1) {
          if (__popc(m) > EK_MERGE) {  // many at once: one merge instead of serial inserts
            W.merge_lanes((m >> lane) & 1u ? key : ~0ull);
            thr = W.get(K - 1);
            m = 0;
          }
        }
        while (m) {
          const int b = __ffs(m) - 1;
          m &= m - 1;
          const u64 k = __shfl_sync(0xffffffffu, key, b);
          if (k < thr) {
            W.insert(k);
            thr = W.get(K - 1);
          }
        }
      };
      // (a query with a NaN is near nothing)
      if (!(isnan(q.x) || isnan(q.y) || isnan(q.z))) {
        const Box own{{q.x, q.y, q.z}, {q.x, q.y, q.z}};
        if (s0 <= s1) {
          const float4 a = load(s0), b = load(min(s0 + 1, s1)), e = load(s1);
          take(a);
          if (s0 + 1 <= s1) take(b);
          if (s0 + 2 <= s1) take(e);
        }
        auto leaf = [&](u32 l, const float4 &p) {
          if (l < s0 || l > s1) take(p);
        };
        for (u32 f = roots.first; f < roots.end; f += 32)
          each_walk<tree_top<FRAMES>()>(t, own, f, roots.end, limit, load, leaf);
      }
      const int have = min((int)found, K);
      if (o.n_hard && lane == 0) atomicAdd(o.n_hard, 1u);
      if constexpr (MODE == TREE_MEAN || MODE == TREE_LIST) {
        float sum = 0.0f;
#pragma unroll
        for (int p = 0; p < P; ++p) {
          const float r = __fsqrt_rn(nbr_d2(W.e[p]));
          for (int j = p == 0 ? 1 : 0; j < min(32, have - p * 32); ++j)
            sum = fadd(sum, __shfl_sync(0xffffffffu, r, j));
        }
        if (lane == 0) tree_mean_out(sum, have, q, qidx, o);
      }
      if constexpr (MODE != TREE_MEAN) {
#pragma unroll
        for (int p = 0; p < P; ++p) {
          const int j = p * 32 + lane;
          if (j >= K) continue;
          if constexpr (MODE == TREE_PAIRS) {
            const size_t at = (size_t)qidx * K + j;
            if (o.idx) o.idx[at] = j < have ? nbr_idx(W.e[p]) : -1;
            if (o.d2) o.d2[at] = j < have ? nbr_d2(W.e[p]) : INFINITY;
          } else {
            const u32 at =
                j < have ? t.pos_of[(u32)nbr_idx(W.e[p]) & 0x7FFFFFFFu] : 0xFFFFFFFFu;
            if constexpr (NORMALS) columns[j][c] = at;
            else o.rows[(size_t)qs.hard[w0 + c] * K + j] = at;
          }
        }
        if (MODE == TREE_PAIRS && lane == 0 && o.counts) o.counts[qidx] = have;
        if (lane == (int)c) mine = have;
      }
    }
    if constexpr (NORMALS) {
      __syncwarp();
      if (lane < (int)m) {
        const float4 q = query(w0 + lane);
        tree_normal_out<MODE>([&](int j) { return __ldg(&t.pts[columns[j][lane]]); }, mine, q,
                              index_of(q), o);
      }
      __syncwarp();
    }
  }
}

// Normals in high precision from the rows of positions that a search left, a
// thread per query. Bound by the latency of the gather (rows, then points) and
// of the sums. Inside the search, at 14 warps per SM and among code that the
// instruction cache does not hold, this took 650 us for 2 M points of 30
// neighbours; here, with the rows (248 MB), 326.
constexpr int TP_TH = 128;
__global__ __launch_bounds__(TP_TH, 6) void k_tree_precise(TreeView t, int K, u32 packets,
                                                           TreeOut o) {
  const u32 g = blockIdx.x * TP_TH + threadIdx.x, packet = g / 32, lane = g & 31;
  const u32 qi = o.packet0 * 32 + g;
  if (packet >= packets || qi >= t.n) return;
  const u32 *row = o.rows + (size_t)packet * K * 32 + lane;
  int have = 0;
#pragma unroll 8
  for (int j = 0; j < K; ++j) have += row[(size_t)j * 32] != 0xFFFFFFFFu;
  if (have == 0) return;  // left for the second search
  const float4 q = __ldg(&t.pts[qi]);
  tree_normal_out<TREE_PRECISE>(
      [&](int j) { return __ldg(&t.pts[row[(size_t)j * 32]]); }, have, q, __float_as_uint(q.w), o);
}

// queries: how many there can be
template <int MODE, bool FRAMES>
void launch_tree_each(rvp_context *ctx, const TreeView &t, const TreeQueries &q, size_t queries,
                      int K, float bound, const TreeOut &o) {
  static_assert(each_smem<MODE>(64) <= 48 * 1024, "no opt-in to larger shared memory here");
  const unsigned blocks = grid_for(queries, EK_WARPS, ctx->num_sms * 8);
  const size_t smem = each_smem<MODE>(K);
  if (K <= 32)
    k_knn_tree_each<1, MODE, FRAMES><<<blocks, EK_WARPS * 32, smem, ctx->stream>>>(t, q, K, bound,
                                                                                  o);
  else
    k_knn_tree_each<2, MODE, FRAMES><<<blocks, EK_WARPS * 32, smem, ctx->stream>>>(t, q, K, bound,
                                                                                  o);
  RVP_LAUNCH_CHECK(ctx);
}

// packets: how many there can be
template <int KCAP, int MODE, bool FRAMES>
void launch_tree(rvp_context *ctx, const TreeView &t, const TreeQueries &q, u32 packets, int K,
                 float bound, const TreeOut &o) {
  constexpr size_t smem = tree_smem<KCAP, MODE>();
  static_assert(smem <= 48 * 1024, "no opt-in to larger shared memory here");
  if constexpr (MODE == TREE_PRECISE) {
    const u32 most = tree_precise_packets(packets, K);  // as many as have rows
    TreeOut part = o;
    for (u32 p0 = 0; p0 < packets; p0 += most) {
      const u32 n = std::min(most, packets - p0);
      part.packet0 = p0;
      k_knn_tree<KCAP, MODE, FRAMES><<<n, 32, smem, ctx->stream>>>(t, q, K, bound, part);
      RVP_LAUNCH_CHECK(ctx);
      k_tree_precise<<<(n + 3) / 4, TP_TH, 0, ctx->stream>>>(t, K, n, part);
      RVP_LAUNCH_CHECK(ctx);
    }
  } else {
    k_knn_tree<KCAP, MODE, FRAMES><<<packets, 32, smem, ctx->stream>>>(t, q, K, bound, o);
    RVP_LAUNCH_CHECK(ctx);
  }
  launch_tree_each<MODE, FRAMES>(ctx, t, q, packets * 32, K, bound, o);
}

// listed: distances a list needs room for
template <int MODE, bool FRAMES>
void launch_tree_k(rvp_context *ctx, const TreeView &t, const TreeQueries &q, u32 packets, int K,
                   int listed, float bound, const TreeOut &o) {
  if (listed <= 8) launch_tree<8, MODE, FRAMES>(ctx, t, q, packets, K, bound, o);
  else if (listed <= 16) launch_tree<16, MODE, FRAMES>(ctx, t, q, packets, K, bound, o);
  else if (listed <= 32) launch_tree<32, MODE, FRAMES>(ctx, t, q, packets, K, bound, o);
  else launch_tree<64, MODE, FRAMES>(ctx, t, q, packets, K, bound, o);
}
}  // namespace
}  // namespace rvp
