// Radius search and radius normals of one cloud over its box tree
// (knn_tree.cu), for a hash without collisions: the reference's window of
// cells then holds every point with d2 <= radius * radius exactly once
// (spatial_hashing.cpp:110-158), so the cells themselves are not needed.
//
//   count   queries in their own order, one per warp, up to kFewQueries; more
//           by packets of 32 neighbouring ones, a query per lane
//   fill    one warp per query collects its list in shared memory, orders it
//           by (d2, index) and writes it out once, coalesced. The order comes
//           from bins: d2 scaled to as many bins as the list is long, a scan,
//           and a rank among the few of the same bin. (A bitonic sort of the
//           same lists in shared memory took 1855 us of the 2650 us that all
//           neighbours within 0.5 m of 105k LiDAR points, 20M pairs, cost.)
//   normals one warp per packet, the lists (10 to 30 points usually) in a
//           column of shared memory per lane, ordered there by rank; points
//           with longer ones go one per warp
#include <math.h>

#include <algorithm>

#include "internal.cuh"
#include "normals_device.cuh"
#include "tree_device.cuh"

namespace rvp {
using namespace td;

namespace {
constexpr int FT_WARPS = 4;
constexpr u32 FT_SHORT = 256, FT_CAP = 1024;  // pairs a warp orders in shared memory
constexpr u32 FT_BINS = 512;
// (nothing to sort or to compare with the cloud, and more warps to hide each
// other's latency: 20,000 queries among 150,000 LiDAR points within 0.3 m 140
// us, as packets 232, 75,000 193 and 262; where the queries are the cloud
// 50,000 155 and 191, 105,000 220 and 245, 300,000 460 and 432; rooms, planes
// and dense clusters cross there as well)
constexpr size_t kFewQueries = 65536;

// ---------------------------------------------------------------------------
// Can two cells of the grid have one key ix + iy * p1 + iz * p2
// (spatial_hashing.h:43-45)? Only if dx + dy * p1 + dz * p2 = 0 for some
// difference of cells, and with |p1| at least the cells along x each dz leaves
// two candidates for dy. *flag is 1 when there is one, else 0, or when this does not
// settle it (tiny or huge primes, huge grids): the caller then builds the
// reference's grid and looks at the cells that are occupied.
// ---------------------------------------------------------------------------
__global__ __launch_bounds__(1024) void k_hash_check(const float *bb, float cell, long long p1,
                                                     long long p2, int *flag) {
  // the grid's dimensions (spatial_hashing.cpp:86-95), a cell to spare
  long long g[3];
  bool sure = true;
  for (int a = 0; a < 3; ++a) {
    const float eps = fmul(cell, 0.01f);
    const float d = ceilf(fdiv(fsub(fadd(bb[3 + a], eps), fsub(bb[a], eps)), cell));
    sure = sure && d >= 0.0f && d < 1.0e6f;
    g[a] = sure ? (long long)d + 2 : 0;
  }
  const long long a1 = p1 < 0 ? -p1 : p1, a2 = p2 < 0 ? -p2 : p2, most = 1ll << 40;
  sure = sure && a1 < most && a2 < most && a1 >= g[0] && a1 > 0;
  bool hit = !sure;
  for (long long dz = 1 + threadIdx.x; sure && dz < g[2]; dz += blockDim.x) {
    const long long v = dz * p2;  // below 2^60
    const long long dy = -v / p1;
    for (long long y = dy - 1; y <= dy + 1; ++y) {
      const long long s = y * p1 + v;
      if (y < g[1] && -y < g[1] && s < g[0] && -s < g[0]) hit = true;
    }
  }
  const int any = __syncthreads_or(hit);
  if (threadIdx.x == 0) *flag = any ? 1 : 0;
}

// ---------------------------------------------------------------------------
// count
// ---------------------------------------------------------------------------
// leaves a packet tests before its queries go one per warp: of 3277 packets of
// a LiDAR frame a few have every leaf of a wide box to test, and the kernel
// waited for them (468 us; 256 leaves: 140 us and 8 us for the listed ones)
constexpr int kLeafBudget = 128;

__global__ __launch_bounds__(32) void k_radius_packets(TreeView t, TreeQueries qs, float r2,
                                                       u32 *counts, u32 *most) {
  __shared__ __align__(16) float stage[3][32];
  const int lane = threadIdx.x;
  const u32 packet = blockIdx.x;
  const bool self = qs.n_sort == nullptr || *qs.n_sort == 0;
  const float4 *src = self ? t.pts : qs.q;
  const u32 qi = packet * 32 + lane;
  const bool active = qi < qs.n;
  const float4 q = src[active ? qi : packet * 32];
  const Box own{{q.x, q.y, q.z}, {q.x, q.y, q.z}};
  const Box pk = warp_box(q, true);
  const u64 nqx = pack2(-q.x, -q.x), nqy = pack2(-q.y, -q.y), nqz = pack2(-q.z, -q.z);
  u32 cnt = 0;
  int budget = kLeafBudget;
  auto leaf = [&](u32 l) {
    if (--budget < 0) return;
    const u32 i = l * 32 + lane;
    const float4 mate = i < t.n ? __ldg(&t.pts[i]) : make_float4(NAN, NAN, NAN, 0.0f);
    const float at = box_d2(own, t.box[0], t.stride[0], l) <= r2 ? r2 : -1.0f;
    if (!__any_sync(0xffffffffu, at >= 0.0f)) return;
    __syncwarp();
    stage[0][lane] = mate.x;
    stage[1][lane] = mate.y;
    stage[2][lane] = mate.z;
    __syncwarp();
#pragma unroll 2
    for (int c = 0; c < 32; c += 4) {
      const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(&stage[0][c]);
      const ulonglong2 y = *reinterpret_cast<const ulonglong2 *>(&stage[1][c]);
      const ulonglong2 z = *reinterpret_cast<const ulonglong2 *>(&stage[2][c]);
      const u64 a = dist2x2(x.x, y.x, z.x, nqx, nqy, nqz, qs.minus_zero);
      const u64 b = dist2x2(x.y, y.y, z.y, nqx, nqy, nqz, qs.minus_zero);
      cnt += half2f(a, 0) <= at;
      cnt += half2f(a, 1) <= at;
      cnt += half2f(b, 0) <= at;
      cnt += half2f(b, 1) <= at;
    }
  };
  tree_visit_all(t, pk, r2, leaf);
  if (budget < 0) {  // points far apart: one warp each (k_radius_listed)
    u32 at = 0;
    if (lane == 0) at = atomicAdd(qs.hard_count, min(32u, qs.n - packet * 32));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (active) qs.hard[at + lane] = qi;
    return;
  }
  if (active) counts[__float_as_uint(q.w)] = cnt;
  const unsigned b = __ballot_sync(0xffffffffu, active && cnt > FT_SHORT);
  if (b) {  // listed for k_radius_fill_long
    const u32 m = __reduce_max_sync(0xffffffffu, active ? cnt : 0u);
    u32 at = 0;
    if (lane == 0) {
      atomicMax(&most[0], m);
      at = atomicAdd(&most[1], (u32)__popc(b));
    }
    at = __shfl_sync(0xffffffffu, at, 0);
    if ((b >> lane) & 1u) qs.longer[at + __popc(b & ((1u << lane) - 1))] = qi;
  }
}

// hit(pass, d, index): the lane's point of a leaf. Two leaves' points are
// loaded at a time. Every SPLIT-th leaf of a node, from `part` on.
template <int SPLIT, class Hit>
__device__ __forceinline__ void radius_walk(const TreeView &t, float qx, float qy, float qz,
                                            float r2, int part, Hit &&hit) {
  const int lane = threadIdx.x & 31;
  const Box own{{qx, qy, qz}, {qx, qy, qz}};
  auto load = [&](u32 l) {
    const u32 i = l * 32 + lane;
    return i < t.n ? __ldg(&t.pts[i]) : make_float4(NAN, NAN, NAN, 0.0f);
  };
  auto take = [&](const float4 &p) {
    const float d = dist2(p.x, p.y, p.z, qx, qy, qz);
    hit(d <= r2, d, __float_as_uint(p.w));
  };
  auto parent = [&](u32 node) {  // the leaves of a level-1 node
    const u32 first = node * 32, c = first + lane;
    unsigned m = __ballot_sync(
        0xffffffffu, c < t.count[0] && box_d2(own, t.box[0], t.stride[0], c) <= r2);
    if (SPLIT > 1) {  // this part's leaves: by their rank among those near
      const unsigned mine = __ballot_sync(
          0xffffffffu, __popc(m & ((1u << lane) - 1)) % SPLIT == part);
      m &= mine;
    }
    while (m) {
      const int s = __ffs(m) - 1;
      m &= m - 1;
      const float4 p = load(first + s);
      if (m) {
        const int s2 = __ffs(m) - 1;
        m &= m - 1;
        const float4 p2 = load(first + s2);
        take(p);
        take(p2);
      } else {
        take(p);
      }
    }
  };
  tree_visit_all<1>(t, own, r2, parent);
}

// queries in their own order, one per warp
__global__ __launch_bounds__(128) void k_radius_each(TreeView t, const float *qx, const float *qy,
                                                     const float *qz, u32 nq, float r2,
                                                     u32 *counts, u32 *most, u32 *longer) {
  const u32 w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= nq) return;
  u32 cnt = 0;
  radius_walk<1>(t, qx[w], qy[w], qz[w], r2, 0, [&](bool pass, float, u32) {
    cnt += __popc(__ballot_sync(0xffffffffu, pass));
  });
  if ((threadIdx.x & 31) == 0) {
    counts[w] = cnt;
    if (cnt > FT_SHORT) {
      atomicMax(&most[0], cnt);
      longer[atomicAdd(&most[1], 1u)] = w;
    }
  }
}

// the queries packets gave up on
__global__ __launch_bounds__(128) void k_radius_listed(TreeView t, TreeQueries qs, float r2,
                                                       u32 *counts, u32 *most) {
  const u32 n = *qs.hard_count;
  const bool self = qs.n_sort == nullptr || *qs.n_sort == 0;
  for (u32 w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n;
       w += (gridDim.x * blockDim.x) >> 5) {
    const float4 q = self ? t.pts[qs.hard[w]] : qs.q[qs.hard[w]];
    u32 cnt = 0;
    radius_walk<1>(t, q.x, q.y, q.z, r2, 0, [&](bool pass, float, u32) {
      cnt += __popc(__ballot_sync(0xffffffffu, pass));
    });
    if ((threadIdx.x & 31) == 0) {
      counts[__float_as_uint(q.w)] = cnt;
      if (cnt > FT_SHORT) {
        atomicMax(&most[0], cnt);
        qs.longer[atomicAdd(&most[1], 1u)] = qs.hard[w];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// fill
// ---------------------------------------------------------------------------
__device__ __forceinline__ u32 bin_of(u64 key, float scale, u32 bins) {
  const float b = fmul(nbr_d2(key), scale);  // monotone in d2
  return b < (float)(bins - 1) ? (u32)b : bins - 1;
}

// The cnt keys of `keys` ordered: write(rank, key), by the TH threads of a warp
// or a block. Bin b lies at bin_at(b): the run of bins that a thread scans is
// then free of bank conflicts.
template <u32 TH, u32 BINS, class Write>
__device__ __forceinline__ void order_keys(const u64 *keys, u32 cnt, float r2, u32 *bins,
                                           unsigned short *perm, u32 *warp_sum, Write &&write) {
  const u32 tid = threadIdx.x & (TH - 1), lane = threadIdx.x & 31;
  auto sync = [] {
    if constexpr (TH == 32) __syncwarp();
    else __syncthreads();
  };
  if (cnt <= 32) {
    if (tid < cnt) {
      const u64 k = keys[tid];
      u32 rank = 0;
      for (u32 j = 0; j < cnt; ++j) rank += keys[j] < k;
      write(rank, k);
    }
    return;
  }
  u32 nb = 2 * TH, per_log = 1;  // bins, bins per thread
  while (nb < cnt && nb < BINS) {
    nb <<= 1;
    ++per_log;
  }
  const u32 per = 1u << per_log;
  auto bin_at = [&](u32 b) { return (b & (per - 1)) * TH + (b >> per_log); };
  const float scale = r2 > 0.0f ? fdiv((float)nb, r2) : 0.0f;
  for (u32 i = tid; i < nb; i += TH) bins[i] = 0;
  sync();
  for (u32 i = tid; i < cnt; i += TH) atomicAdd(&bins[bin_at(bin_of(keys[i], scale, nb))], 1u);
  sync();
  {  // exclusive scan of the bins
    u32 sum = 0;
    for (u32 j = 0; j < per; ++j) sum += bins[j * TH + tid];
    u32 incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (u32)o) incl += v;
    }
    u32 run = incl - sum;
    if constexpr (TH > 32) {
      if (lane == 31) warp_sum[tid >> 5] = incl;
      sync();
      for (u32 w = 0; w < tid >> 5; ++w) run += warp_sum[w];
    }
    for (u32 j = 0; j < per; ++j) {
      const u32 c = bins[j * TH + tid];
      bins[j * TH + tid] = run;
      run += c;
    }
  }
  sync();
  for (u32 i = tid; i < cnt; i += TH) {
    const u32 at = atomicAdd(&bins[bin_at(bin_of(keys[i], scale, nb))], 1u);
    perm[at] = (unsigned short)i;
  }
  sync();  // a bin now holds its end
  for (u32 p = tid; p < cnt; p += TH) {
    const u64 k = keys[perm[p]];
    const u32 b = bin_of(k, scale, nb);
    const u32 s = b ? bins[bin_at(b - 1)] : 0, e = bins[bin_at(b)];
    u32 rank = s;
    if (e - s > 1)
      for (u32 j = s; j < e; ++j) rank += keys[perm[j]] < k;
    write(rank, k);
  }
}

// Query w: the w-th in tree order (or of the sorted queries), or with qx the
// w-th in its own order. cut > 0: only the first cut of a list are written.
__device__ __forceinline__ float4 fill_query(const TreeView &t, const TreeQueries &qs,
                                             const float *qx, const float *qy, const float *qz,
                                             u32 w) {
  if (qx) return make_float4(qx[w], qy[w], qz[w], __uint_as_float(w));
  const bool self = qs.n_sort == nullptr || *qs.n_sort == 0;
  return self ? t.pts[w] : qs.q[w];
}

// one pair of a list; an output that is not wanted is null
__device__ __forceinline__ void pair_out(u64 key, u64 at, int32_t *idx, float *d2) {
  if (idx) idx[at] = nbr_idx(key);
  if (d2) d2[at] = nbr_d2(key);
}

// lists of up to FT_SHORT points, one warp each
__global__ __launch_bounds__(FT_WARPS * 32) void k_radius_fill(
    TreeView t, TreeQueries qs, const float *qx, const float *qy, const float *qz, float r2,
    const u64 *full, const u64 *offsets, u32 cut, int32_t *out_idx, float *out_d2) {
  __shared__ u64 s_keys[FT_WARPS][FT_SHORT];
  __shared__ u32 s_bins[FT_WARPS][FT_SHORT];
  __shared__ unsigned short s_perm[FT_WARPS][FT_SHORT];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const u32 w = blockIdx.x * FT_WARPS + wib;
  if (w >= qs.n) return;
  const float4 q = fill_query(t, qs, qx, qy, qz, w);
  const u32 qi = __float_as_uint(q.w);
  const u64 from = full[qi];
  const u32 cnt = (u32)(full[qi + 1] - from);
  if (cnt == 0 || cnt > FT_SHORT) return;
  u32 pos = 0;
  radius_walk<1>(t, q.x, q.y, q.z, r2, 0, [&](bool pass, float d, u32 idx) {
    const unsigned b = __ballot_sync(0xffffffffu, pass);
    const u32 at = pos + __popc(b & ((1u << lane) - 1));
    if (pass && at < cnt) s_keys[wib][at] = pack_nbr(d, (int)idx);
    pos += __popc(b);
  });
  __syncwarp();
  const u64 off = offsets[qi];
  order_keys<32, FT_SHORT>(s_keys[wib], cnt, r2, s_bins[wib], s_perm[wib], nullptr,
                           [&](u32 rank, u64 k) {
                             if (cut && rank >= cut) return;
                             pair_out(k, off + rank, out_idx, out_d2);
                           });
}

// The queries with longer lists, one block each: its warps take turns at the
// leaves and order the list together. (One warp per list, with shared memory
// for 1024 pairs each, left 16 warps to an SM: 394 us for the 15M pairs of a
// LiDAR frame's lists over 256 points.) Lists over FT_CAP go unordered to
// big_pairs and are listed in big.
__global__ __launch_bounds__(FT_WARPS * 32) void k_radius_fill_long(
    TreeView t, TreeQueries qs, const float *qx, const float *qy, const float *qz, float r2,
    const u64 *full, const u64 *offsets, u32 cut, int32_t *out_idx, float *out_d2, u64 *big_pairs,
    u32 *big, u32 *big_count) {
  __shared__ u64 s_keys[FT_CAP];
  __shared__ u32 s_bins[FT_BINS];
  __shared__ unsigned short s_perm[FT_CAP];
  __shared__ u32 s_pos, s_warp[FT_WARPS];
  const int lane = threadIdx.x & 31;
  const float4 q = fill_query(t, qs, qx, qy, qz, qs.longer[blockIdx.x]);
  const u32 qi = __float_as_uint(q.w);
  const u64 from = full[qi];
  const u32 cnt = (u32)(full[qi + 1] - from);
  const bool small = cnt <= FT_CAP;
  u64 *to = small ? s_keys : big_pairs + from;
  if (threadIdx.x == 0) s_pos = 0;
  __syncthreads();
  radius_walk<FT_WARPS>(t, q.x, q.y, q.z, r2, threadIdx.x >> 5, [&](bool pass, float d, u32 idx) {
    const unsigned b = __ballot_sync(0xffffffffu, pass);
    if (!b) return;
    u32 at = 0;
    if (lane == 0) at = atomicAdd(&s_pos, (u32)__popc(b));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(b & ((1u << lane) - 1));
    if (pass && at < cnt) to[at] = pack_nbr(d, (int)idx);
  });
  __syncthreads();
  if (!small) {
    if (threadIdx.x == 0) big[atomicAdd(big_count, 1u)] = qi;
    return;
  }
  const u64 off = offsets[qi];
  order_keys<FT_WARPS * 32, FT_BINS>(s_keys, cnt, r2, s_bins, s_perm, s_warp,
                                     [&](u32 rank, u64 k) {
                                       if (cut && rank >= cut) return;
                                       pair_out(k, off + rank, out_idx, out_d2);
                                     });
}

// the listed long lists, ordered in place in `pairs`
__global__ void k_radius_big_out(const u64 *pairs, const u32 *big, const u32 *big_count,
                                 const u64 *full, const u64 *offsets, u32 cut, int32_t *out_idx,
                                 float *out_d2) {
  for (u32 b = blockIdx.x; b < *big_count; b += gridDim.x) {
    const u32 qi = big[b];
    const u64 from = full[qi], off = offsets[qi];
    u64 cnt = full[qi + 1] - from;
    if (cut && cnt > cut) cnt = cut;
    for (u64 i = threadIdx.x; i < cnt; i += blockDim.x)
      pair_out(pairs[from + i], off + i, out_idx, out_d2);
  }
}

// ---------------------------------------------------------------------------
// normals
// ---------------------------------------------------------------------------
// A packet of 32 queries per warp, each lane with its own neighbours; points
// with more than a lane holds, and packets of points far apart (past
// kLeafBudget leaves; one such packet kept the kernel busy for 421 us where the
// others take 119), go one per warp. Bound by issue, and with many long lists
// by the listed points. 87,477 points of a room, radius 0.03 (10 neighbours
// each): 119 us and 18 for the listed ones; 100,000 and 0.05 (30 each, 28% with
// more than 48): 161 and 100.
constexpr int RN_CAP = 48;  // neighbours a lane holds
// Up to so many points are all taken one per warp: packets of few points have
// nothing to hide their latency (5000 points of a LiDAR frame 88 us, with packets
// 114; 20,000 119 and 152, of a room 166 and 234; 40,000 156 and 162, 80,000 238
// and 219).
constexpr u32 kFewNormals = 32768;

__global__ __launch_bounds__(32) void k_radius_normals(TreeView t, u64 minus_zero, float r2,
                                                       int iters, float vpx, float vpy, float vpz,
                                                       float *nx, float *ny, float *nz, u32 *hard,
                                                       u32 *hard_count) {
  __shared__ __align__(16) float stage[3][32];
  __shared__ uint2 near[RN_CAP][32];           // distance, tree position
  __shared__ unsigned char order[RN_CAP][32];  // row of each rank
  const int lane = threadIdx.x;
  const u32 qi = blockIdx.x * 32 + lane;
  const bool active = qi < t.n;
  const float4 q = t.pts[active ? qi : blockIdx.x * 32];
  const Box own{{q.x, q.y, q.z}, {q.x, q.y, q.z}};
  const Box pk = warp_box(q, true);
  const u64 nqx = pack2(-q.x, -q.x), nqy = pack2(-q.y, -q.y), nqz = pack2(-q.z, -q.z);
  int cnt = 0, budget = kLeafBudget;
  auto leaf = [&](u32 l) {
    if (--budget < 0) return;
    const u32 i = l * 32 + lane;
    const float4 mate = i < t.n ? __ldg(&t.pts[i]) : make_float4(NAN, NAN, NAN, 0.0f);
    const float at = active && box_d2(own, t.box[0], t.stride[0], l) <= r2 ? r2 : -1.0f;
    if (!__any_sync(0xffffffffu, at >= 0.0f)) return;
    __syncwarp();
    stage[0][lane] = mate.x;
    stage[1][lane] = mate.y;
    stage[2][lane] = mate.z;
    __syncwarp();
#pragma unroll 2
    for (int c = 0; c < 32; c += 4) {
      const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(&stage[0][c]);
      const ulonglong2 y = *reinterpret_cast<const ulonglong2 *>(&stage[1][c]);
      const ulonglong2 z = *reinterpret_cast<const ulonglong2 *>(&stage[2][c]);
      const u64 a = dist2x2(x.x, y.x, z.x, nqx, nqy, nqz, minus_zero);
      const u64 b = dist2x2(x.y, y.y, z.y, nqx, nqy, nqz, minus_zero);
      const float d[4] = {half2f(a, 0), half2f(a, 1), half2f(b, 0), half2f(b, 1)};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (d[u] <= at) {
          if (cnt < RN_CAP) near[cnt][lane] = make_uint2(__float_as_uint(d[u]), l * 32 + c + u);
          ++cnt;
        }
      }
    }
  };
  tree_visit_all(t, pk, r2, leaf);
  __syncwarp();
  if (!active) return;
  const u32 qidx = __float_as_uint(q.w);
  if (cnt > RN_CAP || budget < 0) {  // (or a packet of points far apart)
    hard[atomicAdd(hard_count, 1u)] = qi;
    return;
  }
  float ax = 0.0f, ay = 0.0f, az = 0.0f;
  if (cnt >= 3) {  // normal_estimation.cpp:203
    for (int i = 0; i < cnt; ++i) {
      const uint2 e = near[i][lane];
      int rank = 0, same = 0;
#pragma unroll 8
      for (int j = 0; j < cnt; ++j) {
        const u32 f = near[j][lane].x;  // (distances are not negative: ordered as bits)
        rank += f < e.x;
        same += f == e.x;
      }
      if (same > 1) {
        const u32 own = __float_as_uint(__ldg(&t.pts[e.y]).w);
        for (int j = 0; j < cnt; ++j) {
          const uint2 f = near[j][lane];
          if (f.x == e.x) rank += __float_as_uint(__ldg(&t.pts[f.y]).w) < own;
        }
      }
      order[rank][lane] = (unsigned char)i;
    }
    nd::normal_from_points([&](int j) { return __ldg(&t.pts[near[order[j][lane]][lane].y]); }, cnt,
                           false, iters, q.x, q.y, q.z, vpx, vpy, vpz, ax, ay, az);
  }
  nx[qidx] = ax;
  ny[qidx] = ay;
  nz[qidx] = az;
}

// The points with more neighbours than a lane holds, and those of wide packets
// (hard: places in the tree), one warp each; those past CAP neighbours go on to
// `more` (places, or indices where `last`). Up to 32 points per turn: a point's sums go one to a lane
// (each in the neighbours' order, as one lane would add them), and at the end of
// the turn every lane makes the normal of one point. With all of it by one lane
// per point and room for 1024 in every block, 150,000 points of 60
// neighbours each took 1.89 ms (1.13 from lists in memory), now 0.94.
template <u32 CAP, u32 BINS>
__global__ __launch_bounds__(32) void k_radius_normals_listed(
    TreeView t, float r2, int iters, float vpx, float vpy, float vpz, float *nx, float *ny,
    float *nz, const u32 *hard, const u32 *hard_count, u32 *more, u32 *more_count, bool last) {
  __shared__ u64 s_keys[CAP];
  __shared__ u32 s_bins[BINS];
  __shared__ float s_near[3][CAP];  // in order
  __shared__ unsigned short s_perm[CAP];
  const int lane = threadIdx.x;
  const u32 n = hard ? *hard_count : t.n, chunk = min(32u, (n + gridDim.x - 1) / gridDim.x);
  // the products of the covariance: lane l adds up axis a times axis b
  const int a = lane < 3 ? 0 : (lane < 5 ? 1 : 2), b = lane < 3 ? lane : (lane == 3 ? 1 : 2);
  auto place = [&](u32 w) { return hard ? hard[w] : w; };  // (null: all points)
  for (u32 w0 = blockIdx.x * chunk; w0 < n; w0 += gridDim.x * chunk) {
    const u32 m = min(chunk, n - w0);
    float C[6] = {};
    int mine = -1;  // the lane's point's neighbours; -1: no point, or left for `more`
    for (u32 c = 0; c < m; ++c) {
      const float4 q = t.pts[place(w0 + c)];
      u32 cnt = 0;
      radius_walk<1>(t, q.x, q.y, q.z, r2, 0, [&](bool pass, float d, u32 idx) {
        const unsigned b = __ballot_sync(0xffffffffu, pass);
        const u32 at = cnt + __popc(b & ((1u << lane) - 1));
        if (pass && at < CAP) s_keys[at] = pack_nbr(d, (int)idx);
        cnt += __popc(b);
      });
      __syncwarp();
      if (cnt > CAP) {
        if (lane == 0)
          more[atomicAdd(more_count, 1u)] = last ? __float_as_uint(q.w) : place(w0 + c);
        continue;
      }
      if (lane == (int)c) mine = (int)cnt;
      if (cnt < 3) continue;
      order_keys<32, BINS>(s_keys, cnt, r2, s_bins, s_perm, nullptr, [&](u32 rank, u64 k) {
        const float4 p = __ldg(&t.pts[t.pos_of[nbr_idx(k)]]);
        s_near[0][rank] = p.x;
        s_near[1][rank] = p.y;
        s_near[2][rank] = p.z;
      });
      __syncwarp();
      // (nd::normal_from_points: the centroid, then the six products about it)
      float sum = 0.0f;
      const float *axis = s_near[lane < 3 ? lane : 0];
#pragma unroll 8
      for (u32 j = 0; j < cnt; ++j) sum = fadd(sum, axis[j]);
      sum = fmul(sum, fdiv(1.0f, (float)(int)cnt));
      const float ca = __shfl_sync(0xffffffffu, sum, a), cb = __shfl_sync(0xffffffffu, sum, b);
      float prod = 0.0f;
      const float *pa = s_near[a], *pb = s_near[b];
#pragma unroll 8
      for (u32 j = 0; j < cnt; ++j) prod = fadd(prod, fmul(fsub(pa[j], ca), fsub(pb[j], cb)));
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const float v = __shfl_sync(0xffffffffu, prod, k);
        if (lane == (int)c) C[k] = v;
      }
      __syncwarp();
    }
    if (mine >= 0) {
      const float4 q = t.pts[place(w0 + lane)];
      const u32 qidx = __float_as_uint(q.w);
      float ax = 0.0f, ay = 0.0f, az = 0.0f;
      if (mine >= 3) {  // normal_estimation.cpp:203
        float A[3][3] = {{C[0], C[1], C[2]}, {C[1], C[3], C[4]}, {C[2], C[4], C[5]}};
        nd::eigen_smallest_ref(A, iters, ax, ay, az);
        nd::flip_ref(q.x, q.y, q.z, vpx, vpy, vpz, ax, ay, az);
      }
      nx[qidx] = ax;
      ny[qidx] = ay;
      nz[qidx] = az;
    }
    __syncwarp();
  }
}

// listed queries: their coordinates
__global__ void k_gather_queries(const float *x, const float *y, const float *z, const u32 *list,
                                 size_t n, float *qx, float *qy, float *qz) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  qx[i] = x[list[i]];
  qy[i] = y[list[i]];
  qz[i] = z[list[i]];
}
}  // namespace

void hash_collision_check(rvp_context *ctx, const TreeView &t, float cell, long long p1,
                          long long p2, int *flag) {
  k_hash_check<<<1, 1024, 0, ctx->stream>>>(t.bb, cell, p1, p2, flag);
  RVP_LAUNCH_CHECK(ctx);
}

// the bound on d2, rounded once; below zero (nothing is near) for no radius
static float square_of(float radius) {
  volatile float r = radius;
  return radius >= 0.0f ? r * r : -1.0f;
}

bool tree_radius_few(size_t nq) { return nq <= kFewQueries; }
u32 tree_radius_cap() { return FT_CAP; }

void tree_radius_count(rvp_context *ctx, const TreeView &t, const TreeQueries &q, const float *qx,
                       const float *qy, const float *qz, float radius, u32 *counts, u32 *most) {
  const float r2 = square_of(radius);
  RVP_CUDA_TRY(cudaMemsetAsync(most, 0, 8, ctx->stream));
  if (tree_radius_few(q.n))
    k_radius_each<<<(q.n + 3) / 4, 128, 0, ctx->stream>>>(t, qx, qy, qz, q.n, r2, counts, most,
                                                             q.longer);
  else
    k_radius_packets<<<(q.n + 31) / 32, 32, 0, ctx->stream>>>(t, q, r2, counts, most);
  RVP_LAUNCH_CHECK(ctx);
  if (!tree_radius_few(q.n)) {
    k_radius_listed<<<ctx->num_sms * 4, 128, 0, ctx->stream>>>(t, q, r2, counts, most);
    RVP_LAUNCH_CHECK(ctx);
  }
}

void tree_radius_fill(rvp_context *ctx, const TreeView &t, const TreeQueries &q, const float *qx,
                      const float *qy, const float *qz, float radius, const u64 *full,
                      const u64 *offsets, u32 cut, u32 n_long, int32_t *idx, float *d2,
                      u64 *big_pairs, u32 *big, u32 *big_count) {
  const float r2 = square_of(radius);
  if (big_count) RVP_CUDA_TRY(cudaMemsetAsync(big_count, 0, 4, ctx->stream));
  const bool few = tree_radius_few(q.n);
  const unsigned blocks = (q.n + FT_WARPS - 1) / FT_WARPS;
  k_radius_fill<<<blocks, FT_WARPS * 32, 0, ctx->stream>>>(t, q, few ? qx : nullptr, qy, qz, r2,
                                                          full, offsets, cut, idx, d2);
  RVP_LAUNCH_CHECK(ctx);
  if (n_long) {
    k_radius_fill_long<<<n_long, FT_WARPS * 32, 0, ctx->stream>>>(
        t, q, few ? qx : nullptr, qy, qz, r2, full, offsets, cut, idx, d2, big_pairs, big,
        big_count);
    RVP_LAUNCH_CHECK(ctx);
  }
  if (big_count) {  // lists past a warp's reach
    sort_big_segments(ctx, full, big_pairs, big, big_count, std::min(q.n, 4096u));
    k_radius_big_out<<<std::min(q.n, 4096u), 256, 0, ctx->stream>>>(big_pairs, big, big_count, full,
                                                                   offsets, cut, idx, d2);
    RVP_LAUNCH_CHECK(ctx);
  }
}

void tree_radius_normals(rvp_context *ctx, const TreeView &t, float radius, int iters, float vpx,
                         float vpy, float vpz, float *nx, float *ny, float *nz, u32 *hard,
                         u32 *longer, u32 *counts) {
  const float r2 = square_of(radius);
  RVP_CUDA_TRY(cudaMemsetAsync(counts, 0, 12, ctx->stream));
  const bool few = t.n <= kFewNormals;
  if (!few) {
    k_radius_normals<<<(t.n + 31) / 32, 32, 0, ctx->stream>>>(
        t, kMinusZero2, r2, iters, vpx, vpy, vpz, nx, ny, nz, hard, counts);
    RVP_LAUNCH_CHECK(ctx);
  }
  // (by shared memory: 32 short lists at once on an SM, or 9 long ones)
  k_radius_normals_listed<FT_SHORT, FT_SHORT>
      <<<grid_for(t.n, 1, ctx->num_sms * 32), 32, 0, ctx->stream>>>(
          t, r2, iters, vpx, vpy, vpz, nx, ny, nz, few ? nullptr : hard, counts, longer, counts + 1,
          false);
  RVP_LAUNCH_CHECK(ctx);
}

void tree_radius_normals_longer(rvp_context *ctx, const TreeView &t, float radius, int iters,
                                float vpx, float vpy, float vpz, float *nx, float *ny, float *nz,
                                const u32 *longer, u32 *huge, u32 *counts) {
  const float r2 = square_of(radius);
  k_radius_normals_listed<FT_CAP, FT_BINS>
      <<<grid_for(t.n, 1, ctx->num_sms * 9), 32, 0, ctx->stream>>>(
          t, r2, iters, vpx, vpy, vpz, nx, ny, nz, longer, counts + 1, huge, counts + 2, true);
  RVP_LAUNCH_CHECK(ctx);
}

void gather_queries(rvp_context *ctx, const float *x, const float *y, const float *z,
                    const u32 *list, size_t n, float *qx, float *qy, float *qz) {
  k_gather_queries<<<grid_for(n, 256, 0), 256, 0, ctx->stream>>>(x, y, z, list, n, qx, qy, qz);
  RVP_LAUNCH_CHECK(ctx);
}

}  // namespace rvp
