// Exact k nearest neighbours in one cloud (k <= 64) over a 32-wide box tree.
//
// Build: the points sorted by the Hilbert code of their quantised position
// (32 bits or more, one power-of-two cell for all axes), every 32 consecutive points
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
// its rank. Queries that do not fit this (far from their packet, many equal
// distances) are listed and answered one per warp by a second kernel, as are
// few queries of their own (tree_knn_few).
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
#include <algorithm>

#include "internal.cuh"
#include "knn_tree_kernels.cuh"

namespace rvp {

namespace {
// ---------------------------------------------------------------------------
// build
// ---------------------------------------------------------------------------
// KnnTree::misc
struct TreeMisc {
  float bb[8];                    // the box
  alignas(16) TreeSample sample;  // and a sample
  u64 n_sort;                     // queries to sort
};
__global__ void k_tree_init(TreeMisc *m) {
  if (threadIdx.x < 3) m->bb[threadIdx.x] = INFINITY;
  else if (threadIdx.x < 6) m->bb[threadIdx.x] = -INFINITY;
}

// The cloud's box, six atomics per block (at most kBoxBlocks blocks per SM: the
// atomics meet on the same words), and beside them a block for the sample.
constexpr int kBoxBlocks = 4;
__global__ __launch_bounds__(256) void k_tree_box(const float *__restrict__ x,
                                                  const float *__restrict__ y,
                                                  const float *__restrict__ z, size_t n,
                                                  TreeMisc *misc) {
  __shared__ float part[6][8];
  __shared__ TreeSample S;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const u32 blocks = gridDim.x - 1;
  if (blockIdx.x == blocks) {
    tree_sample(x, y, z, n, &S);
    __syncthreads();
    if (tid == 0) misc->sample = S;
    return;
  }
  const size_t per = ((n + blocks - 1) / blocks + 255) & ~(size_t)255;
  const size_t from = blockIdx.x * per, to = from + per < n ? from + per : n;
  float m[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 4
  for (size_t i = from + tid; i < to; i += 256) {
    const float v[3] = {x[i], y[i], z[i]};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      m[a] = fminf(m[a], v[a]);
      m[3 + a] = fmaxf(m[3 + a], v[a]);
    }
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const float t = __shfl_xor_sync(0xffffffffu, m[k], o);
      m[k] = k < 3 ? fminf(m[k], t) : fmaxf(m[k], t);
    }
    if (lane == 0) part[k][wid] = m[k];
  }
  __syncthreads();
  if (tid < 6) {
    float v = part[tid][0];
#pragma unroll
    for (int w = 1; w < 8; ++w) v = tid < 3 ? fminf(v, part[tid][w]) : fmaxf(v, part[tid][w]);
    if (tid < 3) {
      if (v < INFINITY) atomic_min_f(misc->bb + tid, v);
    } else if (v > -INFINITY) {
      atomic_max_f(misc->bb + tid, v);
    }
  }
}

__global__ __launch_bounds__(256) void k_tree_keys(const float *__restrict__ x,
                                                   const float *__restrict__ y,
                                                   const float *__restrict__ z, size_t n_max,
                                                   const u64 *n_dev, const TreeMisc *misc,
                                                   size_t n_cloud, u64 *keys, u32 *vals,
                                                   u64 *bits) {
  __shared__ TreeFrame F;
  __shared__ unsigned short table[192];
  const size_t n = n_dev ? *n_dev : n_max;
  if (n == 0) return;
  if (threadIdx.x == 255)
    tree_frame_fine(n_cloud, misc->bb, misc->sample, tree_key_bits(n_cloud), F);
  tree_key_table(table);
  __syncthreads();
  u64 ones = 0, zeros = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const u64 k = tree_key<u64>(F, table, x[i], y[i], z[i]);
    keys[i] = k;
    vals[i] = (u32)i;
    ones |= k;
    zeros |= ~k;
  }
  if (bits) note_key_bits(ones, zeros, bits);
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

}  // namespace

void KnnTree::release() {
  keys.release(); vals.release(); sort.release(); pts.release(); pos.release(); boxes.release();
  misc.release(); qkeys.release(); qvals.release(); qpts.release(); hard.release();
  rows.release();
}

TreeView tree_build(rvp_context *ctx, KnnTree &w, const float *x, const float *y, const float *z,
                    size_t n) {
  w.keys.reserve(n * 8);
  w.vals.reserve(n * 4);
  w.sort.reserve(sort_temp_bytes(n));
  w.pts.reserve(n * 16);
  w.pos.reserve(n * 4);
  w.misc.reserve(sizeof(TreeMisc));
  TreeMisc *misc = w.misc.as<TreeMisc>();
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
  t.bb = misc->bb;
  cudaStream_t st = ctx->stream;
  const int sms = ctx->num_sms;
  k_tree_init<<<1, 32, 0, st>>>(misc);
  RVP_LAUNCH_CHECK(ctx);
  k_tree_box<<<grid_for(n, 256, sms * kBoxBlocks) + 1, 256, 0, st>>>(x, y, z, n, misc);
  RVP_LAUNCH_CHECK(ctx);
  SortTemp tmp;
  sort_temp_carve(tmp, w.sort.ptr, n);
  u64 *bits = sort_key_bits(ctx, tmp, n);
  k_tree_keys<<<grid_for(n, 256, sms * 8), 256, 0, st>>>(x, y, z, n, nullptr, misc, n,
                                                         w.keys.as<u64>(), w.vals.as<u32>(), bits);
  RVP_LAUNCH_CHECK(ctx);
  radix_sort_pairs(ctx, w.keys.as<u64>(), w.vals.as<u32>(), n, nullptr, tmp, bits);
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
  u64 *n_sort = &w.misc.as<TreeMisc>()->n_sort;
  cudaStream_t st = ctx->stream;
  const unsigned gb = grid_for(nq, 256, ctx->num_sms * 8);
  k_tree_count<<<1, 1, 0, st>>>(n_sort, nq == t.n ? 0 : (u64)nq);
  RVP_LAUNCH_CHECK(ctx);
  if (nq == t.n) {
    k_tree_same<<<gb, 256, 0, st>>>(qx, qy, qz, x, y, z, nq, n_sort);
    RVP_LAUNCH_CHECK(ctx);
  }
  SortTemp tmp;
  sort_temp_carve(tmp, w.sort.ptr, nq);
  u64 *bits = sort_key_bits(ctx, tmp, nq);
  k_tree_keys<<<gb, 256, 0, st>>>(qx, qy, qz, nq, n_sort, w.misc.as<TreeMisc>(), t.n, w.qkeys.as<u64>(),
                                  w.qvals.as<u32>(), bits);
  RVP_LAUNCH_CHECK(ctx);
  radix_sort_pairs(ctx, w.qkeys.as<u64>(), w.qvals.as<u32>(), nq, n_sort, tmp, bits);
  k_tree_queries<<<gb, 256, 0, st>>>(qx, qy, qz, w.qvals.as<u32>(), n_sort, w.qpts.as<float4>());
  RVP_LAUNCH_CHECK(ctx);
  q.q = w.qpts.as<float4>();
  q.keys = w.qkeys.as<u64>();
  q.n_sort = n_sort;
  return q;
}

// A packet of 32 queries takes some 200 us from end to end (with the sort that
// makes packets of queries), however few there are; one query per warp takes
// none of this, but five times the work. Queries among 400,000 LiDAR points,
// k 16, packets and warps: 1000 queries 309 and 90 us, 16,000 360 and 200, 32,000
// 338 and 313, 64,000 334 and 590. Within 0.3 m of 150,000: 10,000 201 and 59,
// 75,000 206 and 148, 110,000 228 and 203; within 1.5 m 256 and 72, 250 and 243,
// 280 and 331; of a room's points within 0.1 m 75,000 260 and 238, 110,000 295
// and 335.
bool tree_knn_few(size_t nq, float radius) { return nq <= (radius > 0.0f ? 81920u : 24576u); }

void tree_knn(rvp_context *ctx, const TreeView &t, const TreeQueries &q, int k, float radius,
              int mode, const TreeOut &o) {
  // the radius search's bound: d2 <= radius * radius in float
  volatile float r = radius;
  const float bound = radius > 0.0f ? r * r : INFINITY;
  if (q.each[0]) {
    if (mode == TREE_MEAN) launch_tree_each<TREE_MEAN, false>(ctx, t, q, q.n, k, bound, o);
    else launch_tree_each<TREE_PAIRS, false>(ctx, t, q, q.n, k, bound, o);
    return;
  }
  const u32 packets = (q.n + 31) / 32;
  // the list leaves the point itself out where the host knows that the
  // queries are the cloud (n_sort: the device finds out)
  const int listed = q.n_sort || k == 1 ? k : k - 1;
  switch (mode) {
    case TREE_MEAN:
      launch_tree_k<TREE_MEAN, false>(ctx, t, q, packets, k, listed, bound, o);
      break;
    case TREE_PAIRS:
      launch_tree_k<TREE_PAIRS, false>(ctx, t, q, packets, k, listed, bound, o);
      break;
    case TREE_NORMALS:
      launch_tree_k<TREE_NORMALS, false>(ctx, t, q, packets, k, listed, bound, o);
      break;
    default: launch_tree_k<TREE_PRECISE, false>(ctx, t, q, packets, k, listed, bound, o);
  }
}

}  // namespace rvp
