// The box tree (knn_tree.cu) over the points of many frames, for the batched
// pipeline: one sort by (frame, Hilbert code), every frame's points starting
// at a multiple of 1024 tree positions, so that no leaf (32 points) and no
// level-1 node (1024) holds two frames; a search starts from its frame's
// level-1 nodes. Counts and offsets stay on the device. Positions between a
// frame's end and the next multiple hold no point (NaN coordinates, index
// 0xFFFFFFFF).
#include <algorithm>

#include "internal.cuh"
#include "knn_tree_kernels.cuh"

namespace rvp {
namespace {
inline size_t al(size_t b) { return (b + 255) & ~(size_t)255; }

// one block: each frame's quantisation and level-1 nodes
__global__ __launch_bounds__(1024) void k_frames_setup(const float *bb, const int64_t *offs,
                                                       int n_frames, int key_bits, TreeFrame *F,
                                                       uint2 *nodes, u64 *n_positions) {
  __shared__ u32 warp_sum[32];
  __shared__ u32 carry;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid == 0) carry = 0;
  __syncthreads();
  for (int f0 = 0; f0 < n_frames; f0 += 1024) {
    const int f = f0 + tid;
    u32 n = 0;
    if (f < n_frames) {
      tree_frame(bb + 6 * f, key_bits, F[f]);
      n = (u32)((offs[f + 1] - offs[f] + 1023) / 1024);
    }
    u32 incl = n;
    for (int o = 1; o < 32; o <<= 1) {
      const u32 t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sum[wid] = incl;
    __syncthreads();
    u32 before = carry;
    for (int k = 0; k < wid; ++k) before += warp_sum[k];
    if (f < n_frames) nodes[f] = make_uint2(before + incl - n, before + incl);
    __syncthreads();
    if (tid == 1023) carry = before + incl;
    __syncthreads();
  }
  if (tid == 0) *n_positions = (u64)carry * 1024;
}

__device__ __forceinline__ int frame_of(const int64_t *offs, int lo, int hi, int64_t i) {
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (offs[mid] <= i) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Keys of 2048 consecutive points per block turn: the frames they can belong
// to are found once per turn (one or two, mostly).
constexpr int FK_CHUNK = 2048;
__global__ __launch_bounds__(256) void k_frames_keys(const float *__restrict__ x,
                                                     const float *__restrict__ y,
                                                     const float *__restrict__ z,
                                                     const int64_t *offs, int n_frames,
                                                     const TreeFrame *F, int key_bits, u64 *keys,
                                                     u32 *vals, u64 *bits) {
  const int64_t n = offs[n_frames];
  __shared__ int s_lo, s_hi;
  __shared__ unsigned short table[192];
  tree_key_table(table);
  u64 ones = 0, zeros = 0;
  for (int64_t base = (int64_t)blockIdx.x * FK_CHUNK; base < n;
       base += (int64_t)gridDim.x * FK_CHUNK) {
    const int64_t end = base + FK_CHUNK < n ? base + FK_CHUNK : n;
    if (threadIdx.x == 0) s_lo = frame_of(offs, 0, n_frames - 1, base);
    if (threadIdx.x == 32) s_hi = frame_of(offs, 0, n_frames - 1, end - 1);
    __syncthreads();
    const int lo = s_lo, hi = s_hi;
    for (int64_t i = base + threadIdx.x; i < end; i += 256) {
      const int f = frame_of(offs, lo, hi, i);
      const u64 k = ((u64)f << key_bits) | tree_key<u32>(F[f], table, x[i], y[i], z[i]);
      keys[i] = k;
      vals[i] = (u32)i;
      ones |= k;
      zeros |= ~k;
    }
    __syncthreads();
  }
  if (bits) note_key_bits(ones, zeros, bits);
}

// one block per level-1 node: its 1024 records, 32 leaf boxes and own box
__global__ __launch_bounds__(1024) void k_frames_nodes(const float *__restrict__ x,
                                                       const float *__restrict__ y,
                                                       const float *__restrict__ z,
                                                       const float *__restrict__ aos,
                                                       const u32 *__restrict__ vals,
                                                       const int64_t *offs, int n_frames,
                                                       const uint2 *nodes, TreeView t,
                                                       u32 *node_frame) {
  __shared__ int s_f;
  __shared__ float s_box[6][32];
  const u32 node = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) {  // the last frame that starts at or before the node
    int lo = 0, hi = n_frames - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (nodes[mid].x <= node) lo = mid; else hi = mid - 1;
    }
    s_f = node < nodes[lo].y ? lo : -1;
    node_frame[node] = (u32)s_f;
  }
  __syncthreads();
  const int f = s_f;
  if (f < 0) return;  // past the last frame
  const int64_t r = offs[f] + (int64_t)(node - nodes[f].x) * 1024 + threadIdx.x;
  const u32 p = node * 1024 + threadIdx.x;
  float m[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  float4 rec = make_float4(NAN, NAN, NAN, __uint_as_float(0xFFFFFFFFu));
  if (r < offs[f + 1]) {
    const u32 v = vals[r];
    const float c[3] = {aos[3 * (size_t)v], aos[3 * (size_t)v + 1], aos[3 * (size_t)v + 2]};
    rec = make_float4(c[0], c[1], c[2], __uint_as_float(v));
    t.pos_of[v] = p;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      m[a] = fminf(m[a], c[a]);
      m[3 + a] = fmaxf(m[3 + a], c[a]);
    }
  }
  t.pts[p] = rec;
  box_out(m, t.box[0], t.stride[0], node * 32 + w);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < 6; ++k) s_box[k][w] = m[k];
  __syncthreads();
  if (w == 0) {
    float b[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) b[k] = s_box[k][lane];
    box_out(b, t.box[1], t.stride[1], node);
  }
}

// Small frames: a block sorts its frame's points by Hilbert code in registers
// and shared memory (bitonic, 21 bits of code and the point's number; R points
// per thread) and writes its leaves and the one or two level-1 nodes that
// every frame has room for. Bound by the latency of the sort's 55 or 66 steps;
// 512 frames of 1024 points 41 us.
template <int R>
__device__ __forceinline__ void small_frame_sort(u32 (&key)[R], u32 *s_key) {
  const u32 tid = threadIdx.x;
  constexpr u32 N = 1024 * R;  // element r of a thread: r * 1024 + tid
#pragma unroll 1
  for (u32 k = 2; k <= N; k <<= 1) {
#pragma unroll 1
    for (u32 j = k >> 1; j > 0; j >>= 1) {
      if (j == 1024) {  // (R = 2, k = 2048: both in this thread, ascending)
        const u32 a = min(key[0], key[R - 1]), b = max(key[0], key[R - 1]);
        key[0] = a;
        key[R - 1] = b;
        continue;
      }
      if (j >= 32) {
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) s_key[r * 1024 + tid] = key[r];
        __syncthreads();
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const u32 i = r * 1024 + tid;
        const u32 o = j >= 32 ? s_key[i ^ j] : __shfl_xor_sync(0xffffffffu, key[r], j);
        const bool low = ((i & j) == 0) == ((i & k) == 0);  // keeps the smaller
        key[r] = low ? min(key[r], o) : max(key[r], o);
      }
    }
  }
}

template <int R>
__device__ __forceinline__ void small_frame(const float *x, const float *y, const float *z,
                                            int64_t a, int m, int f, const TreeFrame &F,
                                            const unsigned short *table, u32 *s_key,
                                            float (*s_box)[32], const TreeView &t) {
  const u32 tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  u32 key[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const u32 i = r * 1024 + tid;
    key[r] = 0xFFFFFFFFu;
    if ((int)i < m) key[r] = (tree_key<u32>(F, table, x[a + i], y[a + i], z[a + i]) << 11) | i;
  }
  small_frame_sort<R>(key, s_key);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const u32 p = (u32)f * kSmallFrame + r * 1024 + tid;
    float b[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    float4 rec = make_float4(NAN, NAN, NAN, __uint_as_float(0xFFFFFFFFu));
    if ((int)(r * 1024 + tid) < m) {
      const u32 v = (u32)a + (key[r] & 2047u);
      rec = make_float4(x[v], y[v], z[v], __uint_as_float(v));
      t.pos_of[v] = p;
      b[0] = b[3] = rec.x;
      b[1] = b[4] = rec.y;
      b[2] = b[5] = rec.z;
    }
    t.pts[p] = rec;
    box_out(b, t.box[0], t.stride[0], p / 32);
    __syncthreads();
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < 6; ++k) s_box[k][w] = b[k];
    __syncthreads();
    if (w == 0) {
#pragma unroll
      for (int k = 0; k < 6; ++k) b[k] = s_box[k][lane];
      box_out(b, t.box[1], t.stride[1], p / 1024);
    }
  }
}

__global__ __launch_bounds__(1024) void k_small_frames(const float *__restrict__ x,
                                                       const float *__restrict__ y,
                                                       const float *__restrict__ z,
                                                       const int64_t *offs, TreeView t,
                                                       uint2 *nodes, u32 *node_frame,
                                                       int32_t *skipped) {
  __shared__ u32 s_key[kSmallFrame];
  __shared__ float s_box[6][32];
  __shared__ float s_bb[6];
  __shared__ TreeFrame F;
  __shared__ unsigned short table[192];
  const u32 tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int f = blockIdx.x;
  const int64_t a = offs[f], n = offs[f + 1] - a;
  const int m = n <= kSmallFrame ? (int)n : 0;
  float b[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  bool odd = n > kSmallFrame;
  for (int i = tid; i < m; i += 1024) {
    const float c[3] = {x[a + i], y[a + i], z[a + i]};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      odd = odd || !(fabsf(c[k]) < 1e18f);
      b[k] = fminf(b[k], c[k]);
      b[3 + k] = fmaxf(b[3 + k], c[k]);
    }
  }
  tree_key_table(table);
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    for (int o = 16; o; o >>= 1) {
      const float v = __shfl_xor_sync(0xffffffffu, b[k], o);
      b[k] = k < 3 ? fminf(b[k], v) : fmaxf(b[k], v);
    }
    if (lane == 0) s_box[k][w] = b[k];
  }
  odd = __syncthreads_or(odd);
  const int used = odd ? 0 : (m + 1023) / 1024;  // level-1 nodes
  if (tid < 2) node_frame[2 * f + tid] = (int)tid < used ? (u32)f : 0xFFFFFFFFu;
  if (tid == 0) {
    nodes[f] = make_uint2(2 * f, 2 * f + used);
    skipped[f] = odd ? 1 : 0;
  }
  if (!used) return;
  if (w < 6) {
    float v = s_box[w][lane];
    for (int o = 16; o; o >>= 1) {
      const float u = __shfl_xor_sync(0xffffffffu, v, o);
      v = w < 3 ? fminf(v, u) : fmaxf(v, u);
    }
    if (lane == 0) s_bb[w] = v;
  }
  __syncthreads();
  if (tid == 0) tree_frame(s_bb, 21, F);
  __syncthreads();
  if (used == 1) small_frame<1>(x, y, z, a, m, f, F, table, s_key, s_box, t);
  else small_frame<2>(x, y, z, a, m, f, F, table, s_key, s_box, t);
}

// points removed by an earlier stage: flagged, and nowhere near anything
__global__ void k_frames_mark(float4 *pts, const u64 *n_positions, const uint8_t *keep) {
  const u64 n = *n_positions;
  for (u64 p = blockIdx.x * (u64)blockDim.x + threadIdx.x; p < n;
       p += (u64)gridDim.x * blockDim.x) {
    const u32 idx = __float_as_uint(pts[p].w);
    if (idx != 0xFFFFFFFFu && !keep[idx])
      pts[p] = make_float4(NAN, NAN, NAN, __uint_as_float(idx | 0x80000000u));
  }
}
}  // namespace

size_t tree_frames_positions(size_t n_max, int n_frames) {
  return (n_max + 1023 + (size_t)n_frames * 1023) / 1024 * 1024;
}

void KnnTree::reserve_frames(size_t n_max, int n_frames) {
  const size_t P = tree_frames_positions(n_max, n_frames), nf = (size_t)n_frames;
  pts.reserve(P * 16);
  pos.reserve(n_max * 4);
  hard.reserve(P * 4 + 256);
  boxes.reserve((P / 32 + P / 1024 + 32) * 24);
  misc.reserve(256 + al(nf * 24) + al(nf * sizeof(TreeFrame)) + al(nf * 8) + al(P / 1024 * 4));
}

TreeView tree_build_frames(rvp_context *ctx, KnnTree &w, const float *x, const float *y,
                           const float *z, const float *aos, const int64_t *offs, int n_frames,
                           size_t n_max, u64 *keys, u32 *vals, void *sort_temp) {
  const size_t P = tree_frames_positions(n_max, n_frames);
  w.reserve_frames(n_max, n_frames);
  TreeView t{};
  t.n = (u32)P;
  t.count[0] = t.stride[0] = (u32)(P / 32);
  t.count[1] = (u32)(P / 1024);
  t.stride[1] = (t.count[1] + 31) & ~31u;
  t.box[0] = w.boxes.as<float>();
  t.box[1] = t.box[0] + (size_t)t.stride[0] * 6;
  const size_t nf = (size_t)n_frames;
  char *m = w.misc.as<char>();
  u64 *n_positions = reinterpret_cast<u64 *>(m); m += 256;
  float *bb = reinterpret_cast<float *>(m); m += al(nf * 24);
  TreeFrame *F = reinterpret_cast<TreeFrame *>(m); m += al(nf * sizeof(TreeFrame));
  uint2 *nodes = reinterpret_cast<uint2 *>(m); m += al(nf * 8);
  u32 *node_frame = reinterpret_cast<u32 *>(m);
  t.pts = w.pts.as<float4>();
  t.pos_of = w.pos.as<u32>();
  t.frame_nodes = nodes;
  t.node_frame = node_frame;
  t.n_positions = n_positions;
  // the frame's number and the code share 32 bits (four digits to sort), the
  // code at least 18 of them
  int fb = 0;
  while (((size_t)1 << fb) < nf) ++fb;
  const int key_bits = kTreeKeyBits - (fb < 14 ? fb : 14);
  cudaStream_t st = ctx->stream;
  frames_bbox(ctx, x, y, z, offs, n_frames, n_max, bb);
  k_frames_setup<<<1, 1024, 0, st>>>(bb, offs, n_frames, key_bits, F, nodes, n_positions);
  RVP_LAUNCH_CHECK(ctx);
  SortTemp tmp;
  sort_temp_carve(tmp, sort_temp, n_max);
  u64 *bits = sort_key_bits(ctx, tmp, n_max);
  k_frames_keys<<<grid_for(n_max, FK_CHUNK, ctx->num_sms * 8), 256, 0, st>>>(
      x, y, z, offs, n_frames, F, key_bits, keys, vals, bits);
  RVP_LAUNCH_CHECK(ctx);
  radix_sort_pairs(ctx, keys, vals, n_max, reinterpret_cast<const u64 *>(offs + n_frames), tmp,
                   bits);
  k_frames_nodes<<<t.count[1], 1024, 0, st>>>(x, y, z, aos, vals, offs, n_frames,
                                              nodes, t, node_frame);
  RVP_LAUNCH_CHECK(ctx);
  return t;
}

TreeView tree_build_small_frames(rvp_context *ctx, KnnTree &w, const float *x, const float *y,
                                 const float *z, const int64_t *offs, int n_frames, size_t n_max,
                                 int32_t *skipped) {
  const size_t nf = (size_t)n_frames, P = nf * kSmallFrame;
  w.pts.reserve(P * 16);
  w.pos.reserve(n_max * 4);
  w.hard.reserve(P * 4 + 256);
  TreeView t{};
  t.n = (u32)P;
  t.count[0] = t.stride[0] = (u32)(P / 32);
  t.count[1] = (u32)(P / 1024);
  t.stride[1] = (t.count[1] + 31) & ~31u;
  w.boxes.reserve(((size_t)t.stride[0] + t.stride[1]) * 24);
  w.misc.reserve(al(nf * 8) + nf * 8);
  t.box[0] = w.boxes.as<float>();
  t.box[1] = t.box[0] + (size_t)t.stride[0] * 6;
  t.pts = w.pts.as<float4>();
  t.pos_of = w.pos.as<u32>();
  uint2 *nodes = w.misc.as<uint2>();
  u32 *node_frame = reinterpret_cast<u32 *>(w.misc.as<char>() + al(nf * 8));
  t.frame_nodes = nodes;
  t.node_frame = node_frame;
  k_small_frames<<<(unsigned)nf, 1024, 0, ctx->stream>>>(x, y, z, offs, t, nodes, node_frame,
                                                         skipped);
  RVP_LAUNCH_CHECK(ctx);
  return t;
}

void tree_frames_mark_removed(rvp_context *ctx, const TreeView &t, const uint8_t *keep) {
  k_frames_mark<<<grid_for(t.n, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(
      t.pts, t.n_positions, keep);
  RVP_LAUNCH_CHECK(ctx);
}

void tree_knn_frames(rvp_context *ctx, KnnTree &w, const TreeView &t, const u32 *list,
                     const u64 *n_list, int k, int mode, const TreeOut &o) {
  TreeQueries q{};
  q.n = t.n;
  q.list = list;
  q.n_list = n_list;
  q.hard_count = w.hard.as<u32>();
  q.hard = q.hard_count + 64;
  RVP_CUDA_TRY(cudaMemsetAsync(q.hard_count, 0, 4, ctx->stream));
  const u32 packets = t.n / 32;
  const int listed = k == 1 ? 1 : k - 1;
  switch (mode) {
    case TREE_MEAN:
      launch_tree_k<TREE_MEAN, true>(ctx, t, q, packets, k, listed, INFINITY, o);
      break;
    case TREE_PAIRS:
      launch_tree_k<TREE_PAIRS, true>(ctx, t, q, packets, k, listed, INFINITY, o);
      break;
    case TREE_LIST:
      launch_tree_k<TREE_LIST, true>(ctx, t, q, packets, k, listed, INFINITY, o);
      break;
    default: launch_tree_k<TREE_NORMALS, true>(ctx, t, q, packets, k, listed, INFINITY, o);
  }
}

}  // namespace rvp
