// Device-side helpers of the box tree (knn_tree.cu, radius_tree.cu): distances
// to boxes and to two points at once, and the walk within a fixed radius.
#pragma once

#include "internal.cuh"

namespace rvp {
namespace td {

// dist2 of two points: p + (-q) is p - q
__device__ __forceinline__ u64 dist2x2(u64 px, u64 py, u64 pz, u64 nqx, u64 nqy, u64 nqz,
                                        u64 mz) {
  const u64 dx = add2(px, nqx), dy = add2(py, nqy), dz = add2(pz, nqz);
  return add2(add2(mul2(dx, dx, mz), mul2(dy, dy, mz)), mul2(dz, dz, mz));
}

// the squared distance between two boxes (a point is a box), with the
// operations of dist2
__device__ __forceinline__ float box_gap(float alo, float ahi, float blo, float bhi) {
  return fmaxf(fmaxf(fsub(blo, ahi), fsub(alo, bhi)), 0.0f);
}
struct Box {
  float lo[3], hi[3];
};
__device__ __forceinline__ float box_d2(const Box &q, const float *box, u32 stride, u32 c) {
  float g[3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
    g[a] = box_gap(q.lo[a], q.hi[a], __ldg(&box[(size_t)a * stride + c]),
                   __ldg(&box[(size_t)(3 + a) * stride + c]));
  return fadd(fadd(fmul(g[0], g[0]), fmul(g[1], g[1])), fmul(g[2], g[2]));
}

// the leaf where a query of this key would lie
__device__ __forceinline__ u32 leaf_of_key(const TreeView &t, u64 key) {
  u32 lo = 0, hi = t.n - 1;
  while (lo < hi) {
    const u32 m = (lo + hi) >> 1;
    if (t.keys[m] < key) lo = m + 1; else hi = m;
  }
  return lo / 32;
}

// the box of a warp's points (those with `in`)
__device__ __forceinline__ Box warp_box(const float4 &q, bool in) {
  Box b;
  const float v[3] = {q.x, q.y, q.z};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float lo = in ? v[a] : INFINITY, hi = in ? v[a] : -INFINITY;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    b.lo[a] = lo;
    b.hi[a] = hi;
  }
  return b;
}

// Visits every node of level END within sqrt(lim) of the box q, in tree order
// (END 0: leaves). All lanes take part.
template <int LV, int END, class Leaf>
__device__ __forceinline__ void tree_visit(const TreeView &t, const Box &q, u32 first, float lim,
                                           Leaf &leaf) {
  const u32 c = first + (threadIdx.x & 31);
  unsigned m = __ballot_sync(
      0xffffffffu, c < t.count[LV] && box_d2(q, t.box[LV], t.stride[LV], c) <= lim);
  while (m) {
    const int s = __ffs(m) - 1;
    m &= m - 1;
    if constexpr (LV == END) leaf(first + s);
    else tree_visit<LV - 1, END>(t, q, (first + s) * 32, lim, leaf);
  }
}
template <int END = 0, class Leaf>
__device__ __forceinline__ void tree_visit_all(const TreeView &t, const Box &q, float lim,
                                               Leaf &leaf) {
  for (u32 f = 0; f < t.count[kTreeLevels - 1]; f += 32)
    tree_visit<kTreeLevels - 1, END>(t, q, f, lim, leaf);
}

}  // namespace td
}  // namespace rvp
