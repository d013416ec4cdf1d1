// PCA normals (features/normal_estimation.cpp).
//
// Reference path: per point, the neighbour list in (d2, index) order,
// centroid (sum then "* (1.0f / n)" in compute_covariance_rvv :117-142, or
// "/ (k+1)" in normal_estimation_sc :90-95), six covariance sums, then
// simple_eigen3x3_smallest (:16-52: `iters` rotations on the largest
// off-diagonal entry, updating only A[p][p], A[q][q], A[p][q] and V) and the
// viewpoint flip (:55-67). Every step keeps the reference's operation order
// with separately rounded products and sums; atan2f/cosf/sinf are CUDA's,
// which is why normals are compared within a tolerance.
//
#include <math.h>

#include "internal.cuh"
#include "normals_device.cuh"

namespace rvp {
using namespace nd;

namespace {

// One thread per list slot i: query qi = order ? order[i] : i, neighbours
// pairs[offsets[i] ..) or pairs[i*fixed_k ..), result at out_pos[qi] (or qi).
__global__ void k_normals_lists(const float *__restrict__ x, const float *__restrict__ y,
                                const float *__restrict__ z, const u64 *__restrict__ pairs,
                                const u64 *__restrict__ offsets,
                                const int32_t *__restrict__ fixed_counts, int fixed_k,
                                size_t n_max, const u64 *n_dev, bool div_centroid, int iters,
                                float vpx, float vpy, float vpz, const float *qx,
                                const float *qy, const float *qz, float *nx, float *ny,
                                float *nz, const u32 *order, const u64 *out_pos) {
  const size_t n = n_dev ? *n_dev : n_max;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const u64 *l;
    int m;
    if (offsets) {
      l = pairs + offsets[i];
      m = (int)(offsets[i + 1] - offsets[i]);
    } else {
      l = pairs + i * (size_t)fixed_k;
      m = fixed_counts ? fixed_counts[i] : fixed_k;
    }
    const size_t qi = order ? (size_t)order[i] : i;
    const size_t oi = out_pos ? (size_t)out_pos[qi] : qi;
    if (m < 3) {  // normal_estimation.cpp:203
      nx[oi] = ny[oi] = nz[oi] = 0.0f;
      continue;
    }
    float a, b, c;
    normal_from_list(x, y, z, [&](int t) { return nbr_idx(l[t]) & 0x7FFFFFFF; }, m, div_centroid,
                     iters, qx[qi], qy[qi], qz[qi], vpx, vpy, vpz, a, b, c);
    nx[oi] = a;
    ny[oi] = b;
    nz[oi] = c;
  }
}

}  // namespace

void normals_from_lists(rvp_context *ctx, const float *x, const float *y, const float *z,
                        const u64 *pairs, const u64 *offsets, const int32_t *fixed_counts,
                        int fixed_k, size_t n_max, const u64 *n_dev, bool div_centroid, int iters,
                        float vpx, float vpy, float vpz, const float *qx, const float *qy,
                        const float *qz, float *nx, float *ny, float *nz, const u32 *order,
                        const u64 *out_pos) {
  k_normals_lists<<<grid_for(n_max, 128, ctx->num_sms * 32), 128, 0, ctx->stream>>>(
      x, y, z, pairs, offsets, fixed_counts, fixed_k, n_max, n_dev, div_centroid, iters, vpx, vpy,
      vpz, qx, qy, qz, nx, ny, nz, order, out_pos);
  RVP_LAUNCH_CHECK(ctx);
}

}  // namespace rvp
