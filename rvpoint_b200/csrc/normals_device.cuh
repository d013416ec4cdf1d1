// Reference normal arithmetic shared by the normal kernels (normals.cu) and
// the fused kNN + normal tile kernel (knn_tile.cu):
// simple_eigen3x3_smallest (normal_estimation.cpp:16-52) and
// flipNormalTowardsViewpoint (:55-67), every product and sum rounded on its
// own in the reference's order.
#pragma once

#include <math.h>

#include "internal.cuh"

namespace rvp {
namespace nd {

// One Jacobi rotation of the reference's loop body on the pair (P, Q), with
// every index static so that A and V stay in registers.
template <int P, int Q>
__device__ __forceinline__ void jacobi_rotate_ref(float (&A)[3][3], float (&V)[3][3]) {
  const float app = A[P][P], aqq = A[Q][Q], apq = A[P][Q];
  const float phi = fmul(0.5f, atan2f(fmul(2.0f, apq), fsub(app, aqq)));
  const float c = cosf(phi), s = sinf(phi);
  const float cc = fmul(c, c), ss = fmul(s, s), s2c = fmul(fmul(2.0f, s), c);
  // c*c*app - 2*s*c*apq + s*s*aqq ; s*s*app + 2*s*c*apq + c*c*aqq
  A[P][P] = fadd(fsub(fmul(cc, app), fmul(s2c, apq)), fmul(ss, aqq));
  A[Q][Q] = fadd(fadd(fmul(ss, app), fmul(s2c, apq)), fmul(cc, aqq));
  A[P][Q] = 0.0f;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const float vip = V[r][P], viq = V[r][Q];
    V[r][P] = fsub(fmul(c, vip), fmul(s, viq));
    V[r][Q] = fadd(fmul(s, vip), fmul(c, viq));
  }
}

// The reference's Jacobi loop: each iteration rotates the pair with the
// largest upper off-diagonal |A[p][q]| (first of equals), which it reads from
// the upper triangle only; the lower triangle is never read.
__device__ __forceinline__ void eigen_smallest_ref(float A[3][3], int iters, float &nx, float &ny, float &nz) {
  float (&M)[3][3] = *reinterpret_cast<float (*)[3][3]>(A);
  float V[3][3] = {{1.f, 0.f, 0.f}, {0.f, 1.f, 0.f}, {0.f, 0.f, 1.f}};
  for (int it = 0; it < iters; ++it) {
    int pq = 0;  // 0: (0,1), 1: (0,2), 2: (1,2)
    float max_off = fabsf(M[0][1]);
    if (fabsf(M[0][2]) > max_off) { pq = 1; max_off = fabsf(M[0][2]); }
    if (fabsf(M[1][2]) > max_off) pq = 2;
    if (pq == 0) jacobi_rotate_ref<0, 1>(M, V);
    else if (pq == 1) jacobi_rotate_ref<0, 2>(M, V);
    else jacobi_rotate_ref<1, 2>(M, V);
  }
  float d0 = M[0][0], d1 = M[1][1], d2 = M[2][2];
  int m = 0;
  float dm = d0;
  if (d1 < dm) { m = 1; dm = d1; }
  if (d2 < dm) m = 2;
  nx = m == 0 ? V[0][0] : (m == 1 ? V[0][1] : V[0][2]);
  ny = m == 0 ? V[1][0] : (m == 1 ? V[1][1] : V[1][2]);
  nz = m == 0 ? V[2][0] : (m == 1 ? V[2][1] : V[2][2]);
}

__device__ __forceinline__ void flip_ref(float px, float py, float pz, float vpx, float vpy,
                                         float vpz, float &nx, float &ny, float &nz) {
  const float vx = fsub(vpx, px), vy = fsub(vpy, py), vz = fsub(vpz, pz);
  const float dot = fadd(fadd(fmul(vx, nx), fmul(vy, ny)), fmul(vz, nz));
  if (dot < 0.0f) {
    nx = -nx;
    ny = -ny;
    nz = -nz;
  }
}


// Centroid, six covariance sums, eigen-solve and flip over the neighbour
// list nb(0..m-1) (indices into x, y, z), in list order. div_centroid:
// normal_estimation_sc's "/ (k+1)"; else compute_covariance_rvv's
// "* (1.0f / n)" (normal_estimation.cpp:90-95 / :117-142).
template <class Idx>
__device__ __forceinline__ void normal_from_list(const float *__restrict__ x,
                                                 const float *__restrict__ y,
                                                 const float *__restrict__ z, Idx nb, int m,
                                                 bool div_centroid, int iters, float qx,
                                                 float qy, float qz, float vpx, float vpy,
                                                 float vpz, float &nx, float &ny, float &nz) {
  float cx = 0.0f, cy = 0.0f, cz = 0.0f;
  for (int t = 0; t < m; ++t) {
    const int j = nb(t);
    cx = fadd(cx, x[j]);
    cy = fadd(cy, y[j]);
    cz = fadd(cz, z[j]);
  }
  if (div_centroid) {
    const float fm = (float)m;
    cx = fdiv(cx, fm);
    cy = fdiv(cy, fm);
    cz = fdiv(cz, fm);
  } else {
    const float inv_n = fdiv(1.0f, (float)m);
    cx = fmul(cx, inv_n);
    cy = fmul(cy, inv_n);
    cz = fmul(cz, inv_n);
  }
  float c00 = 0, c01 = 0, c02 = 0, c11 = 0, c12 = 0, c22 = 0;
  for (int t = 0; t < m; ++t) {
    const int j = nb(t);
    const float dx = fsub(x[j], cx), dy = fsub(y[j], cy), dz = fsub(z[j], cz);
    c00 = fadd(c00, fmul(dx, dx));
    c01 = fadd(c01, fmul(dx, dy));
    c02 = fadd(c02, fmul(dx, dz));
    c11 = fadd(c11, fmul(dy, dy));
    c12 = fadd(c12, fmul(dy, dz));
    c22 = fadd(c22, fmul(dz, dz));
  }
  float A[3][3] = {{c00, c01, c02}, {c01, c11, c12}, {c02, c12, c22}};
  eigen_smallest_ref(A, iters, nx, ny, nz);
  flip_ref(qx, qy, qz, vpx, vpy, vpz, nx, ny, nz);
}

}  // namespace nd
}  // namespace rvp

namespace rvp {
namespace nd {
// normal_from_list over a register-resident list of M neighbours'
// coordinates (compile-time length: every index below is static).
template <int M>
__device__ __forceinline__ void normal_from_coords(const float (&px)[M], const float (&py)[M],
                                                   const float (&pz)[M], bool div_centroid,
                                                   int iters, float qx, float qy, float qz,
                                                   float vpx, float vpy, float vpz, float &nx,
                                                   float &ny, float &nz) {
  float cx = 0.0f, cy = 0.0f, cz = 0.0f;
#pragma unroll
  for (int t = 0; t < M; ++t) {
    cx = fadd(cx, px[t]);
    cy = fadd(cy, py[t]);
    cz = fadd(cz, pz[t]);
  }
  if (div_centroid) {
    const float fm = (float)M;
    cx = fdiv(cx, fm);
    cy = fdiv(cy, fm);
    cz = fdiv(cz, fm);
  } else {
    const float inv_n = fdiv(1.0f, (float)M);
    cx = fmul(cx, inv_n);
    cy = fmul(cy, inv_n);
    cz = fmul(cz, inv_n);
  }
  float c00 = 0, c01 = 0, c02 = 0, c11 = 0, c12 = 0, c22 = 0;
#pragma unroll
  for (int t = 0; t < M; ++t) {
    const float dx = fsub(px[t], cx), dy = fsub(py[t], cy), dz = fsub(pz[t], cz);
    c00 = fadd(c00, fmul(dx, dx));
    c01 = fadd(c01, fmul(dx, dy));
    c02 = fadd(c02, fmul(dx, dz));
    c11 = fadd(c11, fmul(dy, dy));
    c12 = fadd(c12, fmul(dy, dz));
    c22 = fadd(c22, fmul(dz, dz));
  }
  float A[3][3] = {{c00, c01, c02}, {c01, c11, c12}, {c02, c12, c22}};
  eigen_smallest_ref(A, iters, nx, ny, nz);
  flip_ref(qx, qy, qz, vpx, vpy, vpz, nx, ny, nz);
}

// The same over M indices (compile-time length) given by idx(t) into x, y, z.
template <int M, class IdxF>
__device__ __forceinline__ void normal_from_regs(const float *__restrict__ x,
                                                 const float *__restrict__ y,
                                                 const float *__restrict__ z, IdxF idx,
                                                 bool div_centroid, int iters, float qx, float qy,
                                                 float qz, float vpx, float vpy, float vpz,
                                                 float &nx, float &ny, float &nz) {
  float px[M], py[M], pz[M];
#pragma unroll
  for (int t = 0; t < M; ++t) {
    const int j = idx(t);
    px[t] = __ldg(&x[j]);
    py[t] = __ldg(&y[j]);
    pz[t] = __ldg(&z[j]);
  }
  normal_from_coords<M>(px, py, pz, div_centroid, iters, qx, qy, qz, vpx, vpy, vpz, nx, ny, nz);
}

template <int M>
__device__ __forceinline__ void normal_from_keys(const float *__restrict__ x,
                                                 const float *__restrict__ y,
                                                 const float *__restrict__ z, const u64 (&L)[M],
                                                 bool div_centroid, int iters, float qx, float qy,
                                                 float qz, float vpx, float vpy, float vpz,
                                                 float &nx, float &ny, float &nz) {
  normal_from_regs<M>(x, y, z, [&](int t) { return nbr_idx(L[t]) & 0x7FFFFFFF; }, div_centroid,
                      iters, qx, qy, qz, vpx, vpy, vpz, nx, ny, nz);
}
}  // namespace nd
}  // namespace rvp

namespace rvp {
namespace nd {
// normal_from_list over points: nbr(t) is the t-th neighbour's record
template <class Nbr>
__device__ __forceinline__ void normal_from_points(Nbr nbr, int m, bool div_centroid, int iters,
                                                   float qx, float qy, float qz, float vpx,
                                                   float vpy, float vpz, float &nx, float &ny,
                                                   float &nz) {
  float cx = 0.0f, cy = 0.0f, cz = 0.0f;
  for (int t = 0; t < m; ++t) {
    const float4 p = nbr(t);
    cx = fadd(cx, p.x);
    cy = fadd(cy, p.y);
    cz = fadd(cz, p.z);
  }
  if (div_centroid) {
    const float fm = (float)m;
    cx = fdiv(cx, fm);
    cy = fdiv(cy, fm);
    cz = fdiv(cz, fm);
  } else {
    const float inv_n = fdiv(1.0f, (float)m);
    cx = fmul(cx, inv_n);
    cy = fmul(cy, inv_n);
    cz = fmul(cz, inv_n);
  }
  float c00 = 0, c01 = 0, c02 = 0, c11 = 0, c12 = 0, c22 = 0;
  for (int t = 0; t < m; ++t) {
    const float4 p = nbr(t);
    const float dx = fsub(p.x, cx), dy = fsub(p.y, cy), dz = fsub(p.z, cz);
    c00 = fadd(c00, fmul(dx, dx));
    c01 = fadd(c01, fmul(dx, dy));
    c02 = fadd(c02, fmul(dx, dz));
    c11 = fadd(c11, fmul(dy, dy));
    c12 = fadd(c12, fmul(dy, dz));
    c22 = fadd(c22, fmul(dz, dz));
  }
  float A[3][3] = {{c00, c01, c02}, {c01, c11, c12}, {c02, c12, c22}};
  eigen_smallest_ref(A, iters, nx, ny, nz);
  flip_ref(qx, qy, qz, vpx, vpy, vpz, nx, ny, nz);
}

// ---------------------------------------------------------------------------
// precision path: covariance accumulated in FP32 about the query point
// (differences of nearby points are exact) with compensated (Kahan) sums,
// converged cyclic Jacobi in FP32, and the eigen-solve redone in FP64 only
// when lambda_max / lambda_min exceeds a threshold.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void kahan_add(float &s, float &c, float v) {
  const float y = fsub(v, c);
  const float t = fadd(s, y);
  c = fsub(fsub(t, s), y);
  s = t;
}

template <class T>
__device__ void jacobi_sym3(T A[3][3], T V[3][3], int sweeps) {
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) V[i][j] = (i == j) ? T(1) : T(0);
  for (int sw = 0; sw < sweeps; ++sw) {
    const T off = A[0][1] * A[0][1] + A[0][2] * A[0][2] + A[1][2] * A[1][2];
    const T dia = A[0][0] * A[0][0] + A[1][1] * A[1][1] + A[2][2] * A[2][2];
    if (!(off > (sizeof(T) == 4 ? T(1e-14) : T(1e-30)) * dia)) break;
#pragma unroll
    for (int pq = 0; pq < 3; ++pq) {
      const int p = pq == 2 ? 1 : 0;
      const int q = pq == 0 ? 1 : 2;
      if (A[p][q] == T(0)) continue;
      const T theta = (A[q][q] - A[p][p]) / (T(2) * A[p][q]);
      const T t = (theta >= T(0) ? T(1) : T(-1)) / (fabs(theta) + sqrt(theta * theta + T(1)));
      const T c = T(1) / sqrt(t * t + T(1)), s = t * c;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const T arp = A[r][p], arq = A[r][q];
        A[r][p] = c * arp - s * arq;
        A[r][q] = s * arp + c * arq;
      }
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const T apr = A[p][r], aqr = A[q][r];
        A[p][r] = c * apr - s * aqr;
        A[q][r] = s * apr + c * aqr;
      }
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const T vrp = V[r][p], vrq = V[r][q];
        V[r][p] = c * vrp - s * vrq;
        V[r][q] = s * vrp + c * vrq;
      }
    }
  }
}

// column of the smallest / largest diagonal entry (first of equals)
template <class T>
__device__ __forceinline__ int smallest_diag(const T (&A)[3][3]) {
  int m = 0;
  T d = A[0][0];
  if (A[1][1] < d) { m = 1; d = A[1][1]; }
  if (A[2][2] < d) m = 2;
  return m;
}
template <class T>
__device__ __forceinline__ T pick3(int m, T a, T b, T c) {
  return m == 0 ? a : (m == 1 ? b : c);
}

template <class Nbr>
__device__ __forceinline__ void precise_normal(Nbr nbr, int kk, float qx, float qy, float qz,
                                               float vpx, float vpy, float vpz, double cond_fp64,
                                               float &nx, float &ny, float &nz, float &cond,
                                               bool &wide) {
  // shifted, compensated centroid of (p - q)
  float sx = 0, sy = 0, sz = 0, ex = 0, ey = 0, ez = 0;
#pragma unroll 4
  for (int t = 0; t < kk; ++t) {
    const float4 p = nbr(t);
    kahan_add(sx, ex, fsub(p.x, qx));
    kahan_add(sy, ey, fsub(p.y, qy));
    kahan_add(sz, ez, fsub(p.z, qz));
  }
  const float inv = fdiv(1.0f, (float)kk);
  const float cx = fmul(sx, inv), cy = fmul(sy, inv), cz = fmul(sz, inv);
  float s[6] = {0, 0, 0, 0, 0, 0}, e[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 4
  for (int t = 0; t < kk; ++t) {
    const float4 p = nbr(t);
    const float dx = fsub(fsub(p.x, qx), cx);
    const float dy = fsub(fsub(p.y, qy), cy);
    const float dz = fsub(fsub(p.z, qz), cz);
    kahan_add(s[0], e[0], fmul(dx, dx));
    kahan_add(s[1], e[1], fmul(dx, dy));
    kahan_add(s[2], e[2], fmul(dx, dz));
    kahan_add(s[3], e[3], fmul(dy, dy));
    kahan_add(s[4], e[4], fmul(dy, dz));
    kahan_add(s[5], e[5], fmul(dz, dz));
  }
  float A[3][3] = {{s[0], s[1], s[2]}, {s[1], s[3], s[4]}, {s[2], s[4], s[5]}};
  float V[3][3];
  jacobi_sym3<float>(A, V, 8);
  const int mi = smallest_diag(A);
  const float lo = fabsf(pick3(mi, A[0][0], A[1][1], A[2][2]));
  const float hi = fabsf(A[2][2] > fmaxf(A[0][0], A[1][1])
                             ? A[2][2] : (A[1][1] > A[0][0] ? A[1][1] : A[0][0]));
  const double cnd = lo > 0.0f ? (double)hi / (double)lo : 1e300;
  double ax, ay, az;
  wide = cnd > cond_fp64;
  if (wide) {
    // fold the compensation terms back in
    const double d00 = (double)s[0] - e[0], d01 = (double)s[1] - e[1], d02 = (double)s[2] - e[2],
                 d11 = (double)s[3] - e[3], d12 = (double)s[4] - e[4], d22 = (double)s[5] - e[5];
    double D[3][3] = {{d00, d01, d02}, {d01, d11, d12}, {d02, d12, d22}};
    double W[3][3];
    jacobi_sym3<double>(D, W, 32);
    const int m2 = smallest_diag(D);
    ax = pick3(m2, W[0][0], W[0][1], W[0][2]);
    ay = pick3(m2, W[1][0], W[1][1], W[1][2]);
    az = pick3(m2, W[2][0], W[2][1], W[2][2]);
  } else {
    ax = pick3(mi, V[0][0], V[0][1], V[0][2]);
    ay = pick3(mi, V[1][0], V[1][1], V[1][2]);
    az = pick3(mi, V[2][0], V[2][1], V[2][2]);
  }
  const double nr = sqrt(ax * ax + ay * ay + az * az);
  ax /= nr; ay /= nr; az /= nr;
  const double dot = ((double)vpx - qx) * ax + ((double)vpy - qy) * ay + ((double)vpz - qz) * az;
  if (dot < 0) { ax = -ax; ay = -ay; az = -az; }
  nx = (float)ax;
  ny = (float)ay;
  nz = (float)az;
  cond = (float)cnd;
}
}  // namespace nd
}  // namespace rvp
