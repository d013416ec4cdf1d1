// C ABI of rvpoint_b200 (include/rvpoint_b200.h): host/device staging,
// status codes and the orchestration of the kernels for each reference
// entry point.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <new>

#include "internal.cuh"

using rvp::u32;
using rvp::u64;

// ---------------------------------------------------------------------------
// buffers
// ---------------------------------------------------------------------------
namespace rvp {
// Every device and pinned allocation of the library goes through DevBuf /
// HostBuf: the live byte counts are kept here, and a test hook
// (rvp_debug_fail_allocation) can make the allocations after the next n
// fail as an out-of-memory would.
namespace {
std::atomic<long long> g_live_device{0}, g_live_pinned{0};
std::atomic<long long> g_fail_after{-1};  // < 0: off

void check_injected_failure() {
  long long left = g_fail_after.load();
  while (left >= 0) {
    if (left == 0) throw Error{RVP_ERR_OOM, "allocation failed (injected by rvp_debug_fail_allocation)"};
    if (g_fail_after.compare_exchange_weak(left, left - 1)) return;
  }
}
}  // namespace

void DevBuf::reserve(size_t b) {
  if (b <= bytes && ptr) return;
  release();
  if (b == 0) b = 256;
  check_injected_failure();
  RVP_CUDA_TRY(cudaMalloc(&ptr, b));
  bytes = b;
  g_live_device += (long long)b;
}
void DevBuf::release() {
  if (ptr) {
    cudaFree(ptr);
    g_live_device -= (long long)bytes;
  }
  ptr = nullptr;
  bytes = 0;
}
void HostBuf::reserve(size_t b) {
  if (b <= bytes && ptr) return;
  release();
  if (b == 0) b = 256;
  check_injected_failure();
  RVP_CUDA_TRY(cudaMallocHost(&ptr, b));
  bytes = b;
  g_live_pinned += (long long)b;
}
void HostBuf::release() {
  if (ptr) {
    cudaFreeHost(ptr);
    g_live_pinned -= (long long)bytes;
  }
  ptr = nullptr;
  bytes = 0;
}
}  // namespace rvp

extern "C" {
rvp_status rvp_debug_fail_allocation(long long after) {
  rvp::g_fail_after = after < 0 ? -1 : after;
  return RVP_OK;
}

rvp_status rvp_debug_live_bytes(long long *device_bytes, long long *pinned_bytes) {
  if (device_bytes) *device_bytes = rvp::g_live_device.load();
  if (pinned_bytes) *pinned_bytes = rvp::g_live_pinned.load();
  return RVP_OK;
}
}

struct rvp_hash {
  rvp_context *ctx = nullptr;
  rvp::DevBuf x, y, z, offs;
  size_t n = 0;
  float cell = 0.0f;
  long long p1 = 73856093LL, p2 = 19349663LL;
  rvp::Grid grid;     // the reference's buckets, where cells may share a key
  rvp::KnnTree tree;  // searched unless cells share a key
  rvp::TreeView tree_view{};
  bool has_cloud = false, built = false, tree_built = false;
  int collision = 0;
};

namespace {

template <class F>
rvp_status guard(rvp_context *ctx, F &&f) {
  try {
    f();
    return RVP_OK;
  } catch (const rvp::Error &e) {
    if (ctx) ctx->last_error = e.msg;
    return e.status;
  } catch (const std::bad_alloc &) {
    if (ctx) ctx->last_error = "host allocation failed";
    return RVP_ERR_OOM;
  } catch (...) {
    if (ctx) ctx->last_error = "unknown error";
    return RVP_ERR_CUDA;
  }
}

void set_device(rvp_context *ctx) { RVP_CUDA_TRY(cudaSetDevice(ctx->device)); }

void *scratch(rvp_context *ctx, int slot, size_t bytes) {
  ctx->scratch[slot].reserve(bytes);
  return ctx->scratch[slot].ptr;
}

// input: device pointer as is, or a staged copy of the host array
template <class T>
const T *in_dev(rvp_context *ctx, int slot, const T *p, size_t n, int mem) {
  if (mem == RVP_MEM_DEVICE || n == 0) return p;
  T *d = static_cast<T *>(scratch(ctx, slot, n * sizeof(T)));
  RVP_CUDA_TRY(cudaMemcpyAsync(d, p, n * sizeof(T), cudaMemcpyHostToDevice, ctx->stream));
  return d;
}

template <class T>
T *out_dev(rvp_context *ctx, int slot, T *p, size_t n, int mem) {
  if (p == nullptr) return nullptr;
  if (mem == RVP_MEM_DEVICE) return p;
  return static_cast<T *>(scratch(ctx, slot, (n ? n : 1) * sizeof(T)));
}

template <class T>
void out_copy(rvp_context *ctx, T *user, const T *dev, size_t n, int mem) {
  if (user == nullptr || mem == RVP_MEM_DEVICE || n == 0) return;
  RVP_CUDA_TRY(cudaMemcpyAsync(user, dev, n * sizeof(T), cudaMemcpyDeviceToHost, ctx->stream));
}

// memory of the context's own GPU
bool on_device(rvp_context *ctx, const void *p) {
  cudaPointerAttributes a{};
  RVP_CUDA_TRY(cudaPointerGetAttributes(&a, p));
  return a.type == cudaMemoryTypeDevice && a.device == ctx->device;
}

void sync(rvp_context *ctx) { RVP_CUDA_TRY(cudaStreamSynchronize(ctx->stream)); }

template <class T>
T read_back(rvp_context *ctx, const T *dev) {
  T v;
  RVP_CUDA_TRY(cudaMemcpyAsync(&v, dev, sizeof(T), cudaMemcpyDeviceToHost, ctx->stream));
  sync(ctx);
  return v;
}

// [0, n] on the device: a single frame
int64_t *single_frame_offsets(rvp_context *ctx, int slot, size_t n) {
  int64_t h[2] = {0, (int64_t)n};
  int64_t *d = static_cast<int64_t *>(scratch(ctx, slot, 16));
  RVP_CUDA_TRY(cudaMemcpyAsync(d, h, 16, cudaMemcpyHostToDevice, ctx->stream));
  sync(ctx);  // h lives on this stack frame
  return d;
}

__global__ void k_pack(const int32_t *idx, const float *d2, size_t total, u64 *pairs) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x)
    pairs[i] = rvp::pack_nbr(d2[i], idx[i]);
}

__global__ void k_scatter3(const float *x, const float *y, const float *z, const u32 *to, size_t n,
                           float *ox, float *oy, float *oz) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    ox[to[i]] = x[i];
    oy[to[i]] = y[i];
    oz[to[i]] = z[i];
  }
}

__global__ void k_copy3(const float *x, const float *y, const float *z, size_t n, float *ox,
                        float *oy, float *oz) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    ox[i] = x[i];
    oy[i] = y[i];
    oz[i] = z[i];
  }
}

__global__ void k_unpack(const u64 *pairs, size_t total, int32_t *idx, float *d2) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const u64 k = pairs[i];
    if (idx) idx[i] = (int32_t)(u32)(k & 0x7FFFFFFFull);
    if (d2) d2[i] = __uint_as_float((u32)(k >> 32));
  }
}

// fixed-stride rows (nq x K, counts[q] valid) -> CSR rows
__global__ void k_rows_to_csr(const int32_t *row_idx, const float *row_d2, int K,
                              const int32_t *counts, const u64 *offs, size_t nq, int32_t *idx,
                              float *d2) {
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nq * (size_t)K;
       t += (size_t)gridDim.x * blockDim.x) {
    const size_t q = t / K;
    const int j = (int)(t % K);
    if (j >= counts[q]) continue;
    const u64 o = offs[q] + j;
    if (idx) idx[o] = row_idx[t];
    if (d2) d2[o] = row_d2[t];
  }
}

// CSR rows cut to at most `cut` entries
__global__ void k_csr_cut(const u64 *pairs, const u64 *offs_in, const u64 *offs_out, size_t nq,
                          int32_t *idx, float *d2) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < nq;
       q += (size_t)gridDim.x * blockDim.x) {
    const u64 a = offs_in[q], o = offs_out[q], c = offs_out[q + 1] - o;
    for (u64 j = 0; j < c; ++j) {
      const u64 k = pairs[a + j];
      if (idx) idx[o + j] = (int32_t)(u32)(k & 0x7FFFFFFFull);
      if (d2) d2[o + j] = __uint_as_float((u32)(k >> 32));
    }
  }
}

__global__ void k_min_counts(const u32 *in, size_t n, u32 cut, u32 *out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = in[i] < cut ? in[i] : cut;
}

__global__ void k_i32_to_u32(const int32_t *in, size_t n, u32 *out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = (u32)max(in[i], 0);
}

// one scratch tree per context, kept across calls so its buffers are reused
rvp::KnnTree &ctx_tree(rvp_context *ctx) {
  if (!ctx->tree) ctx->tree = new rvp::KnnTree();
  return *ctx->tree;
}

// the k nearest of every point of a device cloud
void knn_cloud(rvp_context *ctx, const float *x, const float *y, const float *z, size_t n, int K,
               int mode, const rvp::TreeOut &o) {
  rvp::KnnTree &w = ctx_tree(ctx);
  const rvp::TreeView t = rvp::tree_build(ctx, w, x, y, z, n);
  rvp::TreeOut out = o;
  if (mode == rvp::TREE_PRECISE) {
    const u32 packets = (u32)((n + 31) / 32);
    w.rows.reserve((size_t)rvp::tree_precise_packets(packets, K) * K * 128);
    out.rows = w.rows.as<u32>();
  }
  rvp::tree_knn(ctx, t, rvp::tree_queries(ctx, w, t, x, y, z, x, y, z, n), K, 0.0f, mode, out);
}

// the tree over a hash's points (kept until it takes another cloud)
void hash_tree(rvp_hash *h) {
  if (h->tree_built) return;
  h->tree_view = rvp::tree_build(h->ctx, h->tree, h->x.as<float>(), h->y.as<float>(),
                                 h->z.as<float>(), h->n);
  h->tree_built = true;
}

// (32-bit query numbers in the tree's kernels: a billion queries at a time)
constexpr size_t kMostQueries = (size_t)1 << 30;

// the k nearest among a hash's points
void knn_hash(rvp_hash *h, const float *qx, const float *qy, const float *qz, size_t nq, int K,
              float radius, int mode, const rvp::TreeOut &o) {
  const float *x = h->x.as<float>(), *y = h->y.as<float>(), *z = h->z.as<float>();
  hash_tree(h);
  for (size_t a = 0; a < nq; a += kMostQueries) {
    const size_t m = std::min(kMostQueries, nq - a);
    rvp::TreeOut p = o;
    if (p.mean) p.mean += a;
    if (p.idx) p.idx += a * K;
    if (p.d2) p.d2 += a * K;
    if (p.counts) p.counts += a;
    rvp::TreeQueries q{};
    if (rvp::tree_knn_few(m, radius)) {
      q.n = (u32)m;
      q.each[0] = qx + a;
      q.each[1] = qy + a;
      q.each[2] = qz + a;
    } else {
      q = rvp::tree_queries(h->ctx, h->tree, h->tree_view, x, y, z, qx + a, qy + a, qz + a, m);
    }
    rvp::tree_knn(h->ctx, h->tree_view, q, K, radius, mode, p);
  }
}

// one scratch grid per context, kept across calls so its buffers are reused
rvp::Grid &ctx_grid(rvp_context *ctx) {
  if (!ctx->grid) ctx->grid = new rvp::Grid();
  return *ctx->grid;
}

}  // namespace

// ===========================================================================
// context
// ===========================================================================
extern "C" {

const char *rvp_version(void) { return "rvpoint_b200 0.1 (sm_100a)"; }

const char *rvp_status_string(rvp_status s) {
  switch (s) {
    case RVP_OK: return "ok";
    case RVP_ERR_INVALID_ARG: return "invalid argument";
    case RVP_ERR_OOM: return "out of memory";
    case RVP_ERR_CAPACITY: return "output capacity too small";
    case RVP_ERR_TIMEOUT: return "device wait timed out";
    case RVP_ERR_CUDA: return "CUDA error";
    case RVP_ERR_NO_DEVICE: return "no CUDA device";
  }
  return "unknown status";
}

rvp_status rvp_context_create(int device, rvp_context **out) {
  if (!out) return RVP_ERR_INVALID_ARG;
  *out = nullptr;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
    cudaGetLastError();
    return RVP_ERR_NO_DEVICE;
  }
  if (device < 0 || device >= count) return RVP_ERR_INVALID_ARG;
  rvp_context *ctx = new (std::nothrow) rvp_context();
  if (!ctx) return RVP_ERR_OOM;
  ctx->device = device;
  rvp_status s = guard(ctx, [&] {
    set_device(ctx);
    RVP_CUDA_TRY(cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, device));
  });
  if (s != RVP_OK) {
    delete ctx;
    return s;
  }
  *out = ctx;
  return RVP_OK;
}

rvp_status rvp_context_destroy(rvp_context *ctx) {
  if (!ctx) return RVP_ERR_INVALID_ARG;
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  for (auto &b : ctx->scratch) b.release();
  for (auto &b : ctx->pinned) b.release();
  ctx->rand_table.release();
  if (ctx->grid) {
    ctx->grid->release();
    delete ctx->grid;
  }
  if (ctx->tree) {
    ctx->tree->release();
    delete ctx->tree;
  }
  if (ctx->vwork) {
    ctx->vwork->release();
    delete ctx->vwork;
  }
  delete ctx;
  return RVP_OK;
}

rvp_status rvp_context_set_stream(rvp_context *ctx, void *stream) {
  if (!ctx) return RVP_ERR_INVALID_ARG;
  ctx->stream = static_cast<cudaStream_t>(stream);
  return RVP_OK;
}

rvp_status rvp_context_synchronize(rvp_context *ctx) {
  if (!ctx) return RVP_ERR_INVALID_ARG;
  return guard(ctx, [&] { set_device(ctx); sync(ctx); });
}

const char *rvp_last_error(const rvp_context *ctx) { return ctx ? ctx->last_error.c_str() : ""; }

uint64_t rvp_context_launch_count(const rvp_context *ctx) { return ctx ? ctx->launches : 0; }

// ===========================================================================
// SpatialHash
// ===========================================================================
rvp_status rvp_hash_create(rvp_context *ctx, rvp_hash **out) {
  if (!ctx || !out) return RVP_ERR_INVALID_ARG;
  rvp_hash *h = new (std::nothrow) rvp_hash();
  if (!h) return RVP_ERR_OOM;
  h->ctx = ctx;
  *out = h;
  return RVP_OK;
}

rvp_status rvp_hash_destroy(rvp_hash *h) {
  if (!h) return RVP_ERR_INVALID_ARG;
  cudaSetDevice(h->ctx->device);
  cudaStreamSynchronize(h->ctx->stream);
  h->x.release(); h->y.release(); h->z.release(); h->offs.release();
  h->grid.release();
  h->tree.release();
  delete h;
  return RVP_OK;
}

rvp_status rvp_hash_set_primes(rvp_hash *h, int64_t p1, int64_t p2) {
  if (!h) return RVP_ERR_INVALID_ARG;
  h->p1 = p1;
  h->p2 = p2;
  h->built = false;
  return RVP_OK;
}

rvp_status rvp_hash_set_input_cloud(rvp_hash *h, const float *x, const float *y, const float *z,
                                    size_t n, float cell_size, int mem) {
  if (!h) return RVP_ERR_INVALID_ARG;
  rvp_context *ctx = h->ctx;
  return guard(ctx, [&] {
    RVP_REQUIRE(n == 0 || (x && y && z), "null cloud pointer");
    RVP_REQUIRE(n < 0x7FFFFFFFull, "clouds are limited to 2^31 - 1 points");
    RVP_REQUIRE(cell_size > 0.0f && isfinite(cell_size), "cell_size must be > 0");
    set_device(ctx);
    // no cloud until this call has completed (a failed allocation below
    // leaves the hash without one, not with the previous cloud's size)
    h->has_cloud = false;
    h->built = false;
    h->tree_built = false;
    h->n = 0;
    h->x.reserve(n * 4 + 16); h->y.reserve(n * 4 + 16); h->z.reserve(n * 4 + 16);
    if (n && mem == RVP_MEM_DEVICE && on_device(ctx, x) && on_device(ctx, y) &&
        on_device(ctx, z)) {
      k_copy3<<<rvp::grid_for(n, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(
          x, y, z, n, h->x.as<float>(), h->y.as<float>(), h->z.as<float>());
      RVP_LAUNCH_CHECK(ctx);
    } else if (n) {  // (another GPU's memory: a kernel here may not read it)
      const cudaMemcpyKind k =
          mem == RVP_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
      RVP_CUDA_TRY(cudaMemcpyAsync(h->x.ptr, x, n * 4, k, ctx->stream));
      RVP_CUDA_TRY(cudaMemcpyAsync(h->y.ptr, y, n * 4, k, ctx->stream));
      RVP_CUDA_TRY(cudaMemcpyAsync(h->z.ptr, z, n * 4, k, ctx->stream));
    }
    sync(ctx);
    h->n = n;
    h->cell = cell_size;
    h->has_cloud = true;
    h->built = false;
  });
}

rvp_status rvp_hash_build(rvp_hash *h) {
  if (!h) return RVP_ERR_INVALID_ARG;
  rvp_context *ctx = h->ctx;
  return guard(ctx, [&] {
    RVP_REQUIRE(h->has_cloud, "setInputCloud before build");
    set_device(ctx);
    h->built = false;  // set again only when this build has completed
    h->collision = 0;
    if (h->n > 0) {
      hash_tree(h);
      int *flag = static_cast<int *>(scratch(ctx, 4, 256));
      rvp::hash_collision_check(ctx, h->tree_view, h->cell, h->p1, h->p2, flag);
      if (read_back(ctx, flag)) {
        // cells may share a key: the reference's own buckets tell whether
        // occupied ones do (and are searched if so)
        h->offs.reserve(16);
        const int64_t o[2] = {0, (int64_t)h->n};
        RVP_CUDA_TRY(cudaMemcpyAsync(h->offs.ptr, o, 16, cudaMemcpyHostToDevice, ctx->stream));
        rvp::grid_build(ctx, h->grid, h->x.as<float>(), h->y.as<float>(), h->z.as<float>(),
                        h->offs.as<int64_t>(), 1, h->n, h->cell, rvp::KEY_REF_HASH, h->p1, h->p2,
                        nullptr);
        h->collision = read_back(ctx, h->grid.d_collision);
      }
    }
    h->built = true;
  });
}

rvp_status rvp_hash_has_collisions(rvp_hash *h, int *out) {
  if (!h || !out) return RVP_ERR_INVALID_ARG;
  *out = h->collision;
  return RVP_OK;
}

}  // extern "C"

// outputs(total, &indices, &dists): where the caller wants them; false: nowhere
// (the search then ends with the offsets and the total)
template <class Outputs>
static void radius_search(rvp_hash *h, const float *qx, const float *qy, const float *qz,
                          size_t nq, float radius, int max_nn, int mem, int64_t *offsets,
                          size_t *total, Outputs &&outputs) {
  rvp_context *ctx = h->ctx;
  RVP_REQUIRE(h->built, "build before radiusSearch");
  RVP_REQUIRE(offsets && total, "offsets/total required");
  RVP_REQUIRE(nq == 0 || (qx && qy && qz), "null query pointer");
  set_device(ctx);
  *total = 0;
  RVP_REQUIRE(radius >= 0.0f, "radius must be >= 0");
  u64 *offs_d = reinterpret_cast<u64 *>(out_dev(ctx, 0, offsets, nq + 1, mem));
  int32_t *indices = nullptr;
  float *dists = nullptr;
  if (nq == 0 || h->n == 0) {
    RVP_CUDA_TRY(cudaMemsetAsync(offs_d, 0, (nq + 1) * 8, ctx->stream));
    out_copy(ctx, offsets, reinterpret_cast<int64_t *>(offs_d), nq + 1, mem);
    sync(ctx);
    outputs(0, &indices, &dists);
    return;
  }
  const float *dqx = in_dev(ctx, 1, qx, nq, mem);
  const float *dqy = in_dev(ctx, 2, qy, nq, mem);
  const float *dqz = in_dev(ctx, 3, qz, nq, mem);
  const bool refwin = h->collision != 0;
  void *scan_tmp = scratch(ctx, 4, rvp::scan_temp_bytes(nq + 1));
  auto finish = [&](size_t tot) {
    out_copy(ctx, offsets, reinterpret_cast<int64_t *>(offs_d), nq + 1, mem);
    out_copy(ctx, indices, static_cast<int32_t *>(ctx->scratch[8].ptr), tot, mem);
    out_copy(ctx, dists, static_cast<float *>(ctx->scratch[9].ptr), tot, mem);
    sync(ctx);
  };
  if (max_nn > 0 && max_nn <= 64 && !refwin) {
    const int K = max_nn;
    rvp::TreeOut o;
    o.idx = static_cast<int32_t *>(scratch(ctx, 5, nq * (size_t)K * 8));
    o.d2 = reinterpret_cast<float *>(o.idx + nq * (size_t)K);
    int32_t *cnt = o.counts = static_cast<int32_t *>(scratch(ctx, 6, nq * 4));
    knn_hash(h, dqx, dqy, dqz, nq, K, radius, rvp::TREE_PAIRS, o);
    u32 *ucnt = static_cast<u32 *>(scratch(ctx, 7, nq * 4));
    k_i32_to_u32<<<rvp::grid_for(nq, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(cnt, nq, ucnt);
    RVP_LAUNCH_CHECK(ctx);
    rvp::exclusive_scan_u32_to_u64(ctx, ucnt, offs_d, nq, nullptr, scan_tmp);
    const u64 tot = read_back(ctx, offs_d + nq);
    *total = (size_t)tot;
    if (!outputs((size_t)tot, &indices, &dists)) return finish(0);
    int32_t *di = out_dev(ctx, 8, indices, tot, mem);
    float *dd = out_dev(ctx, 9, dists, tot, mem);
    k_rows_to_csr<<<rvp::grid_for(nq * K, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(
        o.idx, o.d2, K, cnt, offs_d, nq, di, dd);
    RVP_LAUNCH_CHECK(ctx);
    return finish(tot);
  }
  // the lists' lengths, their offsets, and the lists (cut: the offsets of the
  // cut ones beside the full ones)
  rvp::QuerySet qs{dqx, dqy, dqz, nq, nullptr, nullptr, nullptr};
  const rvp::GridView gv = refwin ? h->grid.view(rvp::KEY_REF_HASH, h->p1, h->p2)
                                  : rvp::GridView{};
  u32 *cnt = static_cast<u32 *>(scratch(ctx, 6, nq * 4 + 256));
  u64 *full = max_nn > 0 ? static_cast<u64 *>(scratch(ctx, 10, (nq + 2) * 8)) : offs_d;
  u32 *most_d = cnt + nq;
  u32 most[2] = {0, 0};
  // counts of the m queries from a on
  auto count = [&](size_t a, size_t m) {
    rvp::TreeQueries tq{};
    if (rvp::tree_radius_few(m)) tq = rvp::tree_queries_as_given(ctx, h->tree, m);
    else
      tq = rvp::tree_queries(ctx, h->tree, h->tree_view, h->x.as<float>(), h->y.as<float>(),
                             h->z.as<float>(), dqx + a, dqy + a, dqz + a, m);
    rvp::tree_radius_count(ctx, h->tree_view, tq, dqx + a, dqy + a, dqz + a, radius, cnt + a,
                           most_d);
    return tq;
  };
  rvp::TreeQueries tq{};
  if (!refwin)
    for (size_t a = 0; a < nq; a += kMostQueries)
      tq = count(a, std::min(kMostQueries, nq - a));
  else
    rvp::grid_radius_count(ctx, gv, qs, radius, refwin, cnt);
  rvp::exclusive_scan_u32_to_u64(ctx, cnt, full, nq, nullptr, scan_tmp);
  u64 tot = 0;
  if (max_nn > 0) {
    u32 *ccut = static_cast<u32 *>(scratch(ctx, 7, nq * 4));
    k_min_counts<<<rvp::grid_for(nq, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(
        cnt, nq, (u32)max_nn, ccut);
    RVP_LAUNCH_CHECK(ctx);
    rvp::exclusive_scan_u32_to_u64(ctx, ccut, offs_d, nq, nullptr, scan_tmp);
    RVP_CUDA_TRY(cudaMemcpyAsync(&tot, offs_d + nq, 8, cudaMemcpyDeviceToHost, ctx->stream));
  }
  u64 tot_full = 0;
  RVP_CUDA_TRY(cudaMemcpyAsync(&tot_full, full + nq, 8, cudaMemcpyDeviceToHost, ctx->stream));
  if (!refwin)
    RVP_CUDA_TRY(cudaMemcpyAsync(most, most_d, 8, cudaMemcpyDeviceToHost, ctx->stream));
  sync(ctx);
  if (max_nn <= 0) tot = tot_full;
  *total = (size_t)tot;
  if (!outputs((size_t)tot, &indices, &dists)) return finish(0);
  int32_t *di = out_dev(ctx, 8, indices, tot, mem);
  float *dd = out_dev(ctx, 9, dists, tot, mem);
  const u32 cut = max_nn > 0 ? (u32)max_nn : 0;
  if (!refwin) {
    for (size_t a = 0; a < nq; a += kMostQueries) {
      const size_t m = std::min(kMostQueries, nq - a);
      if (nq > kMostQueries) {  // (the part's queries and long lists once more)
        tq = count(a, m);
        RVP_CUDA_TRY(cudaMemcpyAsync(most, most_d, 8, cudaMemcpyDeviceToHost, ctx->stream));
        sync(ctx);
      }
      const bool big = most[0] > rvp::tree_radius_cap();
      u64 *pairs = big ? static_cast<u64 *>(scratch(ctx, 5, tot_full * 8)) : nullptr;
      u32 *list = big ? static_cast<u32 *>(scratch(ctx, 11, m * 4 + 16)) : nullptr;
      rvp::tree_radius_fill(ctx, h->tree_view, tq, dqx + a, dqy + a, dqz + a, radius, full + a,
                            offs_d + a, cut, most[1], di, dd, pairs, list,
                            big ? list + m : nullptr);
    }
    return finish(tot);
  }
  u64 *pairs = static_cast<u64 *>(scratch(ctx, 5, (tot_full ? tot_full : 1) * 8));
  u32 *big = static_cast<u32 *>(scratch(ctx, 11, nq * 4 + 16));
  u32 *big_count = big + nq;
  rvp::grid_radius_fill(ctx, gv, qs, radius, refwin, full, 0, pairs, big, big_count);
  rvp::sort_big_segments(ctx, full, pairs, big, big_count, (u32)std::min<size_t>(nq, 4096));
  if (max_nn > 0) {
    k_csr_cut<<<rvp::grid_for(nq, 128, ctx->num_sms * 16), 128, 0, ctx->stream>>>(
        pairs, full, offs_d, nq, di, dd);
  } else {
    k_unpack<<<rvp::grid_for(tot, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(pairs, tot, di, dd);
  }
  RVP_LAUNCH_CHECK(ctx);
  finish(tot);
}

extern "C" {
rvp_status rvp_hash_radius_search(rvp_hash *h, const float *qx, const float *qy, const float *qz,
                                  size_t nq, float radius, int max_nn, int mem, int64_t *offsets,
                                  int32_t *indices, float *dists, size_t capacity, size_t *total) {
  if (!h) return RVP_ERR_INVALID_ARG;
  bool fits = true;
  rvp_status s = guard(h->ctx, [&] {
    radius_search(h, qx, qy, qz, nq, radius, max_nn, mem, offsets, total,
                  [&](size_t tot, int32_t **i, float **d) {
                    fits = tot <= capacity;
                    *i = indices;
                    *d = dists;
                    return fits;
                  });
  });
  if (s == RVP_OK && !fits) {
    h->ctx->last_error = "radius search: output capacity too small";
    return RVP_ERR_CAPACITY;
  }
  return s;
}

rvp_status rvp_hash_radius_search_alloc(rvp_hash *h, const float *qx, const float *qy,
                                        const float *qz, size_t nq, float radius, int max_nn,
                                        int mem, int64_t *offsets, rvp_alloc_fn alloc, void *user,
                                        size_t *total) {
  if (!h || !alloc) return RVP_ERR_INVALID_ARG;
  return guard(h->ctx, [&] {
    radius_search(h, qx, qy, qz, nq, radius, max_nn, mem, offsets, total,
                  [&](size_t tot, int32_t **i, float **d) {
                    if (alloc(user, tot, i, d) != 0 || (tot && (!*i || !*d)))
                      throw rvp::Error{RVP_ERR_OOM, "radius search: no memory for the lists"};
                    return true;
                  });
  });
}

rvp_status rvp_hash_knn(rvp_hash *h, const float *qx, const float *qy, const float *qz, size_t nq,
                        int k, float radius, int mem, int32_t *indices, float *dists,
                        int32_t *counts) {
  if (!h) return RVP_ERR_INVALID_ARG;
  rvp_context *ctx = h->ctx;
  return guard(ctx, [&] {
    RVP_REQUIRE(h->built, "build before knn");
    RVP_REQUIRE(k >= 1 && k <= 64, "k must be in [1, 64]");
    RVP_REQUIRE(nq == 0 || (qx && qy && qz), "null query pointer");
    RVP_REQUIRE(h->collision == 0, "knn needs a collision-free hash (change the primes)");
    set_device(ctx);
    if (nq == 0) return;
    int32_t *dc = out_dev(ctx, 6, counts, nq, mem);
    int32_t *di = out_dev(ctx, 8, indices, nq * (size_t)k, mem);
    float *dd = out_dev(ctx, 9, dists, nq * (size_t)k, mem);
    if (h->n == 0) {
      if (dc) RVP_CUDA_TRY(cudaMemsetAsync(dc, 0, nq * 4, ctx->stream));
      if (di) RVP_CUDA_TRY(cudaMemsetAsync(di, 0xFF, nq * (size_t)k * 4, ctx->stream));
      out_copy(ctx, counts, dc, nq, mem);
      out_copy(ctx, indices, di, nq * (size_t)k, mem);
      sync(ctx);
      return;
    }
    const float *dqx = in_dev(ctx, 1, qx, nq, mem);
    const float *dqy = in_dev(ctx, 2, qy, nq, mem);
    const float *dqz = in_dev(ctx, 3, qz, nq, mem);
    rvp::TreeOut o;
    o.idx = di;
    o.d2 = dd;
    o.counts = dc;
    knn_hash(h, dqx, dqy, dqz, nq, k, radius, rvp::TREE_PAIRS, o);
    out_copy(ctx, counts, dc, nq, mem);
    out_copy(ctx, indices, di, nq * (size_t)k, mem);
    out_copy(ctx, dists, dd, nq * (size_t)k, mem);
    sync(ctx);
  });
}

// ===========================================================================
// voxel grid
// ===========================================================================
rvp_status rvp_voxel_grid(rvp_context *ctx, const float *x, const float *y, const float *z,
                          size_t n, float leaf_size, int mem, float *out_aos, int32_t *keys,
                          size_t *out_count) {
  if (!ctx) return RVP_ERR_INVALID_ARG;
  return guard(ctx, [&] {
    RVP_REQUIRE(out_count, "out_count required");
    RVP_REQUIRE(n == 0 || (x && y && z && out_aos), "null pointer");
    RVP_REQUIRE(leaf_size > 0.0f && isfinite(leaf_size), "leaf_size must be > 0");
    RVP_REQUIRE(n < 0x7FFFFFFFull, "clouds are limited to 2^31 - 1 points");
    *out_count = 0;
    if (n == 0) return;  // voxel_grid_downsamp.cpp:185
    set_device(ctx);
    const float *dx = in_dev(ctx, 1, x, n, mem);
    const float *dy = in_dev(ctx, 2, y, n, mem);
    const float *dz = in_dev(ctx, 3, z, n, mem);
    int64_t *offs = single_frame_offsets(ctx, 4, n);
    float *dout = out_dev(ctx, 5, out_aos, 3 * n, mem);
    int32_t *dkeys = out_dev(ctx, 6, keys, 3 * n, mem);
    int64_t *vo = static_cast<int64_t *>(scratch(ctx, 7, 64));
    int *err = reinterpret_cast<int *>(vo + 4);
    if (!ctx->vwork) ctx->vwork = new rvp::VoxelWork();
    const float inv_leaf = 1.0f / leaf_size;  // voxel_grid_downsamp.cpp:189
    rvp::voxel_grid_run(ctx, *ctx->vwork, dx, dy, dz, offs, 1, n, nullptr, inv_leaf, dout, vo, dkeys, err,
                        nullptr, nullptr, nullptr);
    int64_t hv[2];
    int herr = 0;
    RVP_CUDA_TRY(cudaMemcpyAsync(hv, vo, 16, cudaMemcpyDeviceToHost, ctx->stream));
    RVP_CUDA_TRY(cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, ctx->stream));
    sync(ctx);
    RVP_REQUIRE(!herr, "voxel index range does not fit one 64-bit key");
    const size_t v = (size_t)hv[1];
    out_copy(ctx, out_aos, dout, 3 * v, mem);
    out_copy(ctx, keys, dkeys, 3 * v, mem);
    sync(ctx);
    *out_count = v;
  });
}

// ===========================================================================
// SOR
// ===========================================================================
static float *sor_mean_buffer(rvp_context *ctx, float *mean_dists, size_t n, int mem) {
  float *mean = out_dev(ctx, 12, mean_dists, n, mem);
  return mean ? mean : static_cast<float *>(scratch(ctx, 12, n * 4));
}

static void sor_common(rvp_context *ctx, const float *dx, const float *dy, const float *dz,
                       size_t n, float *mean, float alpha, int mem, float *out_aos,
                       size_t *out_count, float *mean_dists, uint8_t *keep) {
  uint8_t *dkeep = out_dev(ctx, 13, keep, n, mem);
  int64_t *offs = single_frame_offsets(ctx, 14, n);
  float *dout = out_dev(ctx, 15, out_aos, 3 * n, mem);
  int64_t *so = static_cast<int64_t *>(scratch(ctx, 16, 64));
  void *tmp = scratch(ctx, 17, rvp::sor_filter_temp_bytes(n, 1));
  rvp::sor_filter_frames(ctx, dx, dy, dz, mean, offs, 1, n, nullptr, alpha, dkeep, dout, so,
                         nullptr, tmp, nullptr, nullptr, nullptr, nullptr);
  int64_t hs[2];
  RVP_CUDA_TRY(cudaMemcpyAsync(hs, so, 16, cudaMemcpyDeviceToHost, ctx->stream));
  sync(ctx);
  const size_t kept = (size_t)hs[1];
  out_copy(ctx, out_aos, dout, 3 * kept, mem);
  out_copy(ctx, mean_dists, mean, n, mem);
  out_copy(ctx, keep, dkeep, n, mem);
  sync(ctx);
  *out_count = kept;
}

rvp_status rvp_sor(rvp_context *ctx, const float *x, const float *y, const float *z, size_t n,
                   int k, float alpha, int mem, float *out_aos, size_t *out_count,
                   float *mean_dists, uint8_t *keep) {
  if (!ctx) return RVP_ERR_INVALID_ARG;
  return guard(ctx, [&] {
    RVP_REQUIRE(out_count, "out_count required");
    *out_count = 0;
    if (n == 0) return;  // statistical_outlier_removal.cpp:70
    RVP_REQUIRE(x && y && z && out_aos, "null pointer");
    RVP_REQUIRE(k >= 1 && k + 1 <= 64, "k must be in [1, 63]");
    RVP_REQUIRE((size_t)k + 1 <= n, "k+1 must not exceed the number of points (the reference reads past its buffer)");
    RVP_REQUIRE(n < 0x7FFFFFFFull, "clouds are limited to 2^31 - 1 points");
    set_device(ctx);
    const float *dx = in_dev(ctx, 1, x, n, mem);
    const float *dy = in_dev(ctx, 2, y, n, mem);
    const float *dz = in_dev(ctx, 3, z, n, mem);
    rvp::TreeOut o;
    o.mean = sor_mean_buffer(ctx, mean_dists, n, mem);
    knn_cloud(ctx, dx, dy, dz, n, k + 1, rvp::TREE_MEAN, o);
    sor_common(ctx, dx, dy, dz, n, o.mean, alpha, mem, out_aos, out_count, mean_dists, keep);
  });
}

rvp_status rvp_sor_spatial_hash(rvp_hash *h, int k, float alpha, float search_radius, int mem,
                                float *out_aos, size_t *out_count, float *mean_dists,
                                uint8_t *keep) {
  if (!h) return RVP_ERR_INVALID_ARG;
  rvp_context *ctx = h->ctx;
  return guard(ctx, [&] {
    RVP_REQUIRE(out_count, "out_count required");
    RVP_REQUIRE(h->built, "build before sor_spatial_hash");
    *out_count = 0;
    const size_t n = h->n;
    if (n == 0) return;
    RVP_REQUIRE(out_aos, "null output");
    RVP_REQUIRE(k >= 1 && k + 1 <= 64, "k must be in [1, 63]");
    RVP_REQUIRE(h->collision == 0, "sor_spatial_hash needs a collision-free hash");
    set_device(ctx);
    const float *dx = h->x.as<float>(), *dy = h->y.as<float>(), *dz = h->z.as<float>();
    rvp::TreeOut o;
    o.mean = sor_mean_buffer(ctx, mean_dists, n, mem);
    o.radius_mode = true;
    o.fallback = search_radius;
    knn_hash(h, dx, dy, dz, n, k + 1, search_radius, rvp::TREE_MEAN, o);
    sor_common(ctx, dx, dy, dz, n, o.mean, alpha, mem, out_aos, out_count, mean_dists, keep);
  });
}

// ===========================================================================
// normals
// ===========================================================================
rvp_status rvp_normals_radius(rvp_hash *h, float radius, float vp_x, float vp_y, float vp_z,
                              int eigen_iters, int mem, float *nx, float *ny, float *nz) {
  if (!h) return RVP_ERR_INVALID_ARG;
  rvp_context *ctx = h->ctx;
  return guard(ctx, [&] {
    RVP_REQUIRE(h->built, "build before normal estimation");
    const size_t n = h->n;
    if (n == 0) return;  // normal_estimation.cpp:193
    RVP_REQUIRE(nx && ny && nz, "null output");
    set_device(ctx);
    const float *dx = h->x.as<float>(), *dy = h->y.as<float>(), *dz = h->z.as<float>();
    float *dnx = out_dev(ctx, 12, nx, n, mem), *dny = out_dev(ctx, 13, ny, n, mem),
          *dnz = out_dev(ctx, 14, nz, n, mem);
    // the points of `list` (or all) from their lists in memory
    auto from_lists = [&](const u32 *list, size_t m) {
      const float *lx = dx, *ly = dy, *lz = dz;
      if (list) {
        float *g = static_cast<float *>(scratch(ctx, 7, m * 12));
        rvp::gather_queries(ctx, dx, dy, dz, list, m, g, g + m, g + 2 * m);
        lx = g;
        ly = g + m;
        lz = g + 2 * m;
      }
      u32 *cnt = static_cast<u32 *>(scratch(ctx, 6, m * 4 + 256));
      u64 *offs = static_cast<u64 *>(scratch(ctx, 10, (m + 1) * 8));
      void *scan_tmp = scratch(ctx, 4, rvp::scan_temp_bytes(m + 1));
      u32 *big = static_cast<u32 *>(scratch(ctx, 11, m * 4 + 16));
      rvp::QuerySet qs{lx, ly, lz, m, nullptr, nullptr, nullptr};
      const rvp::GridView gv = h->grid.view(rvp::KEY_REF_HASH, h->p1, h->p2);
      rvp::TreeQueries tq{};
      if (h->collision) {
        rvp::grid_radius_count(ctx, gv, qs, radius, true, cnt);
      } else {
        tq = rvp::tree_queries(ctx, h->tree, h->tree_view, dx, dy, dz, lx, ly, lz, m);
        rvp::tree_radius_count(ctx, h->tree_view, tq, lx, ly, lz, radius, cnt, cnt + m);
      }
      rvp::exclusive_scan_u32_to_u64(ctx, cnt, offs, m, nullptr, scan_tmp);
      u64 tot = 0;
      u32 most[2] = {0, 0};
      RVP_CUDA_TRY(cudaMemcpyAsync(&tot, offs + m, 8, cudaMemcpyDeviceToHost, ctx->stream));
      RVP_CUDA_TRY(cudaMemcpyAsync(most, cnt + m, 8, cudaMemcpyDeviceToHost, ctx->stream));
      sync(ctx);
      u64 *pairs = static_cast<u64 *>(scratch(ctx, 5, (tot ? tot : 1) * 8));
      if (h->collision) {
        rvp::grid_radius_fill(ctx, gv, qs, radius, true, offs, 0, pairs, big, big + m);
        rvp::sort_big_segments(ctx, offs, pairs, big, big + m, (u32)std::min<size_t>(m, 4096));
      } else {
        u64 *rows = static_cast<u64 *>(scratch(ctx, 8, (tot ? tot : 1) * 8));
        int32_t *ri = reinterpret_cast<int32_t *>(rows);
        float *rd = reinterpret_cast<float *>(ri + tot);
        rvp::tree_radius_fill(ctx, h->tree_view, tq, lx, ly, lz, radius, offs, offs, 0, most[1], ri, rd,
                              pairs, big, big + m);
        k_pack<<<rvp::grid_for(tot, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(ri, rd, tot,
                                                                                  pairs);
        RVP_LAUNCH_CHECK(ctx);
      }
      float *o[3] = {dnx, dny, dnz};
      if (list) {
        float *g = static_cast<float *>(scratch(ctx, 9, m * 12));
        for (int a = 0; a < 3; ++a) o[a] = g + a * m;
      }
      rvp::normals_from_lists(ctx, dx, dy, dz, pairs, offs, nullptr, 0, m, nullptr, false,
                              eigen_iters, vp_x, vp_y, vp_z, lx, ly, lz, o[0], o[1], o[2]);
      if (list) {
        k_scatter3<<<rvp::grid_for(m, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(
            o[0], o[1], o[2], list, m, dnx, dny, dnz);
        RVP_LAUNCH_CHECK(ctx);
      }
    };
    if (h->collision) {
      from_lists(nullptr, n);
    } else {
      u32 *hard = static_cast<u32 *>(scratch(ctx, 15, n * 12 + 16));
      u32 *longer = hard + n, *huge = longer + n;
      u32 *counts = huge + n;
      rvp::tree_radius_normals(ctx, h->tree_view, radius, eigen_iters, vp_x, vp_y, vp_z, dnx, dny,
                               dnz, hard, longer, counts);
      if (read_back(ctx, counts + 1)) {  // (seldom)
        rvp::tree_radius_normals_longer(ctx, h->tree_view, radius, eigen_iters, vp_x, vp_y, vp_z,
                                        dnx, dny, dnz, longer, huge, counts);
        const u32 m = read_back(ctx, counts + 2);
        if (m) from_lists(huge, m);
      }
    }
    out_copy(ctx, nx, dnx, n, mem);
    out_copy(ctx, ny, dny, n, mem);
    out_copy(ctx, nz, dnz, n, mem);
    sync(ctx);
  });
}

rvp_status rvp_normals_knn(rvp_context *ctx, const float *x, const float *y, const float *z,
                           size_t n, int k, float vp_x, float vp_y, float vp_z, int eigen_iters,
                           int mem, float *nx, float *ny, float *nz) {
  if (!ctx) return RVP_ERR_INVALID_ARG;
  return guard(ctx, [&] {
    if (n == 0) return;  // normal_estimation.cpp:75
    RVP_REQUIRE(x && y && z && nx && ny && nz, "null pointer");
    RVP_REQUIRE(k >= 1 && k + 1 <= 64, "k must be in [1, 63]");
    RVP_REQUIRE((size_t)k + 1 <= n, "k+1 must not exceed the number of points");
    set_device(ctx);
    const float *dx = in_dev(ctx, 1, x, n, mem);
    const float *dy = in_dev(ctx, 2, y, n, mem);
    const float *dz = in_dev(ctx, 3, z, n, mem);
    float *dnx = out_dev(ctx, 12, nx, n, mem), *dny = out_dev(ctx, 13, ny, n, mem),
          *dnz = out_dev(ctx, 14, nz, n, mem);
    rvp::TreeOut o;
    o.nx = dnx;
    o.ny = dny;
    o.nz = dnz;
    o.iters = eigen_iters;
    o.vpx = vp_x;
    o.vpy = vp_y;
    o.vpz = vp_z;
    knn_cloud(ctx, dx, dy, dz, n, k + 1, rvp::TREE_NORMALS, o);
    out_copy(ctx, nx, dnx, n, mem);
    out_copy(ctx, ny, dny, n, mem);
    out_copy(ctx, nz, dnz, n, mem);
    sync(ctx);
  });
}

rvp_status rvp_normals_knn_precise(rvp_context *ctx, const float *x, const float *y,
                                   const float *z, size_t n, int k, float vp_x, float vp_y,
                                   float vp_z, double cond_fp64, int mem, float *nx, float *ny,
                                   float *nz, float *cond, uint8_t *used_fp64) {
  if (!ctx) return RVP_ERR_INVALID_ARG;
  return guard(ctx, [&] {
    if (n == 0) return;
    RVP_REQUIRE(x && y && z && nx && ny && nz, "null pointer");
    RVP_REQUIRE(k >= 1 && k + 1 <= 64, "k must be in [1, 63]");
    RVP_REQUIRE((size_t)k + 1 <= n, "k+1 must not exceed the number of points");
    set_device(ctx);
    const float *dx = in_dev(ctx, 1, x, n, mem);
    const float *dy = in_dev(ctx, 2, y, n, mem);
    const float *dz = in_dev(ctx, 3, z, n, mem);
    float *dnx = out_dev(ctx, 12, nx, n, mem), *dny = out_dev(ctx, 13, ny, n, mem),
          *dnz = out_dev(ctx, 14, nz, n, mem);
    float *dc = out_dev(ctx, 15, cond, n, mem);
    uint8_t *du = out_dev(ctx, 16, used_fp64, n, mem);
    rvp::TreeOut o;
    o.nx = dnx;
    o.ny = dny;
    o.nz = dnz;
    o.vpx = vp_x;
    o.vpy = vp_y;
    o.vpz = vp_z;
    o.cond_fp64 = cond_fp64;
    o.cond = dc;
    o.used64 = du;
    knn_cloud(ctx, dx, dy, dz, n, k + 1, rvp::TREE_PRECISE, o);
    out_copy(ctx, nx, dnx, n, mem);
    out_copy(ctx, ny, dny, n, mem);
    out_copy(ctx, nz, dnz, n, mem);
    out_copy(ctx, cond, dc, n, mem);
    out_copy(ctx, used_fp64, du, n, mem);
    sync(ctx);
  });
}

// ===========================================================================
// RANSAC
// ===========================================================================
rvp_status rvp_ransac_plane(rvp_context *ctx, const float *x, const float *y, const float *z,
                            size_t n, float dist_thresh, int max_iters, float collinear_thresh,
                            float probability, const int32_t *rand_stream, int mem, float *model,
                            int *best_count, int *iters_run, int32_t *counts) {
  if (!ctx) return RVP_ERR_INVALID_ARG;
  return guard(ctx, [&] {
    RVP_REQUIRE(model && best_count, "model/best_count required");
    RVP_REQUIRE(max_iters >= 0, "max_iters must be >= 0");
    if (iters_run) *iters_run = 0;
    *best_count = 0;
    if (n < 3) {  // ransac_plane.cpp:59 (no srand, no rand calls)
      return;
    }
    RVP_REQUIRE(x && y && z, "null cloud pointer");
    RVP_REQUIRE(n < 0x7FFFFFFFull, "clouds are limited to 2^31 - 1 points");
    set_device(ctx);
    const float *dx = in_dev(ctx, 1, x, n, mem);
    const float *dy = in_dev(ctx, 2, y, n, mem);
    const float *dz = in_dev(ctx, 3, z, n, mem);
    const size_t R = 3 * (size_t)max_iters;
    const bool own_stream = rand_stream == nullptr;
    int *drand = nullptr;
    if (own_stream) {
      // the reference's srand(0) + rand() sequence, drawn from libc itself
      // once per context: it is the same for every call
      if (ctx->rand_count < R) {
        ctx->rand_count = 0;
        ctx->rand_table.reserve(R * 4 + 16);
        std::vector<int32_t> rs(R);
        srand(0);
        for (size_t i = 0; i < R; ++i) rs[i] = rand();
        RVP_CUDA_TRY(cudaMemcpyAsync(ctx->rand_table.ptr, rs.data(), R * 4,
                                     cudaMemcpyHostToDevice, ctx->stream));
        sync(ctx);
        ctx->rand_count = R;
      }
      drand = ctx->rand_table.as<int>();
    } else {
      drand = static_cast<int *>(scratch(ctx, 4, R * 4 + 16));
      if (R)
        RVP_CUDA_TRY(cudaMemcpyAsync(drand, rand_stream, R * 4,
                                     mem == RVP_MEM_DEVICE ? cudaMemcpyDeviceToDevice
                                                           : cudaMemcpyHostToDevice,
                                     ctx->stream));
    }
    double pc = (double)probability;
    pc = pc < 0.5 ? 0.5 : (pc > 0.9999 ? 0.9999 : pc);
    rvp::RansacParams prm{dist_thresh, max_iters, collinear_thresh, log(1.0 - pc)};
    rvp::RansacState r{};
    if (max_iters > 0 && !counts) {
      rvp::RansacState *dstate = static_cast<rvp::RansacState *>(scratch(ctx, 6, 64));
      rvp::ransac_one(ctx, dx, dy, dz, n, drand, prm, dstate,
                      scratch(ctx, 7, rvp::ransac_one_bytes()));
      RVP_CUDA_TRY(cudaMemcpyAsync(&r, dstate, sizeof(r), cudaMemcpyDeviceToHost, ctx->stream));
    } else if (max_iters > 0) {
      // every hypothesis's count is wanted: none is left out
      int64_t *offs = single_frame_offsets(ctx, 5, n);
      float *dm = static_cast<float *>(scratch(ctx, 6, 64));
      int32_t *db = reinterpret_cast<int32_t *>(dm + 8);
      int32_t *di = db + 2;
      int32_t *dcounts = static_cast<int32_t *>(scratch(ctx, 7, (size_t)max_iters * 4 + 4));
      rvp::ransac_frames(ctx, dx, dy, dz, offs, 1, drand, prm, dm, db, di, dcounts, true,
                         rvp::RansacSampler{}, 8);
      RVP_CUDA_TRY(cudaMemcpyAsync(&r.model, dm, 16, cudaMemcpyDeviceToHost, ctx->stream));
      RVP_CUDA_TRY(cudaMemcpyAsync(&r.best, db, 4, cudaMemcpyDeviceToHost, ctx->stream));
      RVP_CUDA_TRY(cudaMemcpyAsync(&r.iters, di, 4, cudaMemcpyDeviceToHost, ctx->stream));
      RVP_CUDA_TRY(cudaMemcpyAsync(counts, dcounts, (size_t)max_iters * 4,
                                   mem == RVP_MEM_DEVICE ? cudaMemcpyDeviceToDevice
                                                         : cudaMemcpyDeviceToHost,
                                   ctx->stream));
    }
    sync(ctx);
    if (own_stream) {
      // leave libc's generator where the reference leaves it: srand(0) and
      // three rand() calls per executed iteration
      srand(0);
      for (long i = 0; i < 3L * r.iters; ++i) (void)rand();
    }
    memcpy(model, &r.model, 16);
    *best_count = r.best;
    if (iters_run) *iters_run = r.iters;
  });
}

// ===========================================================================
// Euclidean clustering
// ===========================================================================
rvp_status rvp_euclidean_clusters(rvp_context *ctx, const float *x, const float *y,
                                  const float *z, size_t n, float tolerance, int min_size,
                                  int max_size, int mem, int64_t *offsets, int32_t *indices,
                                  size_t *n_clusters) {
  if (!ctx) return RVP_ERR_INVALID_ARG;
  return guard(ctx, [&] {
    RVP_REQUIRE(offsets && n_clusters, "offsets / n_clusters required");
    *n_clusters = 0;
    if (n == 0) {  // euclidean_clustering.cpp:116-118
      if (mem == RVP_MEM_DEVICE) {
        set_device(ctx);
        RVP_CUDA_TRY(cudaMemsetAsync(offsets, 0, 8, ctx->stream));
        sync(ctx);
      } else {
        offsets[0] = 0;
      }
      return;
    }
    RVP_REQUIRE(x && y && z && indices, "null pointer");
    RVP_REQUIRE(tolerance > 0.0f, "tolerance must be > 0");
    RVP_REQUIRE(n < 0x7FFFFFFFull, "clouds are limited to 2^31 - 1 points");
    set_device(ctx);
    const float *dx = in_dev(ctx, 1, x, n, mem);
    const float *dy = in_dev(ctx, 2, y, n, mem);
    const float *dz = in_dev(ctx, 3, z, n, mem);
    int64_t *doffs = out_dev(ctx, 4, offsets, n + 1, mem);
    int32_t *didx = out_dev(ctx, 5, indices, n, mem);
    int64_t *fo = single_frame_offsets(ctx, 6, n);
    u64 *dcount = static_cast<u64 *>(scratch(ctx, 7, 64));
    rvp::euclidean_clusters_run(ctx, ctx_grid(ctx), dx, dy, dz, n, fo, tolerance, min_size,
                                max_size, doffs, didx, dcount,
                                scratch(ctx, 8, rvp::euclidean_temp_bytes(n)));
    u64 k = 0;
    RVP_CUDA_TRY(cudaMemcpyAsync(&k, dcount, 8, cudaMemcpyDeviceToHost, ctx->stream));
    sync(ctx);
    *n_clusters = (size_t)k;
    if (mem != RVP_MEM_DEVICE) {
      out_copy(ctx, offsets, doffs, (size_t)k + 1, mem);
      int64_t total = 0;
      RVP_CUDA_TRY(cudaMemcpyAsync(&total, doffs + k, 8, cudaMemcpyDeviceToHost, ctx->stream));
      sync(ctx);
      out_copy(ctx, indices, didx, (size_t)total, mem);
      sync(ctx);
    }
  });
}

rvp_status rvp_extract_plane(rvp_context *ctx, const float *x, const float *y, const float *z,
                             size_t n, const float *model, float dist_thresh, int mem,
                             float *inliers_aos, float *outliers_aos, size_t *n_inliers,
                             size_t *n_outliers) {
  if (!ctx) return RVP_ERR_INVALID_ARG;
  return guard(ctx, [&] {
    RVP_REQUIRE(model, "model required");
    if (n_inliers) *n_inliers = 0;
    if (n_outliers) *n_outliers = 0;
    if (n == 0) return;
    RVP_REQUIRE(x && y && z, "null cloud pointer");
    set_device(ctx);
    const float *dx = in_dev(ctx, 1, x, n, mem);
    const float *dy = in_dev(ctx, 2, y, n, mem);
    const float *dz = in_dev(ctx, 3, z, n, mem);
    const float *dmod = in_dev(ctx, 4, model, 4, mem);
    float *din = out_dev(ctx, 5, inliers_aos, 3 * n, mem);
    float *dout = out_dev(ctx, 6, outliers_aos, 3 * n, mem);
    u64 *dcnt = static_cast<u64 *>(scratch(ctx, 7, 32));
    rvp::extract_plane_run(ctx, dx, dy, dz, n, dmod, dist_thresh, din, dout, dcnt,
                           scratch(ctx, 8, rvp::extract_temp_bytes(n)));
    u64 hc[2];
    RVP_CUDA_TRY(cudaMemcpyAsync(hc, dcnt, 16, cudaMemcpyDeviceToHost, ctx->stream));
    sync(ctx);
    out_copy(ctx, inliers_aos, din, 3 * hc[0], mem);
    out_copy(ctx, outliers_aos, dout, 3 * hc[1], mem);
    sync(ctx);
    if (n_inliers) *n_inliers = (size_t)hc[0];
    if (n_outliers) *n_outliers = (size_t)hc[1];
  });
}

}  // extern "C"
