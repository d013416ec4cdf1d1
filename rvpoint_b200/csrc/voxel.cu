// Voxel-grid downsampling (voxel_grid_downsamp_sc, voxel_grid_downsamp.cpp
// :183-213, which is what voxel_grid_downsamp_rvv_v2 runs on a non-RISC-V
// host) for many frames at once.
//
//   key     (frame, ix - min_ix, iy - min_iy, iz - min_iz) packed in 64 bits,
//           ix = (int)floor(x * inv_leaf): unsigned order == the reference's
//           std::map<std::tuple<int,int,int>> order within a frame
//   sort    stable radix sort of (key, point index): each voxel becomes a run
//           whose points keep input order
//   reduce  one thread per voxel sums its run sequentially from 0.0f, in
//           input order (bit-identical to the map's running sums), then
//           centroid = sum * (1.0f / count)
#include "internal.cuh"

namespace rvp {

namespace {
inline size_t al(size_t b) { return (b + 255) & ~(size_t)255; }

struct VoxelMeta {  // device scratch
  int shift_x, shift_y, shift_f;
  int error;
};

__device__ __forceinline__ int frame_of_index(const int64_t *offs, int n_frames, size_t i) {
  int lo = 0, hi = n_frames - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((size_t)offs[mid] <= i) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ void voxel_of(float x, float y, float z, float inv, int &vx, int &vy,
                                         int &vz) {
  vx = (int)floorf(fmul(x, inv));
  vy = (int)floorf(fmul(y, inv));
  vz = (int)floorf(fmul(z, inv));
}

__global__ void k_vox_init(int *mm, int n_frames) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < n_frames; f += gridDim.x * blockDim.x) {
    mm[6 * f + 0] = mm[6 * f + 1] = mm[6 * f + 2] = 0x7FFFFFFF;
    mm[6 * f + 3] = mm[6 * f + 4] = mm[6 * f + 5] = (int)0x80000000;
  }
}

// Per-frame voxel-index bounds: one contiguous run of points per block, min /
// max in registers, reduced over the block and flushed with six atomics per
// frame the run touches, at most four blocks per SM (the flushes meet on the
// same six words: with one per warp they were 68 us at 2M points, now 9 us).
constexpr int kMinMaxBlocks = 4;
__global__ __launch_bounds__(256) void k_vox_minmax(const float *__restrict__ x,
                                                    const float *__restrict__ y,
                                                    const float *__restrict__ z,
                                                    const int64_t *offs, int n_frames,
                                                    size_t n_max, const u64 *n_dev, float inv,
                                                    int *mm) {
  __shared__ int part[6][8];
  const size_t n = n_dev ? *n_dev : n_max;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const size_t per = ((n + gridDim.x - 1) / gridDim.x + 255) & ~(size_t)255;
  size_t pos = blockIdx.x * per;
  const size_t e = pos + per < n ? pos + per : n;
  if (pos >= e) return;
  int f = n_frames > 1 ? frame_of_index(offs, n_frames, pos) : 0;
  while (pos < e) {
    while (f + 1 < n_frames && pos >= (size_t)offs[f + 1]) ++f;
    const size_t fe = f + 1 < n_frames ? (size_t)offs[f + 1] : n;
    const size_t seg = fe < e ? fe : e;
    int m[6] = {0x7FFFFFFF, 0x7FFFFFFF, 0x7FFFFFFF,
                (int)0x80000000, (int)0x80000000, (int)0x80000000};
#pragma unroll 4
    for (size_t i = pos + tid; i < seg; i += 256) {
      int vx, vy, vz;
      voxel_of(x[i], y[i], z[i], inv, vx, vy, vz);
      m[0] = min(m[0], vx); m[1] = min(m[1], vy); m[2] = min(m[2], vz);
      m[3] = max(m[3], vx); m[4] = max(m[4], vy); m[5] = max(m[5], vz);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      m[k] = k < 3 ? __reduce_min_sync(0xffffffffu, m[k]) : __reduce_max_sync(0xffffffffu, m[k]);
      if (lane == 0) part[k][wid] = m[k];
    }
    __syncthreads();
    if (tid < 6) {
      int v = part[tid][0];
#pragma unroll
      for (int w = 1; w < 8; ++w) v = tid < 3 ? min(v, part[tid][w]) : max(v, part[tid][w]);
      if (tid < 3) atomicMin(&mm[6 * f + tid], v);
      else atomicMax(&mm[6 * f + tid], v);
    }
    __syncthreads();
    pos = seg;
  }
}

__device__ __forceinline__ int bits_for(unsigned long long r) {
  return r == 0 ? 0 : 64 - __clzll((long long)r);
}

__global__ __launch_bounds__(256) void k_vox_layout(const int *mm, int n_frames,
                                                    VoxelMeta *meta) {
  __shared__ unsigned long long range[3];
  if (threadIdx.x < 3) range[threadIdx.x] = 0;
  __syncthreads();
  unsigned long long r[3] = {0, 0, 0};
  for (int f = threadIdx.x; f < n_frames; f += 256) {
    if (mm[6 * f + 0] > mm[6 * f + 3]) continue;  // empty frame
#pragma unroll
    for (int a = 0; a < 3; ++a)
      r[a] = max(r[a], (unsigned long long)((long long)mm[6 * f + 3 + a] - mm[6 * f + a]));
  }
#pragma unroll
  for (int a = 0; a < 3; ++a)
    if (r[a]) atomicMax(&range[a], r[a]);
  __syncthreads();
  if (threadIdx.x != 0) return;
  const int bx = bits_for(range[0]), by = bits_for(range[1]), bz = bits_for(range[2]);
  const int bf = bits_for((unsigned long long)(n_frames > 0 ? n_frames - 1 : 0));
  meta->shift_y = bz;
  meta->shift_x = bz + by;
  meta->shift_f = bz + by + bx;
  meta->error = (bf + bx + by + bz > 64) ? 1 : 0;
}

// Keys of VK_CHUNK consecutive points per block turn: the frames they can
// belong to are found once per turn (14.5 M points in 256 frames: 87 us; 103
// us with a search over all frames per point and the sort's reading of the
// keys for their bits another 36). bits: for the sort, may be null.
constexpr int VK_CHUNK = 2048;
__global__ __launch_bounds__(256) void k_vox_keys(const float *__restrict__ x,
                                                  const float *__restrict__ y,
                                                  const float *__restrict__ z, const int64_t *offs,
                                                  int n_frames, size_t n_max, const u64 *n_dev,
                                                  float inv, const int *mm, const VoxelMeta *meta,
                                                  u64 *keys, u32 *vals, u64 *bits) {
  __shared__ int s_lo, s_hi;
  const size_t n = n_dev ? *n_dev : n_max;
  const int sx = meta->shift_x, sy = meta->shift_y, sf = meta->shift_f;
  u64 ones = 0, zeros = 0;
  for (size_t base = (size_t)blockIdx.x * VK_CHUNK; base < n;
       base += (size_t)gridDim.x * VK_CHUNK) {
    const size_t end = base + VK_CHUNK < n ? base + VK_CHUNK : n;
    if (n_frames > 1) {
      __syncthreads();
      if (threadIdx.x == 0) s_lo = frame_of_index(offs, n_frames, base);
      if (threadIdx.x == 32) s_hi = frame_of_index(offs, n_frames, end - 1);
      __syncthreads();
    }
    const int flo = n_frames > 1 ? s_lo : 0, fhi = n_frames > 1 ? s_hi : 0;
    for (size_t i = base + threadIdx.x; i < end; i += 256) {
      int f = flo, hi = fhi;
      while (f < hi) {
        const int mid = (f + hi + 1) >> 1;
        if ((size_t)offs[mid] <= i) f = mid; else hi = mid - 1;
      }
      int vx, vy, vz;
      voxel_of(x[i], y[i], z[i], inv, vx, vy, vz);
      const u64 kx = (u64)(unsigned)(vx - mm[6 * f + 0]);
      const u64 ky = (u64)(unsigned)(vy - mm[6 * f + 1]);
      const u64 kz = (u64)(unsigned)(vz - mm[6 * f + 2]);
      const u64 kf = sf >= 64 ? 0 : ((u64)f << sf);
      const u64 k = kf | (sx >= 64 ? 0 : (kx << sx)) | (ky << sy) | kz;
      keys[i] = k;
      vals[i] = (u32)i;
      ones |= k;
      zeros |= ~k;
    }
  }
  if (bits) note_key_bits(ones, zeros, bits);
}

// Voxel heads (a key that differs from the one before) per tile of the sorted
// keys, and after a scan of the tiles' sums the first position of each voxel:
// reads the keys twice (18 us with the scan at 2 M points, 67 us at 14.5 M; a
// flag and a 64-bit rank per point in memory took 27 and 190 us).
constexpr int VH_TH = 256, VH_IT = 8, VH_TILE = VH_TH * VH_IT;
// item j of a thread: a row of the tile's warp, so that loads coalesce
__device__ __forceinline__ size_t vh_index(size_t base, int j) {
  return base + (threadIdx.x >> 5) * (32 * VH_IT) + j * 32 + (threadIdx.x & 31);
}
__device__ __forceinline__ bool vh_head(const u64 *keys, size_t i, size_t n) {
  return i < n && (i == 0 || keys[i] != keys[i - 1]);
}
__global__ __launch_bounds__(VH_TH) void k_vox_heads(const u64 *__restrict__ keys, size_t n_max,
                                                     const u64 *n_dev, u32 *tile_sum) {
  __shared__ u32 sum;
  const size_t n = n_dev ? *n_dev : n_max;
  const size_t base = (size_t)blockIdx.x * VH_TILE;
  if (threadIdx.x == 0) sum = 0;
  __syncthreads();
  u32 c = 0;
#pragma unroll
  for (int j = 0; j < VH_IT; ++j)
    c += __popc(__ballot_sync(0xffffffffu, vh_head(keys, vh_index(base, j), n)));
  if ((threadIdx.x & 31) == 0) atomicAdd(&sum, c);
  __syncthreads();
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = sum;
}

__global__ __launch_bounds__(VH_TH) void k_vox_starts(const u64 *__restrict__ keys, size_t n_max,
                                                      const u64 *n_dev, const u64 *tile_start,
                                                      u32 *vstart) {
  __shared__ u32 warp_sum[VH_TH / 32];
  const size_t n = n_dev ? *n_dev : n_max;
  const size_t base = (size_t)blockIdx.x * VH_TILE;
  if (base >= n) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned m[VH_IT];
  u32 c = 0;
#pragma unroll
  for (int j = 0; j < VH_IT; ++j) {
    m[j] = __ballot_sync(0xffffffffu, vh_head(keys, vh_index(base, j), n));
    c += __popc(m[j]);
  }
  if (lane == 0) warp_sum[w] = c;
  __syncthreads();
  u64 at = tile_start[blockIdx.x];
  for (int q = 0; q < w; ++q) at += warp_sum[q];
#pragma unroll
  for (int j = 0; j < VH_IT; ++j) {
    if ((m[j] >> lane) & 1u)
      vstart[at + __popc(m[j] & ((1u << lane) - 1))] = (u32)vh_index(base, j);
    at += __popc(m[j]);
  }
}

// one thread per voxel: sequential sums in input order, as the map did
__global__ void k_vox_centroids(const float *__restrict__ x, const float *__restrict__ y,
                                const float *__restrict__ z, const u32 *__restrict__ perm,
                                const u32 *__restrict__ vstart, const u64 *n_vox, size_t n_max,
                                const u64 *n_dev, float inv, float *out_aos, float *out_x,
                                float *out_y, float *out_z, int32_t *out_keys,
                                const VoxelMeta *meta) {
  if (meta->error) return;
  const size_t n = n_dev ? *n_dev : n_max;
  const u64 nv = *n_vox;
  for (u64 v = blockIdx.x * (u64)blockDim.x + threadIdx.x; v < nv;
       v += (u64)gridDim.x * blockDim.x) {
    const u32 s = vstart[v];
    const u32 e = (v + 1 < nv) ? vstart[v + 1] : (u32)n;
    float sx = 0.0f, sy = 0.0f, sz = 0.0f;
    for (u32 j = s; j < e; ++j) {
      const u32 p = perm[j];
      sx = fadd(sx, x[p]);
      sy = fadd(sy, y[p]);
      sz = fadd(sz, z[p]);
    }
    const float f = fdiv(1.0f, (float)(int)(e - s));
    const float cx = fmul(sx, f), cy = fmul(sy, f), cz = fmul(sz, f);
    if (out_aos) {
      out_aos[3 * v + 0] = cx;
      out_aos[3 * v + 1] = cy;
      out_aos[3 * v + 2] = cz;
    }
    if (out_x) {
      out_x[v] = cx;
      out_y[v] = cy;
      out_z[v] = cz;
    }
    if (out_keys) {
      const u32 p = perm[s];
      int vx, vy, vz;
      voxel_of(x[p], y[p], z[p], inv, vx, vy, vz);
      out_keys[3 * v + 0] = vx;
      out_keys[3 * v + 1] = vy;
      out_keys[3 * v + 2] = vz;
    }
  }
}

// frames stay contiguous after the sort, so frame f's first voxel is the first
// that starts at or past the frame's first point
__global__ void k_vox_frame_offsets(const int64_t *offs, int n_frames, const u32 *vstart,
                                    const u64 *n_vox, int64_t *out_offsets,
                                    const VoxelMeta *meta) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f <= n_frames;
       f += gridDim.x * blockDim.x) {
    u64 lo = f == n_frames ? *n_vox : 0, hi = f == 0 ? 0 : *n_vox;
    while (lo < hi) {
      const u64 mid = (lo + hi) >> 1;
      if ((int64_t)vstart[mid] < offs[f]) lo = mid + 1; else hi = mid;
    }
    out_offsets[f] = meta->error ? 0 : (int64_t)lo;
  }
}

__global__ void k_vox_error(const VoxelMeta *meta, int *flag) {
  if (threadIdx.x == 0 && blockIdx.x == 0 && flag) *flag = meta->error;
}
}  // namespace

void VoxelWork::reserve(size_t n_max, int nf) {
  if (n_max < 1) n_max = 1;
  if (nf < 1) nf = 1;
  keys.reserve(n_max * 8);
  vals.reserve(n_max * 4);
  sort.reserve(sort_temp_bytes(n_max));
  const size_t tiles = (n_max + VH_TILE - 1) / VH_TILE;
  heads.reserve(al(tiles * 4) + al((tiles + 1) * 8) + al(n_max * 4) + scan_temp_bytes(tiles));
  misc.reserve(al(6 * 4 * (size_t)nf) + al(sizeof(VoxelMeta)));
}

void VoxelWork::release() {
  keys.release(); vals.release(); sort.release(); heads.release(); misc.release();
}

void voxel_grid_run(rvp_context *ctx, VoxelWork &w, const float *x, const float *y,
                    const float *z, const int64_t *offs, int n_frames, size_t n_max,
                    const u64 *n_dev, float inv_leaf, float *out_aos, int64_t *out_offsets,
                    int32_t *out_keys, int *error_flag, float *out_x, float *out_y,
                    float *out_z) {
  w.reserve(n_max, n_frames);
  cudaStream_t st = ctx->stream;
  const int sms = ctx->num_sms;
  int *mm = w.misc.as<int>();
  VoxelMeta *meta = reinterpret_cast<VoxelMeta *>(w.misc.as<char>() + al(6 * 4 * (size_t)n_frames));
  const size_t tiles = (n_max + VH_TILE - 1) / VH_TILE;
  char *hp = w.heads.as<char>();
  u32 *tile_sum = reinterpret_cast<u32 *>(hp); hp += al(tiles * 4);
  u64 *tile_start = reinterpret_cast<u64 *>(hp); hp += al((tiles + 1) * 8);
  u32 *vstart = reinterpret_cast<u32 *>(hp); hp += al(n_max * 4);
  void *scan_tmp = hp;
  const u64 *n_vox = tile_start + tiles;
  SortTemp t;
  sort_temp_carve(t, w.sort.ptr, n_max);

  k_vox_init<<<grid_for(n_frames, 256, 64), 256, 0, st>>>(mm, n_frames);
  RVP_LAUNCH_CHECK(ctx);
  k_vox_minmax<<<grid_for(n_max, 256, sms * kMinMaxBlocks), 256, 0, st>>>(
      x, y, z, offs, n_frames, n_max, n_dev, inv_leaf, mm);
  RVP_LAUNCH_CHECK(ctx);
  k_vox_layout<<<1, 256, 0, st>>>(mm, n_frames, meta);
  RVP_LAUNCH_CHECK(ctx);
  u64 *bits = sort_key_bits(ctx, t, n_max);
  k_vox_keys<<<grid_for(n_max, VK_CHUNK, sms * 8), 256, 0, st>>>(
      x, y, z, offs, n_frames, n_max, n_dev, inv_leaf, mm, meta, w.keys.as<u64>(),
      w.vals.as<u32>(), bits);
  RVP_LAUNCH_CHECK(ctx);
  radix_sort_pairs(ctx, w.keys.as<u64>(), w.vals.as<u32>(), n_max, n_dev, t, bits);
  // (tiles past the live count hold no heads)
  k_vox_heads<<<(unsigned)tiles, VH_TH, 0, st>>>(w.keys.as<u64>(), n_max, n_dev, tile_sum);
  RVP_LAUNCH_CHECK(ctx);
  exclusive_scan_u32_to_u64(ctx, tile_sum, tile_start, tiles, nullptr, scan_tmp);
  k_vox_starts<<<(unsigned)tiles, VH_TH, 0, st>>>(w.keys.as<u64>(), n_max, n_dev, tile_start,
                                                  vstart);
  RVP_LAUNCH_CHECK(ctx);
  k_vox_centroids<<<grid_for(n_max, 256, sms * 16), 256, 0, st>>>(
      x, y, z, w.vals.as<u32>(), vstart, n_vox, n_max, n_dev, inv_leaf, out_aos, out_x, out_y,
      out_z, out_keys, meta);
  RVP_LAUNCH_CHECK(ctx);
  if (out_offsets) {
    k_vox_frame_offsets<<<grid_for(n_frames + 1, 256, 64), 256, 0, st>>>(offs, n_frames, vstart,
                                                                        n_vox, out_offsets, meta);
    RVP_LAUNCH_CHECK(ctx);
  }
  if (error_flag) {
    k_vox_error<<<1, 32, 0, st>>>(meta, error_flag);
    RVP_LAUNCH_CHECK(ctx);
  }
}

}  // namespace rvp
