// Stable LSD radix sort of (u64 key, u32 value) pairs for sm_100a.
//
// Per live 8-bit digit: (1) tile histogram, (2) per-digit scan over tiles,
// (3) tile-local stable ranking with ballots, reorder in shared
// memory, coalesced scatter of each digit run. A digit is live when the keys
// differ in it (some have a one, some a zero there), so a 64-bit key with 30 live
// bits costs 4 passes. The key count and the live mask are read from device
// memory; nothing returns to the host, so a sort can sit in a graph.
//
// Up to kCoopItems keys per SM (606k on 148 SMs) one cooperative kernel runs
// all passes, each block holding its share of the keys in registers
// (k_sort_coop); larger sorts go by tiles, in one cooperative kernel while
// every tile has a block (2.4M keys), else as launches.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "internal.cuh"

namespace rvp {

namespace {
constexpr int TH = 256;
constexpr int ITEMS = 16;
constexpr int TILE = TH * ITEMS;  // 4096 keys per tile
constexpr int WARPS = TH / 32;
constexpr int CHUNK = TILE / WARPS;  // 512 keys per warp, in order

__host__ __device__ inline size_t tiles_for(size_t n) { return (n + TILE - 1) / TILE; }

inline size_t al(size_t b) { return (b + 255) & ~(size_t)255; }

// the bits in which keys differ: some key has a one there, some a zero
__device__ __forceinline__ u64 live_mask(const u64 *bits) {
  return bits[0] & bits[1];
}
__device__ __forceinline__ bool pass_live(u64 live, int pass) {
  return ((live >> (8 * pass)) & 0xFFull) != 0;
}

// the lanes whose digit equals this lane's (digits of `bits` bits), by one
// ballot per bit
template <int BITS>
__device__ __forceinline__ unsigned digit_peers(unsigned d) {
  unsigned m = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < BITS; ++b) {
    const unsigned v = __ballot_sync(0xffffffffu, (d >> b) & 1u);
    m &= (d >> b) & 1u ? v : ~v;
  }
  return m;
}

// buffer holding the input of `pass`: parity of live passes below it
__device__ __forceinline__ int pass_src(u64 live, int pass) {
  int c = 0;
  for (int q = 0; q < pass; ++q) c += pass_live(live, q) ? 1 : 0;
  return c & 1;
}

__global__ void k_key_bits(const u64 *__restrict__ keys, size_t n_max,
                           const u64 *__restrict__ n_dev, u64 *bits) {
  const size_t n = n_dev ? *n_dev : n_max;
  u64 ones = 0, zeros = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const u64 k = keys[i];
    ones |= k;
    zeros |= ~k;
  }
  note_key_bits(ones, zeros, bits);
}

// ---------------------------------------------------------------------------
// any number of keys: tiles of 4096
// ---------------------------------------------------------------------------
// Per live digit: the tiles' histograms; one block per digit scans its row of
// tile counts; the tiles are ranked, reordered in shared memory and written
// out as digit runs. Bound by the ranking's issue and the scattered writes of
// the last step: 14.5M keys 165 us per live digit (200 us with match.any
// ranking and histograms that waited on each row's load). While every tile
// has a block of its own (four per SM), one cooperative kernel runs all steps
// of all digits with grid barriers between them (k_sort_tiles) and a dead
// digit costs nothing: 2M keys 157 us (202 us as launches). Past that the
// steps are launches of their own, whose blocks start as others end: a block
// that walks several tiles is slower (14.5M keys 1259 us against 890 us).
// Keys written by other SMs in the same kernel are read past L1 (__ldcg).
constexpr size_t kTilesSmem = (size_t)TILE * 12 + (size_t)WARPS * 256 * 2 + 256 * 4 * 2;

__device__ __forceinline__ void tile_histogram(const u64 *kin, size_t n, size_t tile, int shift,
                                               u32 (*h)[256], u32 *tile_hist, size_t t_max) {
  const size_t base = tile * TILE;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int q = 0; q < WARPS; ++q) h[q][threadIdx.x] = 0;
  __syncthreads();
  // all loads first: one memory latency per tile instead of one per row
  unsigned dg[ITEMS];
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const size_t i = base + (size_t)w * CHUNK + (size_t)r * 32 + lane;
    dg[r] = i < n ? (unsigned)((__ldcg(&kin[i]) >> shift) & 0xFF) : 256u;
  }
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    // (a row of one digit, common in the high digits, is one add)
    if (__all_sync(0xffffffffu, dg[r] == __shfl_sync(0xffffffffu, dg[r], 0))) {
      if (lane == 0 && dg[r] < 256u) atomicAdd(&h[w][dg[r]], 32u);
    } else if (dg[r] < 256u) {
      atomicAdd(&h[w][dg[r]], 1u);
    }
  }
  __syncthreads();
  u32 sum = 0;
#pragma unroll
  for (int q = 0; q < WARPS; ++q) sum += h[q][threadIdx.x];
  __stcg(&tile_hist[(size_t)threadIdx.x * t_max + tile], sum);
  __syncthreads();
}

// exclusive scan of one value per thread over the block's 256 threads
__device__ __forceinline__ u32 block_exclusive_256(u32 v, u32 *wsum, u32 &total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  u32 incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) wsum[w] = incl;
  __syncthreads();
  u32 before = 0;
  total = 0;
#pragma unroll
  for (int q = 0; q < WARPS; ++q) {
    if (q < w) before += wsum[q];
    total += wsum[q];
  }
  __syncthreads();
  return before + incl - v;
}

// exclusive scan over the tiles of digit d, in place; totals[d]
__device__ __forceinline__ void scan_digit(u32 *row, size_t T, u32 *total_out, u32 *wsum) {
  const size_t per = (T + TH - 1) / TH;
  const size_t a = threadIdx.x * per;
  const size_t b = a + per < T ? a + per : T;
  u32 s = 0;
  for (size_t t = a; t < b; ++t) s += __ldcg(&row[t]);
  u32 total;
  u32 run = block_exclusive_256(s, wsum, total);
  for (size_t t = a; t < b; ++t) {
    const u32 c = __ldcg(&row[t]);
    __stcg(&row[t], run);
    run += c;
  }
  if (threadIdx.x == 0) __stcg(total_out, total);
}

__device__ __forceinline__ void scatter_tile(const u64 *kin, const u32 *vin, u64 *kout, u32 *vout,
                                             size_t n, size_t tile, int shift,
                                             const u32 *tile_scan, size_t t_max, u32 digit_base,
                                             unsigned char *smem, u32 *wsum) {
  u64 *skeys = reinterpret_cast<u64 *>(smem);                            // TILE
  u32 *svals = reinterpret_cast<u32 *>(skeys + TILE);                    // TILE
  u32 *dstart = svals + TILE;                                            // 256
  u32 *gbase = dstart + 256;                                             // 256
  unsigned short *wh = reinterpret_cast<unsigned short *>(gbase + 256);  // WARPS*256
  const size_t base = tile * TILE;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const unsigned lt = (1u << lane) - 1;
  u64 key[ITEMS];
  u32 pos[ITEMS];
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const size_t i = base + (size_t)w * CHUNK + (size_t)r * 32 + lane;
    key[r] = i < n ? __ldcg(&kin[i]) : 0;
  }
  gbase[tid] = digit_base + __ldcg(&tile_scan[(size_t)tid * t_max + tile]);
  for (int j = tid; j < WARPS * 128; j += TH) reinterpret_cast<u32 *>(wh)[j] = 0;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const size_t i = base + (size_t)w * CHUNK + (size_t)r * 32 + lane;
    const bool valid = i < n;
    const unsigned d = valid ? (unsigned)((key[r] >> shift) & 0xFF) : 256u;
    const unsigned m = digit_peers<9>(d);
    unsigned c = 0;
    if (valid) {
      c = wh[w * 256 + d];
      pos[r] = c + __popc(m & lt);
    }
    __syncwarp();
    if (valid && (m & lt) == 0) wh[w * 256 + d] = (unsigned short)(c + __popc(m));
    __syncwarp();
  }
  __syncthreads();
  {  // per digit: exclusive over warps, then tile-local digit starts
    u32 run = 0;
#pragma unroll
    for (int q = 0; q < WARPS; ++q) {
      const u32 c = wh[q * 256 + tid];
      wh[q * 256 + tid] = (unsigned short)run;
      run += c;
    }
    u32 total;
    dstart[tid] = block_exclusive_256(run, wsum, total);
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const size_t i = base + (size_t)w * CHUNK + (size_t)r * 32 + lane;
    if (i < n) {
      const unsigned d = (unsigned)((key[r] >> shift) & 0xFF);
      pos[r] += dstart[d] + wh[w * 256 + d];
      skeys[pos[r]] = key[r];
    }
  }
  // (the values only now: both in registers at once would spill)
  u32 val[ITEMS];
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const size_t i = base + (size_t)w * CHUNK + (size_t)r * 32 + lane;
    val[r] = i < n ? __ldcg(&vin[i]) : 0;
  }
#pragma unroll
  for (int r = 0; r < ITEMS; ++r)
    if (base + (size_t)w * CHUNK + (size_t)r * 32 + lane < n) svals[pos[r]] = val[r];
  __syncthreads();
  const size_t cnt = (n - base) < (size_t)TILE ? (n - base) : (size_t)TILE;
  for (int j = tid; j < (int)cnt; j += TH) {
    const u64 k = skeys[j];
    const unsigned d = (unsigned)((k >> shift) & 0xFF);
    const size_t dst = (size_t)gbase[d] + (size_t)(j - (int)dstart[d]);
    __stcg(&kout[dst], k);
    __stcg(&vout[dst], svals[j]);
  }
  __syncthreads();  // shared memory is refilled by the next tile
}

__global__ __launch_bounds__(TH, 4) void k_sort_tiles(u64 *k0, u32 *v0, u64 *k1, u32 *v1,
                                                      size_t n_max, const u64 *n_dev,
                                                      const u64 *bits, u32 *tile_hist,
                                                      size_t t_max, u32 *totals) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ u32 wsum[WARPS];
  const size_t n = n_dev ? *n_dev : n_max;
  const u64 live = n ? live_mask(bits) : 0;
  const size_t T = tiles_for(n);
  int src = 0;
  for (int pass = 0; pass < 8; ++pass) {
    if (!pass_live(live, pass)) continue;
    const u64 *kin = src ? k1 : k0;
    const u32 *vin = src ? v1 : v0;
    for (size_t t = blockIdx.x; t < T; t += gridDim.x)
      tile_histogram(kin, n, t, 8 * pass, reinterpret_cast<u32 (*)[256]>(smem), tile_hist, t_max);
    grid.sync();
    for (unsigned d = blockIdx.x; d < 256; d += gridDim.x)
      scan_digit(tile_hist + (size_t)d * t_max, T, &totals[d], wsum);
    grid.sync();
    u32 all;
    const u32 digit_base = block_exclusive_256(__ldcg(&totals[threadIdx.x]), wsum, all);
    for (size_t t = blockIdx.x; t < T; t += gridDim.x)
      scatter_tile(kin, vin, src ? k0 : k1, src ? v0 : v1, n, t, 8 * pass, tile_hist, t_max,
                   digit_base, smem, wsum);
    src ^= 1;
    grid.sync();
  }
  if (src) {
    for (size_t i = blockIdx.x * (size_t)TH + threadIdx.x; i < n; i += (size_t)gridDim.x * TH) {
      k0[i] = __ldcg(&k1[i]);
      v0[i] = __ldcg(&v1[i]);
    }
  }
}

// the same steps as kernels of their own, a block per tile (or digit)
__global__ __launch_bounds__(TH) void k_hist(const u64 *k0, const u64 *k1, size_t n_max,
                                             const u64 *n_dev, const u64 *bits, int pass,
                                             u32 *tile_hist, size_t t_max) {
  __shared__ u32 h[WARPS][256];
  const u64 live = live_mask(bits);
  if (!pass_live(live, pass)) return;
  const size_t n = n_dev ? *n_dev : n_max;
  if ((size_t)blockIdx.x * TILE >= n) return;
  tile_histogram(pass_src(live, pass) ? k1 : k0, n, blockIdx.x, 8 * pass, h, tile_hist, t_max);
}

__global__ __launch_bounds__(TH) void k_scan_digit(u32 *tile_hist, size_t t_max, size_t n_max,
                                                   const u64 *n_dev, const u64 *bits, int pass,
                                                   u32 *totals) {
  __shared__ u32 wsum[WARPS];
  if (!pass_live(live_mask(bits), pass)) return;
  const size_t n = n_dev ? *n_dev : n_max;
  scan_digit(tile_hist + (size_t)blockIdx.x * t_max, tiles_for(n), &totals[blockIdx.x], wsum);
}

__global__ __launch_bounds__(TH, 3) void k_scatter(u64 *k0, u32 *v0, u64 *k1, u32 *v1,
                                                   size_t n_max, const u64 *n_dev,
                                                   const u64 *bits, int pass,
                                                   const u32 *tile_scan, size_t t_max,
                                                   const u32 *totals) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ u32 wsum[WARPS];
  const u64 live = live_mask(bits);
  if (!pass_live(live, pass)) return;
  const int src = pass_src(live, pass);
  const size_t n = n_dev ? *n_dev : n_max;
  if ((size_t)blockIdx.x * TILE >= n) return;
  u32 all;
  const u32 digit_base = block_exclusive_256(totals[threadIdx.x], wsum, all);
  scatter_tile(src ? k1 : k0, src ? v1 : v0, src ? k0 : k1, src ? v0 : v1, n, blockIdx.x, 8 * pass,
               tile_scan, t_max, digit_base, smem, wsum);
}

__global__ void k_copy_back(u64 *k0, u32 *v0, const u64 *k1, const u32 *v1, size_t n_max,
                            const u64 *n_dev, const u64 *bits) {
  if (!pass_src(live_mask(bits), 8)) return;
  const size_t n = n_dev ? *n_dev : n_max;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    k0[i] = k1[i];
    v0[i] = v1[i];
  }
}

// ---------------------------------------------------------------------------
// few keys: one share of them per block, held in registers
// ---------------------------------------------------------------------------
// Every block owns one contiguous share of the keys in each pass: it ranks
// them in shared memory (stable, as k_scatter), writes its digit counts, and
// after a grid barrier adds up the other blocks' counts for its offsets and
// scatters; a second barrier ends the pass. Bound by the barriers and the
// latency of the steps (about 12 us per live digit at 105k keys, 4 us at
// 2,500); the launches it replaces took 27 us per live digit and 8 us per dead one.
constexpr int CO_TH = 512, CO_WARPS = CO_TH / 32, CO_ITEMS = 8;
constexpr int kCoopItems = CO_TH * CO_ITEMS;  // keys per block

__global__ __launch_bounds__(CO_TH) void k_sort_coop(u64 *k0, u32 *v0, u64 *k1, u32 *v1,
                                                     size_t n_max, const u64 *n_dev,
                                                     u32 *counts) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  __shared__ u32 wh[CO_WARPS * 256];
  __shared__ u32 part[2][256], part_all[2][256];
  __shared__ u32 dbase[256];
  __shared__ u32 wsum[8];
  __shared__ u64 s_bits[2];
  const u32 n = (u32)(n_dev ? *n_dev : n_max);
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const u32 G = gridDim.x, b = blockIdx.x;
  // rows of 32 keys, a contiguous run of `rows` of them per warp
  const int rows = (int)((n + G * CO_TH - 1) / (G * CO_TH));
  const u32 base = (b * CO_WARPS + w) * (u32)(rows * 32) + lane;
  const unsigned lt = (1u << lane) - 1;
  u64 key[CO_ITEMS];
  u32 val[CO_ITEMS];
  u64 ones = 0, zeros = 0;
#pragma unroll
  for (int r = 0; r < CO_ITEMS; ++r) {
    const u32 i = base + r * 32;
    if (r < rows && i < n) {
      key[r] = k0[i];
      val[r] = v0[i];
      ones |= key[r];
      zeros |= ~key[r];
    }
  }
  // the bits that differ: the block's to memory, then everybody's
  u64 *bits = reinterpret_cast<u64 *>(counts + (size_t)G * 256);
  if (tid < 2) s_bits[tid] = 0;
  __syncthreads();
  note_key_bits(ones, zeros, s_bits);
  __syncthreads();
  if (tid < 2) __stcg(&bits[2 * b + tid], s_bits[tid]);
  grid.sync();
  ones = zeros = 0;
  for (u32 t = tid; t < G; t += CO_TH) {
    ones |= __ldcg(&bits[2 * t]);
    zeros |= __ldcg(&bits[2 * t + 1]);
  }
  if ((tid & ~31) < G) note_key_bits(ones, zeros, s_bits);
  __syncthreads();
  const u64 live = n ? live_mask(s_bits) : 0;
  int src = 0;
  bool loaded = true;  // the first live pass has its keys already
  for (int pass = 0; pass < 8; ++pass) {
    if (!pass_live(live, pass)) continue;
    const int shift = 8 * pass;
    const u64 *kin = src ? k1 : k0;
    const u32 *vin = src ? v1 : v0;
    u64 *kout = src ? k0 : k1;
    u32 *vout = src ? v0 : v1;
    if (!loaded) {  // (written by other SMs: past L1)
#pragma unroll
      for (int r = 0; r < CO_ITEMS; ++r) {
        const u32 i = base + r * 32;
        if (r < rows && i < n) {
          key[r] = __ldcg(&kin[i]);
          val[r] = __ldcg(&vin[i]);
        }
      }
    }
    loaded = false;
    for (int j = tid; j < CO_WARPS * 256; j += CO_TH) wh[j] = 0;
    __syncthreads();
    unsigned short pos[CO_ITEMS];
#pragma unroll
    for (int r = 0; r < CO_ITEMS; ++r) {
      if (r < rows) {
        const bool valid = base + r * 32 < n;
        const unsigned d = valid ? (unsigned)((key[r] >> shift) & 0xFF) : 256u;
        const unsigned m = digit_peers<9>(d);
        u32 c = 0;
        if (valid) c = wh[w * 256 + d];
        __syncwarp();
        if (valid) {
          pos[r] = (unsigned short)(c + __popc(m & lt));
          if ((m & lt) == 0) wh[w * 256 + d] = c + __popc(m);
        }
        __syncwarp();
      }
    }
    __syncthreads();
    if (tid < 256) {  // per digit: exclusive over the warps; the block's count
      u32 run = 0;
#pragma unroll
      for (int q = 0; q < CO_WARPS; ++q) {
        const u32 c = wh[q * 256 + tid];
        wh[q * 256 + tid] = run;
        run += c;
      }
      __stcg(&counts[b * 256 + tid], run);
    }
    grid.sync();
    {  // the digit's count in the blocks before this one, and in all
      const int d = tid & 255, half = tid >> 8;
      u32 before = 0, all = 0;
#pragma unroll 16
      for (u32 t = half; t < G; t += 2) {
        const u32 c = __ldcg(&counts[t * 256 + d]);
        all += c;
        if (t < b) before += c;
      }
      part[half][d] = before;
      part_all[half][d] = all;
    }
    __syncthreads();
    u32 t = 0, incl = 0;
    if (tid < 256) {
      t = part_all[0][tid] + part_all[1][tid];
      incl = t;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const u32 v = __shfl_up_sync(0xffffffffu, incl, s);
        if (lane >= s) incl += v;
      }
      if (lane == 31) wsum[w] = incl;
    }
    __syncthreads();
    if (tid < 256) {
      u32 off = incl - t + part[0][tid] + part[1][tid];
      for (int q = 0; q < w; ++q) off += wsum[q];
      dbase[tid] = off;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < CO_ITEMS; ++r) {
      if (r < rows && base + r * 32 < n) {
        const unsigned d = (unsigned)((key[r] >> shift) & 0xFF);
        const u32 p = dbase[d] + wh[w * 256 + d] + pos[r];
        __stcg(&kout[p], key[r]);
        __stcg(&vout[p], val[r]);
      }
    }
    src ^= 1;
    grid.sync();  // the scattered keys and the counts are free
  }
  if (src) {
    for (u32 i = b * CO_TH + tid; i < n; i += G * CO_TH) {
      k0[i] = __ldcg(&k1[i]);
      v0[i] = __ldcg(&v1[i]);
    }
  }
}

}  // namespace

// rows of 256 counts: one per tile, or per block of the cooperative kernel
static size_t hist_tiles(size_t n_max) {
  const size_t t = tiles_for(n_max), c = (n_max + CO_TH - 1) / CO_TH;
  return t + (c < 1024 ? c : 1024) + 1;
}

size_t sort_temp_bytes(size_t n_max) {
  return al(n_max * 8) + al(n_max * 4) + al(hist_tiles(n_max) * 256 * 4) + al(256 * 4) + al(64);
}

void sort_temp_carve(SortTemp &t, void *base, size_t n_max) {
  char *p = static_cast<char *>(base);
  t.keys_alt = reinterpret_cast<u64 *>(p); p += al(n_max * 8);
  t.vals_alt = reinterpret_cast<u32 *>(p); p += al(n_max * 4);
  t.tile_hist = reinterpret_cast<u32 *>(p); p += al(hist_tiles(n_max) * 256 * 4);
  t.global_hist = reinterpret_cast<u32 *>(p); p += al(256 * 4);  // digit totals
  t.pass_info = reinterpret_cast<int *>(p);                      // or/and words
}

// A block's warps take a row of 32 keys each, up to 32 blocks; then four rows:
// at 105k keys of 24 live bits 52 blocks take 38 us, 103 (two rows) 41, 148
// 51 and 26 44, the barriers and counts against the rows. Beyond that all SMs.
static size_t coop_blocks(const rvp_context *ctx, size_t n_max) {
  const size_t most = std::min(ctx->num_sms, 1024), rows4 = (n_max + 4 * CO_TH - 1) / (4 * CO_TH);
  return std::min({(n_max + CO_TH - 1) / CO_TH, std::max<size_t>(rows4, 32), most});
}

u64 *sort_key_bits(rvp_context *ctx, const SortTemp &t, size_t n_max) {
  if (n_max <= coop_blocks(ctx, n_max) * kCoopItems) return nullptr;  // finds them itself
  u64 *bits = reinterpret_cast<u64 *>(t.pass_info);
  RVP_CUDA_TRY(cudaMemsetAsync(bits, 0, 16, ctx->stream));
  return bits;
}

void radix_sort_pairs(rvp_context *ctx, u64 *keys, u32 *vals, size_t n_max,
                      const u64 *n_dev, const SortTemp &t, u64 *bits) {
  if (n_max == 0) return;
  u64 *k0 = keys, *k1 = t.keys_alt;
  u32 *v0 = vals, *v1 = t.vals_alt, *counts = t.tile_hist, *totals = t.global_hist;
  const size_t G = coop_blocks(ctx, n_max);
  if (n_max <= G * kCoopItems) {
    void *args[] = {&k0, &v0, &k1, &v1, &n_max, &n_dev, &counts};
    RVP_CUDA_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(k_sort_coop),
                                             dim3((unsigned)G), dim3(CO_TH), args, 0,
                                             ctx->stream));
    RVP_LAUNCH_CHECK(ctx);
    return;
  }
  static std::atomic<int> per_sm[64];  // blocks of k_sort_tiles an SM holds
  const int dev = ctx->device & 63;
  if (per_sm[dev] == 0) {
    RVP_CUDA_TRY(cudaFuncSetAttribute(k_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kTilesSmem));
    RVP_CUDA_TRY(cudaFuncSetAttribute(k_sort_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kTilesSmem));
    int b = 0;
    RVP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_sort_tiles, TH, kTilesSmem));
    RVP_REQUIRE(b > 0, "the sort kernel does not fit on the device");
    per_sm[dev] = b;
  }
  if (!bits) {
    bits = sort_key_bits(ctx, t, n_max);
    k_key_bits<<<grid_for(n_max, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(keys, n_max, n_dev,
                                                                                bits);
    RVP_LAUNCH_CHECK(ctx);
  }
  size_t T = tiles_for(n_max);
  if (T <= (size_t)ctx->num_sms * per_sm[dev]) {
    void *args[] = {&k0, &v0, &k1, &v1, &n_max, &n_dev, &bits, &counts, &T, &totals};
    RVP_CUDA_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(k_sort_tiles),
                                             dim3((unsigned)T), dim3(TH), args, kTilesSmem,
                                             ctx->stream));
    RVP_LAUNCH_CHECK(ctx);
    return;
  }
  for (int pass = 0; pass < 8; ++pass) {
    k_hist<<<(unsigned)T, TH, 0, ctx->stream>>>(k0, k1, n_max, n_dev, bits, pass, counts, T);
    RVP_LAUNCH_CHECK(ctx);
    k_scan_digit<<<256, TH, 0, ctx->stream>>>(counts, T, n_max, n_dev, bits, pass, totals);
    RVP_LAUNCH_CHECK(ctx);
    k_scatter<<<(unsigned)T, TH, kTilesSmem, ctx->stream>>>(k0, v0, k1, v1, n_max, n_dev, bits,
                                                           pass, counts, T, totals);
    RVP_LAUNCH_CHECK(ctx);
  }
  k_copy_back<<<grid_for(n_max, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(
      k0, v0, k1, v1, n_max, n_dev, bits);
  RVP_LAUNCH_CHECK(ctx);
}

// ---------------------------------------------------------------------------
// exclusive scan u32 -> u64 (3 kernels: tile sums, scan of tile sums, apply)
// ---------------------------------------------------------------------------
namespace {
// a tile: 256 threads x 16 consecutive items (four 16-byte loads each)
constexpr int SC_TH = 256, SC_IT = 16, SC_TILE = SC_TH * SC_IT;

// the thread's 16 items (zero past n): vector loads where the whole run is
// live and 16-byte aligned
__device__ __forceinline__ void scan_load(const u32 *in, size_t i0, size_t n, u32 (&v)[SC_IT]) {
  if (i0 + SC_IT <= n && (reinterpret_cast<uintptr_t>(in + i0) & 15) == 0) {
    const uint4 *p = reinterpret_cast<const uint4 *>(in + i0);
#pragma unroll
    for (int j = 0; j < SC_IT / 4; ++j) {
      const uint4 t = __ldg(p + j);
      v[4 * j] = t.x; v[4 * j + 1] = t.y; v[4 * j + 2] = t.z; v[4 * j + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < SC_IT; ++j) v[j] = (i0 + j < n) ? in[i0 + j] : 0u;
  }
}

// block-wide exclusive scan of one u64 per thread (warp shuffles, then the
// warps' totals); returns the exclusive prefix, *total the block's sum
__device__ __forceinline__ u64 block_exclusive(u64 s, u64 *warp_tot, u64 &total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  u64 incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u64 t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  u64 before = 0;
  total = 0;
#pragma unroll
  for (int k = 0; k < SC_TH / 32; ++k) {
    const u64 t = warp_tot[k];
    if (k < w) before += t;
    total += t;
  }
  return before + incl - s;
}

// (batched scans: blockIdx.y picks the array; strides in elements)
__global__ __launch_bounds__(SC_TH) void k_scan_tiles(const u32 *in, size_t n_max,
                                                      const u64 *n_dev, u64 *tsum,
                                                      size_t in_stride, size_t ts_stride) {
  in += blockIdx.y * in_stride;
  tsum += blockIdx.y * ts_stride;
  const size_t n = n_dev ? *n_dev : n_max;
  const size_t base = (size_t)blockIdx.x * SC_TILE;
  if (base >= n) return;
  u32 v[SC_IT];
  scan_load(in, base + (size_t)threadIdx.x * SC_IT, n, v);
  u64 s64 = 0;
#pragma unroll
  for (int j = 0; j < SC_IT; ++j) s64 += v[j];
  __shared__ u64 sh[SC_TH / 32];
  u64 r = s64;
#pragma unroll
  for (int o = 16; o; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = r;
  __syncthreads();
  if (threadIdx.x == 0) {
    u64 t = 0;
#pragma unroll
    for (int q = 0; q < SC_TH / 32; ++q) t += sh[q];
    tsum[blockIdx.x] = t;
  }
}

__global__ void k_scan_sums(u64 *tsum, size_t nt_max, size_t n_max, const u64 *n_dev,
                            u64 *out, size_t out_stride, size_t ts_stride) {
  tsum += blockIdx.x * ts_stride;
  out += blockIdx.x * out_stride;
  const size_t n = n_dev ? *n_dev : n_max;
  const size_t nt = (n + SC_TILE - 1) / SC_TILE;
  __shared__ u64 sh[1024];
  const size_t per = (nt + 1023) / 1024;
  const size_t a = threadIdx.x * per, b = a + per < nt ? a + per : nt;
  u64 s = 0;
  for (size_t t = a; t < b; ++t) s += tsum[t];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {
    u64 v = threadIdx.x >= (unsigned)off ? sh[threadIdx.x - off] : 0;
    __syncthreads();
    sh[threadIdx.x] += v;
    __syncthreads();
  }
  u64 run = sh[threadIdx.x] - s;
  for (size_t t = a; t < b; ++t) {
    const u64 c = tsum[t];
    tsum[t] = run;
    run += c;
  }
  if (threadIdx.x == 1023) out[n] = sh[1023];
  (void)nt_max;
}

__global__ __launch_bounds__(SC_TH) void k_scan_apply(const u32 *in, size_t n_max,
                                                      const u64 *n_dev, const u64 *tsum,
                                                      u64 *out, size_t in_stride,
                                                      size_t out_stride, size_t ts_stride) {
  in += blockIdx.y * in_stride;
  out += blockIdx.y * out_stride;
  tsum += blockIdx.y * ts_stride;
  const size_t n = n_dev ? *n_dev : n_max;
  const size_t base = (size_t)blockIdx.x * SC_TILE;
  if (base >= n) return;
  // thread t owns SC_IT consecutive items
  const size_t i0 = base + (size_t)threadIdx.x * SC_IT;
  u32 v[SC_IT];
  scan_load(in, i0, n, v);
  u64 s = 0;
#pragma unroll
  for (int j = 0; j < SC_IT; ++j) s += v[j];
  __shared__ u64 warp_tot[SC_TH / 32];
  u64 total;
  u64 run = tsum[blockIdx.x] + block_exclusive(s, warp_tot, total);
  if (i0 + SC_IT <= n && (reinterpret_cast<uintptr_t>(out + i0) & 15) == 0) {
    ulonglong2 *o = reinterpret_cast<ulonglong2 *>(out + i0);
#pragma unroll
    for (int j = 0; j < SC_IT; j += 2) {
      const u64 a0 = run;
      run += v[j];
      const u64 a1 = run;
      run += v[j + 1];
      o[j / 2] = make_ulonglong2(a0, a1);
    }
  } else {
#pragma unroll
    for (int j = 0; j < SC_IT; ++j) {
      if (i0 + j < n) out[i0 + j] = run;
      run += v[j];
    }
  }
}
}  // namespace

// Up to kScanOne items: one block, 16384 at a time with a carry. The three
// kernels of the general case take 12 us and two more launches however few
// items there are; this 5.4 us for 2,500 and 7.7 us for 7,106.
namespace {
constexpr size_t kScanOne = 49152;
constexpr int S1_TH = 1024;
__global__ __launch_bounds__(S1_TH) void k_scan_one(const u32 *in, size_t n_max, const u64 *n_dev,
                                                    u64 *out) {
  __shared__ u64 warp_tot[S1_TH / 32];
  const size_t n = n_dev ? *n_dev : n_max;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  u64 carry = 0;
  for (size_t base = 0; base < n; base += S1_TH * SC_IT) {
    const size_t i0 = base + (size_t)threadIdx.x * SC_IT;
    u32 v[SC_IT];
    scan_load(in, i0, n, v);
    u64 s = 0;
#pragma unroll
    for (int j = 0; j < SC_IT; ++j) s += v[j];
    u64 incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u64 t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    u64 t = warp_tot[lane], ti = t;  // every warp scans the warps' totals
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u64 p = __shfl_up_sync(0xffffffffu, ti, o);
      if (lane >= o) ti += p;
    }
    u64 run = carry + incl - s + __shfl_sync(0xffffffffu, ti - t, w);
    carry += __shfl_sync(0xffffffffu, ti, 31);
#pragma unroll
    for (int j = 0; j < SC_IT; ++j) {
      if (i0 + j < n) out[i0 + j] = run;
      run += v[j];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = carry;
}
}  // namespace

size_t scan_temp_bytes(size_t n_max) {
  return al(((n_max + SC_TILE - 1) / SC_TILE + 1) * 8);
}

void exclusive_scan_u32_to_u64(rvp_context *ctx, const u32 *in, u64 *out, size_t n_max,
                               const u64 *n_dev, void *temp) {
  exclusive_scan_u32_to_u64_batch(ctx, in, 0, out, 0, 1, n_max, n_dev, temp);
}

void exclusive_scan_u32_to_u64_batch(rvp_context *ctx, const u32 *in, size_t in_stride, u64 *out,
                                     size_t out_stride, int batch, size_t n_max,
                                     const u64 *n_dev, void *temp) {
  if (batch == 1 && n_max <= kScanOne) {
    k_scan_one<<<1, S1_TH, 0, ctx->stream>>>(in, n_max, n_dev, out);
    RVP_LAUNCH_CHECK(ctx);
    return;
  }
  const size_t nt = (n_max + SC_TILE - 1) / SC_TILE;
  const size_t ts_stride = scan_temp_bytes(n_max) / 8;
  u64 *tsum = static_cast<u64 *>(temp);
  const dim3 g((unsigned)(nt > 0 ? nt : 1), (unsigned)batch);
  k_scan_tiles<<<g, SC_TH, 0, ctx->stream>>>(in, n_max, n_dev, tsum, in_stride, ts_stride);
  RVP_LAUNCH_CHECK(ctx);
  k_scan_sums<<<(unsigned)batch, 1024, 0, ctx->stream>>>(tsum, nt, n_max, n_dev, out, out_stride,
                                                        ts_stride);
  RVP_LAUNCH_CHECK(ctx);
  k_scan_apply<<<g, SC_TH, 0, ctx->stream>>>(in, n_max, n_dev, tsum, out, in_stride, out_stride,
                                             ts_stride);
  RVP_LAUNCH_CHECK(ctx);
}

}  // namespace rvp
