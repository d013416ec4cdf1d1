// Statistical outlier removal (statistical_outlier_removal.cpp).
//
//  * global mean / std (:43-55): the reference sums sequentially in float,
//    and a sum in another order would round differently and move the
//    threshold; k_sor_stats reproduces those roundings in parallel;
//  * keep mean <= mu + alpha * sigma and copy kept points out in input order
//    (flag scan + scatter).
#include <cooperative_groups.h>

#include "internal.cuh"

namespace rvp {

namespace {
inline size_t al(size_t b) { return (b + 255) & ~(size_t)255; }

__device__ __forceinline__ int frame_of_index(const int64_t *offs, int n_frames, size_t i) {
  int lo = 0, hi = n_frames - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((size_t)offs[mid] <= i) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// The reference's sequential float sums, added in parallel. While the running
// sum A stays in one binade [2^e, 2^(e+1)) it is an integer S times its unit
// u = 2^(e-23), and adding v >= 0, v = (q + r) u, moves S by an integer: q
// (r < 1/2), q + 1 (r > 1/2), or, on a tie, to the even neighbour. Without
// ties the moves do not depend on S: they are summed (exactly, as floats
// below 2^24 u). With a tie among them every value becomes a pair of
// increments (S even, S odd), which compose associatively. Either way S after
// every value has exactly the roundings of the loop.
//   Three steps, twice (the mean, then the squares about it): the blocks of a
// cluster add up their shares in double; knowing about where the sum stands,
// each warp makes the pair of each of its segments of 256 values for that
// binade; and the first block composes the pairs from the true sum, 512
// segments at a time. Where a segment's binade was not foreseen, or the sum
// leaves it within the segment (about log2(n / 256) times), one lane adds the
// segment's values in order; after a run of such segments (sums that rounding
// has taken far from their true values) the block takes 4096 values at a time
// in the binade that it is in.
//   Bound by the first block's steps at each binade: 89,343 values 544 us with
// one lane adding in order (a dependent add per value), 123 us with one block
// making the pairs as it went, 52 us here; 256 frames of 11 M values 379, 182
// and 95 us.
constexpr int ST_TH = 512, ST_IT = 8, ST_CHUNK = ST_TH * ST_IT;
constexpr int ST_SEG = 256;         // values of a segment
constexpr int ST_FEW = 4 * ST_SEG;  // up to these one lane adds all
constexpr u32 ST_TOP = 1u << 24, ST_CAP = 1u << 30;

struct Incr {  // increments of S when it is even / odd, capped at ST_CAP
  u32 a, b;
};
__device__ __forceinline__ Incr incr_then(const Incr &f, const Incr &g) {
  const u32 x = f.a + ((f.a & 1) ? g.b : g.a);
  const u32 y = f.b + ((f.b & 1) ? g.a : g.b);  // odd S: parity flips with f.b
  return Incr{x < ST_CAP ? x : ST_CAP, y < ST_CAP ? y : ST_CAP};
}
// exponent field and 24-bit significand of a float >= 0: v = m * 2^(e - 150)
// (denormals share the smallest normal exponent)
__device__ __forceinline__ int st_exp(float v) { return max((int)(__float_as_uint(v) >> 23), 1); }
__device__ __forceinline__ u32 st_sig(float v) {
  const u32 b = __float_as_uint(v);
  return (b & 0x7FFFFFu) | (b >= 0x800000u ? 0x800000u : 0u);
}
// the increments of S by v, S in units of 2^(ex - 150)
__device__ __forceinline__ Incr incr_of(float v, int ex) {
  const u32 m = st_sig(v);
  const int s = ex - st_exp(v);  // low bits of v below the unit
  if (s <= 0) {
    const u32 q = s >= -6 ? m << -s : (m ? ST_CAP : 0u);
    return Incr{q, q};
  }
  if (s > 25) return Incr{0, 0};
  const u32 q = m >> s, r = m & ((1u << s) - 1u), half = 1u << (s - 1);
  if (r != half) {
    const u32 i = q + (r > half ? 1u : 0u);
    return Incr{i, i};
  }
  return Incr{q + (q & 1), q + ((q & 1) ^ 1)};
}

// S as the sum again: below 2^24 in the binade of exponent ex, else past it
__device__ __forceinline__ float st_float(u32 t, int ex) {
  return t >= ST_TOP ? __uint_as_float((u32)(ex + 1) << 23)
                     : __uint_as_float(t >= 0x800000u ? ((u32)ex << 23) | (t & 0x7FFFFFu) : t);
}
// what pass 1 adds for a value
__device__ __forceinline__ float st_value(float v, int pass, float mu) {
  if (pass == 0) return v;
  v = fsub(v, mu);
  return fmul(v, v);
}
// the moves of S without ties: rounded to units by adding and taking away
// 1.5 * 2^23 u, which needs v < 2^22 u
struct StMoves {
  float magic, half, most;
  __device__ __forceinline__ explicit StMoves(int ex) {
    magic = __uint_as_float(((u32)ex << 23) | 0x400000u);
    half = ex > 30 ? __uint_as_float((u32)(ex - 24) << 23) : 0.0f;  // u / 2
    most = __uint_as_float((u32)(ex - 1) << 23);                    // 2^22 u
  }
  __device__ __forceinline__ float of(float v, bool &hard) const {
    const float q = fsub(fadd(v, magic), magic);
    hard = hard || fabsf(fsub(v, q)) == half || !(v < most);
    return q;
  }
};
// inclusive scan of a block's pairs (warp_tot: one per warp)
__device__ __forceinline__ Incr incr_scan(Incr v, Incr *warp_tot, Incr &before) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto up = [&](Incr x, int o) {
    return Incr{__shfl_up_sync(0xffffffffu, x.a, o), __shfl_up_sync(0xffffffffu, x.b, o)};
  };
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const Incr p = up(v, o);
    if (lane >= o) v = incr_then(p, v);
  }
  if (lane == 31) warp_tot[warp] = v;
  __syncthreads();
  Incr t = lane < ST_TH / 32 ? warp_tot[lane] : Incr{0, 0};  // every warp scans the totals
#pragma unroll
  for (int o = 1; o < ST_TH / 32; o <<= 1) {
    const Incr p = up(t, o);
    if (lane >= o) t = incr_then(p, t);
  }
  const int w = warp > 0 ? warp - 1 : 0;
  Incr pre{__shfl_sync(0xffffffffu, t.a, w), __shfl_sync(0xffffffffu, t.b, w)};
  if (warp == 0) pre = Incr{0, 0};
  before = up(v, 1);
  before = incr_then(pre, lane == 0 ? Incr{0, 0} : before);
  return incr_then(pre, v);
}

// a segment's pair for the binade ex (0: none), as 16 bytes
struct StSeg {
  u64 pair, ex;
};

// by a whole block: acc after m <= ST_CHUNK values, whatever they are
__device__ float st_chunk(const float *mean, int m, int pass, float mu, float acc, float *buf,
                          Incr *warp_tot, float *s_acc, int *s_next) {
  const int tid = threadIdx.x;
  bool odd = false;  // a value the increments cannot express
  for (int i = tid; i < m; i += ST_TH) {
    const float v = st_value(__ldg(&mean[i]), pass, mu);
    odd = odd || !(v >= 0.0f && v < INFINITY);
    buf[i + i / ST_IT] = v;  // (a gap per run: no bank conflicts)
  }
  odd = __syncthreads_or(odd) || !(acc < INFINITY);
  if (odd) {  // (infinities, NaN, negative values): one lane, in order
    if (tid == 0) {
      float s = acc;
      for (int i = 0; i < m; ++i) s = fadd(s, buf[i + i / ST_IT]);
      *s_acc = s;
    }
    __syncthreads();
    return *s_acc;
  }
  const int runs = (m + ST_IT - 1) / ST_IT;  // threads with values
  float v[ST_IT];
#pragma unroll
  for (int j = 0; j < ST_IT; ++j)
    v[j] = tid * ST_IT + j < m ? buf[tid * (ST_IT + 1) + j] : 0.0f;
  int from = 0;  // threads before it are added already
  while (from < runs) {
    const int ex = st_exp(acc);
    const float top = __uint_as_float((u32)(ex + 1) << 23);  // 2^24 u (inf past the last)
    const bool mine = tid >= from && tid < runs;
    Incr run{0, 0};
    if (mine) {
      Incr t[ST_IT];
#pragma unroll
      for (int j = 0; j < ST_IT; ++j) t[j] = incr_of(v[j], ex);
#pragma unroll
      for (int w = 1; w < ST_IT; w <<= 1)  // pairwise, in order: a short chain
#pragma unroll
        for (int j = 0; j < ST_IT; j += 2 * w) t[j] = incr_then(t[j], t[j + w]);
      run = t[0];
    }
    const u32 s0 = st_sig(acc);
    Incr pre;
    const Incr end = incr_scan(run, warp_tot, pre);
    const float pre_acc = st_float(s0 + (s0 & 1 ? pre.b : pre.a), ex);
    const float end_acc = st_float(s0 + (s0 & 1 ? end.b : end.a), ex);
    if (tid == ST_TH - 1 && end_acc < top) *s_acc = end_acc, *s_next = runs;
    if (mine && pre_acc < top && !(end_acc < top)) {  // one thread leaves the binade
      float s = pre_acc;
#pragma unroll
      for (int j = 0; j < ST_IT; ++j) s = fadd(s, v[j]);
      *s_acc = s;
      *s_next = tid + 1;
    }
    __syncthreads();
    acc = *s_acc;
    from = *s_next;
    if (!(acc < INFINITY)) break;  // overflow: every later sum is infinite too
    __syncthreads();
  }
  __syncthreads();
  return acc;
}

__global__ __launch_bounds__(ST_TH, 2) void k_sor_stats(const float *__restrict__ mean_all,
                                                     const int64_t *offs, int n_frames,
                                                     float alpha, float *thresh, u64 *temp) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ float buf[ST_CHUNK + ST_CHUNK / ST_IT];
  __shared__ Incr warp_tot[ST_TH / 32];
  __shared__ double share[ST_TH / 32];  // sums of the warps' shares
  __shared__ float s_acc, s_mu;
  __shared__ int s_next;
  const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int f = blockIdx.x / C;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t a = offs[f], n = offs[f + 1] - a;
  if (n <= 0) {  // (the whole cluster)
    if (rank == 0 && tid == 0) thresh[f] = 0.0f;
    return;
  }
  const float *mean = mean_all + a;
  StSeg *segs = reinterpret_cast<StSeg *>(temp + 2 * ((a + 1) / 2));
  const int64_t n_seg = (n + ST_SEG - 1) / ST_SEG;
  const bool ahead = n > ST_FEW;  // (few enough: nothing is foreseen)
  // each warp's share of the segments
  const int W = C * (ST_TH / 32), me = rank * (ST_TH / 32) + warp;
  const int64_t lo = ahead ? n_seg * me / W : 0, hi = ahead ? n_seg * (me + 1) / W : 0;
  constexpr int IT = ST_SEG / 32;
  float mu = 0.0f;
  for (int pass = 0; pass < 2; ++pass) {
    if (ahead) {
      double sum = 0.0;
      for (int64_t i = lo * ST_SEG + lane, e = min(hi * ST_SEG, n); i < e; i += 32)
        sum += st_value(__ldg(&mean[i]), pass, mu);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) share[warp] = sum;
      cluster.sync();
      double at = 0.0;  // about the sum before the warp's share
      for (int w = lane; w < me; w += 32)
        at += *cluster.map_shared_rank(&share[w % (ST_TH / 32)], w / (ST_TH / 32));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) at += __shfl_xor_sync(0xffffffffu, at, o);
      for (int64_t g = lo; g < hi; ++g) {
        const int m = (int)min((int64_t)ST_SEG, n - g * ST_SEG);
        float v[IT];
        bool odd = false;
        float part = 0.0f;
#pragma unroll
        for (int j = 0; j < IT; ++j) {  // (lane's run is IT consecutive values)
          const int i = lane * IT + j;
          v[j] = i < m ? st_value(__ldg(&mean[g * ST_SEG + i]), pass, mu) : 0.0f;
          odd = odd || !(v[j] >= 0.0f && v[j] < INFINITY);
          part += v[j];
        }
        double total = part;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        const int ex = st_exp((float)at);
        at += total;
        StSeg r{0, 0};
        if (!__any_sync(0xffffffffu, odd) && at < 3.0e38 && ex == st_exp((float)at)) {
          const StMoves mv(ex);
          bool hard = ex <= 30;
          float q = 0.0f;
#pragma unroll
          for (int j = 0; j < IT; ++j) q = fadd(q, mv.of(v[j], hard));
          if (!__any_sync(0xffffffffu, hard)) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) q = fadd(q, __shfl_xor_sync(0xffffffffu, q, o));
            // (2^(150 - ex): units per one; capped as the pairs are)
            const float units = fmul(q, __uint_as_float((u32)(277 - ex) << 23));
            const u32 k = units < 1073741824.0f ? (u32)units : ST_CAP;
            r.pair = ((u64)k << 32) | k;
          } else {
            Incr t{0, 0};
#pragma unroll
            for (int j = 0; j < IT; ++j) t = incr_then(t, incr_of(v[j], ex));
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const Incr p{__shfl_up_sync(0xffffffffu, t.a, o),
                           __shfl_up_sync(0xffffffffu, t.b, o)};
              if (lane >= o) t = incr_then(p, t);
            }
            r.pair = ((u64)__shfl_sync(0xffffffffu, t.b, 31) << 32) |
                     __shfl_sync(0xffffffffu, t.a, 31);
          }
          r.ex = (u64)ex;
        }
        if (lane == 0) {
          __stcg(&segs[g].pair, r.pair);
          __stcg(&segs[g].ex, r.ex);
        }
      }
      cluster.sync();
    }
    if (rank == 0) {
      float acc = 0.0f;
      int alone = 0;  // segments in a row that were not foreseen
      for (int64_t w0 = 0; w0 < n_seg;) {
        const int count = (int)min((int64_t)ST_TH, n_seg - w0);
        StSeg r{0, 0};
        if (ahead && tid < count) {
          r.pair = __ldcg(&segs[w0 + tid].pair);
          r.ex = __ldcg(&segs[w0 + tid].ex);
        }
        int from = 0;
        while (from < count) {
          const int ex = st_exp(acc);
          const u32 s0 = st_sig(acc);
          const bool fits = tid >= from && tid < count && (int)r.ex == ex;
          // (uniform: the next segment was not foreseen)
          if (tid == from) s_next = fits ? ST_TH : from;
          __syncthreads();
          if (s_next > from) {
            Incr pre;
            const Incr run = fits ? Incr{(u32)r.pair, (u32)(r.pair >> 32)} : Incr{0, 0};
            const Incr end = incr_scan(run, warp_tot, pre);
            const u32 s1 = s0 + (s0 & 1 ? end.b : end.a), s = s0 + (s0 & 1 ? pre.b : pre.a);
            const bool stop = tid >= from && (!fits || s1 >= ST_TOP);
            if (stop) atomicMin(&s_next, tid);
            if (tid == ST_TH - 1) s_acc = st_float(s1, ex);
            __syncthreads();
            if (tid == s_next) s_acc = st_float(s, ex);  // the sum before it
            __syncthreads();
            acc = s_acc;
            if (s_next > from) alone = 0;
            from = s_next;
          }
          if (from >= count) break;
          const int64_t i0 = (w0 + from) * ST_SEG;
          if (alone < 8) {
            const int m = (int)min((int64_t)ST_SEG, n - i0);
            __syncthreads();
            if (tid < ST_SEG) buf[tid] = tid < m ? st_value(__ldg(&mean[i0 + tid]), pass, mu) : 0.0f;
            __syncthreads();
            if (tid == 0) {
              float s = acc;
              if (m == ST_SEG) {
#pragma unroll 32
                for (int i = 0; i < ST_SEG; ++i) s = fadd(s, buf[i]);
              } else {
                for (int i = 0; i < m; ++i) s = fadd(s, buf[i]);
              }
              s_acc = s;
            }
            __syncthreads();
            acc = s_acc;
            ++alone;
            ++from;
          } else {
            const int m = (int)min((int64_t)ST_CHUNK, n - i0);
            __syncthreads();
            acc = st_chunk(mean + i0, m, pass, mu, acc, buf, warp_tot, &s_acc, &s_next);
            alone = 8 - 1;  // the next one may be foreseen again
            from += (m + ST_SEG - 1) / ST_SEG;
          }
        }
        __syncthreads();
        w0 += from;
      }
      if (pass == 0) {
        if (tid == 0) s_mu = fdiv(acc, (float)n);
      } else if (tid == 0) {
        const float sd = __fsqrt_rn(fdiv(acc, (float)n));
        thresh[f] = fadd(mu, fmul(alpha, sd));
      }
    }
    if (pass == 0) {
      cluster.sync();
      mu = *cluster.map_shared_rank(&s_mu, 0);
    }
  }
  cluster.sync();  // (its shared memory is read until here)
}

__global__ void k_sor_keep(const float *mean, const int64_t *offs, int n_frames, size_t n_max,
                           const u64 *n_dev, const float *thresh, uint8_t *keep, u32 *flags) {
  const size_t n = n_dev ? *n_dev : n_max;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const int f = n_frames > 1 ? frame_of_index(offs, n_frames, i) : 0;
    const bool k = mean[i] <= thresh[f];
    if (keep) keep[i] = k ? 1 : 0;
    flags[i] = k ? 1u : 0u;
  }
}

__global__ void k_sor_scatter(const float *x, const float *y, const float *z, const u32 *flags,
                              const u64 *pos, size_t n_max, const u64 *n_dev, float *out_aos,
                              float *out_x, float *out_y, float *out_z, u32 *src_index) {
  const size_t n = n_dev ? *n_dev : n_max;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    if (!flags[i]) continue;
    const u64 p = pos[i];
    const float a = x[i], b = y[i], c = z[i];
    if (out_aos) {
      out_aos[3 * p + 0] = a;
      out_aos[3 * p + 1] = b;
      out_aos[3 * p + 2] = c;
    }
    if (out_x) {
      out_x[p] = a;
      out_y[p] = b;
      out_z[p] = c;
    }
    if (src_index) src_index[p] = (u32)i;
  }
}

__global__ void k_sor_frame_offsets(const int64_t *offs, int n_frames, const u64 *pos,
                                    int64_t *out) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f <= n_frames; f += gridDim.x * blockDim.x)
    out[f] = (int64_t)pos[offs[f]];
}
}  // namespace

u64 *sor_positions(void *temp, size_t n_max) {
  return reinterpret_cast<u64 *>(static_cast<char *>(temp) + al(n_max * 4));
}

size_t sor_filter_temp_bytes(size_t n_max, int n_frames) {
  return al(n_max * 4) + al((n_max + 1) * 8) + al((size_t)(n_frames + 1) * 4) +
         scan_temp_bytes(n_max);
}

void sor_filter_frames(rvp_context *ctx, const float *x, const float *y, const float *z,
                       const float *mean, const int64_t *offs, int n_frames, size_t n_max,
                       const u64 *n_dev, float alpha, uint8_t *keep, float *out_aos,
                       int64_t *out_offsets, float *thresh_out, void *temp, float *out_x,
                       float *out_y, float *out_z, u32 *src_index) {
  char *p = static_cast<char *>(temp);
  u32 *flags = reinterpret_cast<u32 *>(p); p += al(n_max * 4);
  u64 *pos = reinterpret_cast<u64 *>(p); p += al((n_max + 1) * 8);
  float *thresh = thresh_out ? thresh_out : reinterpret_cast<float *>(p);
  p += al((size_t)(n_frames + 1) * 4);
  void *scan_tmp = p;
  cudaStream_t st = ctx->stream;
  // 8 blocks per frame while the device holds them all at once (2 per SM: one
  // frame of 89,343 values 52 us); a block each for more frames, whose first
  // blocks would wait their turn with seven idle ones beside them
  const int frames = n_frames > 0 ? n_frames : 1;
  const unsigned C = frames * 8 <= ctx->num_sms * 2 ? 8 : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)frames * C);
  cfg.blockDim = dim3(ST_TH);
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = C;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  // (pos is free until the scan: 8 bytes per value, a segment needs 16)
  RVP_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_sor_stats, mean, offs, n_frames, alpha, thresh, pos));
  RVP_LAUNCH_CHECK(ctx);
  k_sor_keep<<<grid_for(n_max, 256, ctx->num_sms * 16), 256, 0, st>>>(mean, offs, n_frames, n_max,
                                                                     n_dev, thresh, keep, flags);
  RVP_LAUNCH_CHECK(ctx);
  exclusive_scan_u32_to_u64(ctx, flags, pos, n_max, n_dev, scan_tmp);
  k_sor_scatter<<<grid_for(n_max, 256, ctx->num_sms * 16), 256, 0, st>>>(
      x, y, z, flags, pos, n_max, n_dev, out_aos, out_x, out_y, out_z, src_index);
  RVP_LAUNCH_CHECK(ctx);
  if (out_offsets) {
    k_sor_frame_offsets<<<grid_for(n_frames + 1, 256, 64), 256, 0, st>>>(offs, n_frames, pos,
                                                                        out_offsets);
    RVP_LAUNCH_CHECK(ctx);
  }
}

}  // namespace rvp
