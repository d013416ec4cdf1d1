// Statistical outlier removal (statistical_outlier_removal.cpp).
//
//  * global mean / std (:43-55): the reference sums sequentially in float,
//    and a sum in another order would round differently and move the
//    threshold; k_sor_stats reproduces those roundings in parallel;
//  * keep mean <= mu + alpha * sigma and copy kept points out in input order
//    (flag scan + scatter).
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
// below 2^24 u) by a block scan. With a tie among them every value becomes a
// pair of increments (S even, S odd), which compose associatively, and the
// scan runs over the pairs. Either way S after every value has exactly the
// roundings of the loop. The thread in whose run S first reaches 2^24 (the
// next binade) adds its own values one by one in float, and the rest of the
// chunk is scanned again from there: about log2(n) times over the whole sum,
// so the chunks start at 512 values and double up to 8192.
//   Bound by one SM's issue and the scans' latency (a block per frame): 89,343
// values 544 us with one lane adding in order (a dependent add per value),
// 123 us here; 256 frames of 11 M values 379 and 182 us.
constexpr int ST_TH = 512, ST_IT = 16, ST_CHUNK = ST_TH * ST_IT;
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

__global__ __launch_bounds__(ST_TH) void k_sor_stats(const float *__restrict__ mean,
                                                     const int64_t *offs, int n_frames,
                                                     float alpha, float *thresh) {
  __shared__ float buf[ST_CHUNK + ST_CHUNK / ST_IT];  // a gap per run: no bank conflicts
  __shared__ Incr warp_tot[ST_TH / 32];
  __shared__ float warp_sum[ST_TH / 32];
  __shared__ float s_acc;
  __shared__ int s_next;
  const int f = blockIdx.x;
  if (f >= n_frames) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t a = offs[f], n = offs[f + 1] - a;
  if (n <= 0) {
    if (tid == 0) thresh[f] = 0.0f;
    return;
  }
  mean += a;
  float mu = 0.0f;
  for (int pass = 0; pass < 2; ++pass) {
    float acc = 0.0f;
    float nxt[ST_IT];
    auto chunk_at = [&](int64_t base) {
      const int64_t len = base < 512 ? 512 : (base < ST_CHUNK ? base : ST_CHUNK);
      return (int)(n - base < len ? n - base : len);
    };
    auto fetch = [&](int64_t base) {
      const int m = base < n ? chunk_at(base) : 0;
#pragma unroll
      for (int j = 0; j < ST_IT; ++j) {
        const int i = j * ST_TH + tid;
        nxt[j] = i < m ? __ldg(&mean[base + i]) : mu;
      }
    };
    fetch(0);
    for (int64_t base = 0; base < n;) {
      const int m = chunk_at(base);
      bool odd = false;  // a value the increments cannot express
#pragma unroll
      for (int j = 0; j < ST_IT; ++j) {
        const int i = j * ST_TH + tid;
        if (j * ST_TH >= m) break;  // (uniform) rows past the chunk's end
        float v = nxt[j];
        if (pass == 1) {
          v = fsub(v, mu);
          v = fmul(v, v);
        }
        odd = odd || !(v >= 0.0f && v < INFINITY);
        buf[i + i / ST_IT] = v;
      }
      odd = __syncthreads_or(odd) || !(acc < INFINITY);
      base += m;
      if (odd) {  // (infinities, NaN, negative values): one lane, in order
        if (tid == 0) {
          float s = acc;
          for (int i = 0; i < m; ++i) s = fadd(s, buf[i + i / ST_IT]);
          s_acc = s;
        }
        fetch(base);
        __syncthreads();
        acc = s_acc;
        continue;
      }
      const int runs = (m + ST_IT - 1) / ST_IT;  // threads with values
      float v[ST_IT];
#pragma unroll
      for (int j = 0; j < ST_IT; ++j) v[j] = tid < runs ? buf[tid * (ST_IT + 1) + j] : 0.0f;
      fetch(base);
      int from = 0;  // threads before it are added already
      while (from < runs) {
        const int ex = st_exp(acc);
        const bool mine = tid >= from && tid < runs;
        // moves without ties: rounded to units by adding and taking away
        // 1.5 * 2^23 u, which needs v < 2^22 u
        const float magic = __uint_as_float(((u32)ex << 23) | 0x400000u);
        const float top = __uint_as_float((u32)(ex + 1) << 23);  // 2^24 u (inf past the last)
        const float half = ex > 30 ? __uint_as_float((u32)(ex - 24) << 23) : 0.0f;  // u / 2
        const float most = __uint_as_float((u32)(ex - 1) << 23);  // 2^22 u
        float sum = 0.0f;
        bool hard = ex <= 30;
        if (mine) {
#pragma unroll
          for (int j = 0; j < ST_IT; ++j) {
            const float q = fsub(fadd(v[j], magic), magic);
            hard = hard || fabsf(fsub(v[j], q)) == half || !(v[j] < most);
            sum = fadd(sum, q);
          }
        }
        float incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const float p = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl = fadd(p, incl);
        }
        if (lane == 31) warp_sum[warp] = incl;
        hard = __syncthreads_or(hard);
        float pre_acc, end_acc, all_acc;  // the sum before and after this run, and at the end
        if (!hard) {
          float before = 0.0f, total = 0.0f;
#pragma unroll
          for (int w = 0; w < ST_TH / 32; ++w) {
            if (w == warp) before = total;
            total = fadd(total, warp_sum[w]);
          }
          float pre = __shfl_up_sync(0xffffffffu, incl, 1);
          pre = fadd(before, lane == 0 ? 0.0f : pre);
          pre_acc = fadd(acc, pre);
          end_acc = fadd(acc, fadd(before, incl));
          all_acc = fadd(acc, total);
        } else {
          const u32 s0 = st_sig(acc);
          auto to_float = [&](u32 t) {  // below 2^24: in acc's binade; else past it
            return t >= ST_TOP ? top
                               : __uint_as_float(t >= 0x800000u ? ((u32)ex << 23) | (t & 0x7FFFFFu)
                                                                : t);
          };
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
          Incr upto = run;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            Incr p;
            p.a = __shfl_up_sync(0xffffffffu, upto.a, o);
            p.b = __shfl_up_sync(0xffffffffu, upto.b, o);
            if (lane >= o) upto = incr_then(p, upto);
          }
          if (lane == 31) warp_tot[warp] = upto;
          __syncthreads();
          Incr before{0, 0}, total{0, 0};
#pragma unroll
          for (int w = 0; w < ST_TH / 32; ++w) {
            if (w == warp) before = total;
            total = incr_then(total, warp_tot[w]);
          }
          Incr pre;  // everything before this thread's run
          pre.a = __shfl_up_sync(0xffffffffu, upto.a, 1);
          pre.b = __shfl_up_sync(0xffffffffu, upto.b, 1);
          if (lane == 0) pre = Incr{0, 0};
          pre = incr_then(before, pre);
          const Incr end = incr_then(pre, run);
          const bool p0 = s0 & 1;
          pre_acc = to_float(s0 + (p0 ? pre.b : pre.a));
          end_acc = to_float(s0 + (p0 ? end.b : end.a));
          all_acc = to_float(s0 + (p0 ? total.b : total.a));
        }
        if (all_acc < top) {
          acc = all_acc;
          break;
        }
        if (mine && pre_acc < top && !(end_acc < top)) {  // one thread
          float s = pre_acc;
#pragma unroll
          for (int j = 0; j < ST_IT; ++j) s = fadd(s, v[j]);
          s_acc = s;
          s_next = tid + 1;
        }
        __syncthreads();
        acc = s_acc;
        from = s_next;
        if (!(acc < INFINITY)) {  // overflow: every later sum is infinite too
          acc = INFINITY;
          break;
        }
      }
      __syncthreads();  // buf and the warps' totals are refilled
    }
    if (pass == 0) {
      mu = fdiv(acc, (float)n);
    } else if (tid == 0) {
      const float sd = __fsqrt_rn(fdiv(acc, (float)n));
      thresh[f] = fadd(mu, fmul(alpha, sd));
    }
  }
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
  k_sor_stats<<<(unsigned)(n_frames > 0 ? n_frames : 1), ST_TH, 0, st>>>(mean, offs, n_frames,
                                                                       alpha, thresh);
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
