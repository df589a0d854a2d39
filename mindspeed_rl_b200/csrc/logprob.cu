// Row-wise log-softmax statistics over (a shard of) the vocabulary: per token the running
// max, sum-exp, target logit and sum e^{z-m} z, from which log p(label) and the entropy
// follow after a tiny cross-shard combine; and the matching backward that overwrites the logits
// with d loss / d logits.  Used by the chunked LM-head path (logits of a token chunk live only
// between the two GEMMs) and as the epilogue maths of the fused tcgen05 LM-head kernel.
//
// Reference semantics: vocab-parallel cross entropy and entropy with 3 all-reduces each
// (mindspeed_rl/utils/compute.py:29-97); here the shards' 4-float records are combined once.
#include "row_stat.cuh"

namespace msrl {

__global__ void __launch_bounds__(256)
logprob_stats_kernel(const __nv_bfloat16* __restrict__ logits, long long row_stride, int V,
                     int vocab_offset, const long long* __restrict__ labels, float inv_temp,
                     RowStat* __restrict__ out) {
  __shared__ float red[32];
  const long long r = blockIdx.x;
  const __nv_bfloat16* row = logits + r * row_stride;
  const int nvec = V >> 3;
  float m = -INFINITY, s = 0.f, spz = 0.f;
  for (int i = threadIdx.x; i < nvec; i += 256) {
    float f[8];
    unpack8(ld8(row + i * 8), f);
    float lm = -INFINITY;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      f[k] *= inv_temp;
      lm = fmaxf(lm, f[k]);
    }
    if (lm > m) {
      const float c = __expf(m - lm);
      s *= c;
      spz *= c;
      m = lm;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float e = __expf(f[k] - m);
      s += e;
      spz += e * f[k];
    }
  }
  for (int i = (nvec << 3) + threadIdx.x; i < V; i += 256) {  // tail (V % 8)
    const float z = __bfloat162float(row[i]) * inv_temp;
    if (z > m) {
      const float c = __expf(m - z);
      s *= c;
      spz *= c;
      m = z;
    }
    const float e = __expf(z - m);
    s += e;
    spz += e * z;
  }
  const float bm = block_max(m, red);
  const float c = (m == -INFINITY) ? 0.f : __expf(m - bm);
  const float bs = block_sum(s * c, red);
  const float bspz = block_sum(spz * c, red);
  if (threadIdx.x == 0) {
    const long long y = labels[r] - vocab_offset;
    RowStat o;
    o.m = bm;
    o.s = bs;
    o.spz = bspz;
    o.zy = (y >= 0 && y < V) ? __bfloat162float(row[y]) * inv_temp : 0.f;
    out[r] = o;
  }
}

// Combine `nshard` records per row ([nshard, T] layout) -> logp, entropy, lse.  W warps share the records of 32 rows, one row to a
// lane; bound by reading the records once (a thread to a row, as before, left most of the machine idle on the 594 records a row of a
// 152064-entry vocabulary: 16384 rows 211 -> 52 us, 300 rows 79 -> 15 us).  A few records a row need no sharing: see the rule below.
template <int W, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
logprob_finish_kernel(const RowStat* __restrict__ st, int nshard, long long T, float* __restrict__ logp,
                      float* __restrict__ entropy, float* __restrict__ lse_out, bool vec) {
  __shared__ float part[W > 1 ? WARPS : 1][4][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, mine = warp % W, first = warp - mine;
  const long long r = ((long long)blockIdx.x * (WARPS / W) + warp / W) * 32 + lane;
  const bool on = r < T;
  float m = -INFINITY;
#pragma unroll 4
  for (int k = mine; k < nshard; k += W)
    if (on) m = fmaxf(m, st[(long long)k * T + r].m);
  if constexpr (W > 1) {
    part[warp][0][lane] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < W; ++w) m = fmaxf(m, part[first + w][0][lane]);
  }
  float s = 0.f, spz = 0.f, zy = 0.f;
#pragma unroll 4
  for (int k = mine; k < nshard; k += W) {
    if (!on) break;
    const RowStat* at = st + (long long)k * T + r;
    RowStat a;
    if (vec) {
      const float4 x = *reinterpret_cast<const float4*>(at);
      a = RowStat{x.x, x.y, x.z, x.w};
    } else {
      a = *at;
    }
    const float c = __expf(a.m - m);
    s += a.s * c;
    spz += a.spz * c;
    zy += a.zy;
  }
  if constexpr (W > 1) {
    part[warp][1][lane] = s;
    part[warp][2][lane] = spz;
    part[warp][3][lane] = zy;
    __syncthreads();
    if (mine == 0) {
#pragma unroll
      for (int w = 1; w < W; ++w) {
        s += part[first + w][1][lane];
        spz += part[first + w][2][lane];
        zy += part[first + w][3][lane];
      }
    }
  }
  if (mine != 0 || !on) return;
  const float lse = m + __logf(s);
  logp[r] = zy - lse;
  if (entropy != nullptr) entropy[r] = lse - spz / s;
  if (lse_out != nullptr) lse_out[r] = lse;
}

// In place: logits <- d loss / d logits
//   dz_j = dlogp * (1[j == y] - p_j) + dent * p_j * ((lse - H) - z_j),  dlogit = dz * inv_temp
__global__ void __launch_bounds__(256)
logprob_bwd_kernel(__nv_bfloat16* __restrict__ logits, long long row_stride, int V,
                   int vocab_offset, const long long* __restrict__ labels, float inv_temp,
                   const float* __restrict__ lse, const float* __restrict__ entropy,
                   const float* __restrict__ dlogp, const float* __restrict__ dent) {
  const long long r = blockIdx.x;
  __nv_bfloat16* row = logits + r * row_stride;
  const float l = lse[r];
  const float g = dlogp[r];
  const float ge = (dent != nullptr) ? dent[r] : 0.f;
  const float mean_z = (entropy != nullptr) ? (l - entropy[r]) : 0.f;
  const long long y = labels[r] - vocab_offset;
  const int nvec = V >> 3;
  for (int i = threadIdx.x; i < nvec; i += 256) {
    float f[8];
    unpack8(ld8(row + i * 8), f);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float z = f[k] * inv_temp;
      const float pj = __expf(z - l);
      float d = -g * pj + ge * pj * (mean_z - z);
      if ((long long)(i * 8 + k) == y) d += g;
      f[k] = d * inv_temp;
    }
    st8(row + i * 8, pack8(f));
  }
  for (int i = (nvec << 3) + threadIdx.x; i < V; i += 256) {
    const float z = __bfloat162float(row[i]) * inv_temp;
    const float pj = __expf(z - l);
    float d = -g * pj + ge * pj * (mean_z - z);
    if ((long long)i == y) d += g;
    row[i] = __float2bfloat16(d * inv_temp);
  }
}

}  // namespace msrl

using namespace msrl;

MSRL_API int msrl_logprob_stats(const void* logits, long long row_stride, long long T, int V,
                                int vocab_offset, const long long* labels, float inv_temp,
                                void* stats_out, cudaStream_t st) {
  if (T == 0) return 0;
  if (row_stride % 8 != 0) return (int)cudaErrorInvalidValue;
  logprob_stats_kernel<<<(unsigned)T, 256, 0, st>>>((const __nv_bfloat16*)logits, row_stride, V,
                                                    vocab_offset, labels, inv_temp,
                                                    (RowStat*)stats_out);
  MSRL_LAUNCH_CHECK();
}

MSRL_API int msrl_logprob_finish(const void* stats, int nshard, long long T, float* logp,
                                 float* entropy, float* lse, cudaStream_t st) {
  if (T == 0) return 0;
  // A record a vocabulary shard: sharing costs more than it saves.  A thread to a row / 4 / 16 warps to 32 rows: 1 record, 16384 rows
  // 1.8 / 1.9 / 2.6 us, 4 records 1.9 / 2.1 / 2.7, 8 records 2.5 / 2.3 / 2.9, 32 records 4.7 / 3.2 / 3.7 (65536 rows 9.9 / 6.0 / 9.3),
  // 64 records 11.1 / 6.2 / 4.6.
  const bool vec = (reinterpret_cast<uintptr_t>(stats) & 15) == 0;
  const RowStat* in = (const RowStat*)stats;
  if (nshard <= 4)
    logprob_finish_kernel<1, 4><<<(unsigned)ceil_div(T, 128), 128, 0, st>>>(in, nshard, T, logp, entropy, lse, vec);
  else if (nshard <= 32)
    logprob_finish_kernel<4, 4><<<(unsigned)ceil_div(T, 32), 128, 0, st>>>(in, nshard, T, logp, entropy, lse, vec);
  else
    logprob_finish_kernel<16, 16><<<(unsigned)ceil_div(T, 32), 512, 0, st>>>(in, nshard, T, logp, entropy, lse, vec);
  MSRL_LAUNCH_CHECK();
}

MSRL_API int msrl_logprob_bwd(void* logits, long long row_stride, long long T, int V,
                              int vocab_offset, const long long* labels, float inv_temp,
                              const float* lse, const float* entropy, const float* dlogp,
                              const float* dent, cudaStream_t st) {
  if (T == 0) return 0;
  if (row_stride % 8 != 0) return (int)cudaErrorInvalidValue;
  logprob_bwd_kernel<<<(unsigned)T, 256, 0, st>>>((__nv_bfloat16*)logits, row_stride, V,
                                                  vocab_offset, labels, inv_temp, lse, entropy,
                                                  dlogp, dent);
  MSRL_LAUNCH_CHECK();
}
