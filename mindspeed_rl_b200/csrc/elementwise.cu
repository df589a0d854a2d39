// Memory-bound fused ops: RMSNorm (fwd/bwd, optional residual add, per-head variant),
// RoPE (in place, fwd/bwd), SwiGLU (fwd/bwd), residual add, bias-grad column sums.
// All tensors bf16 with fp32 math; rows are moved with 128-bit loads/stores.
//
// Reference call sites these replace: flags use_fused_rmsnorm / use_fused_rotary_pos_emb /
// use_fused_swiglu / qk_layernorm (mindspeed_rl/config_cls/megatron_config.py:209-212,332).
#include "mma_utils.cuh"  // HeadLayout: addressing of heads inside fused QKV rows

namespace msrl {

// --------------------------------------------------------------------------------------------
// RMSNorm forward, one block per row.  Optional residual: s = x + res is written to sum_out
// and normalised (the "add + norm" pair between sub-layers).
// --------------------------------------------------------------------------------------------
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ sum_out, float* __restrict__ rstd_out, int H,
                   float eps) {
  __shared__ float red[32];
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  float* row = reinterpret_cast<float*>(dyn_smem);  // H floats: the (summed) row in fp32
  const long long r = blockIdx.x;
  const __nv_bfloat16* xr = x + r * H;
  const int nvec = H >> 3;
  float ss = 0.f;
  for (int i = threadIdx.x; i < nvec; i += THREADS) {
    float f[8];
    unpack8(ld8(xr + i * 8), f);
    if (res != nullptr) {
      float g[8];
      unpack8(ld8(res + r * H + i * 8), g);
#pragma unroll
      for (int k = 0; k < 8; ++k) f[k] += g[k];
      if (sum_out != nullptr) {
        bf16x8 s = pack8(f);
        st8(sum_out + r * H + i * 8, s);
        unpack8(s, f);  // normalise exactly what was stored
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      row[i * 8 + k] = f[k];
      ss += f[k] * f[k];
    }
  }
  ss = block_sum(ss, red);
  const float rstd = rsqrtf(ss / (float)H + eps);
  if (threadIdx.x == 0 && rstd_out != nullptr) rstd_out[r] = rstd;
  for (int i = threadIdx.x; i < nvec; i += THREADS) {
    float wv[8], o[8];
    unpack8(ld8(w + i * 8), wv);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = row[i * 8 + k] * rstd * wv[k];
    st8(y + r * H + i * 8, pack8(o));
  }
}

// Warp-per-row form (H <= 32 * VPT * 8): every warp owns whole rows (blockIdx / warp strided), reads a row
// into registers with VPT independent 16-byte loads per lane, reduces it with shuffles only (no block
// barrier anywhere), scales and stores it.  With five 128-thread blocks per SM about 140 KB of loads are in
// flight per SM, which is what a streaming kernel with a reduction in the middle needs to stay near the
// copy bandwidth.
template <int VPT, bool RES>
__global__ void __launch_bounds__(128)
rmsnorm_fwd_warp_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                        const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                        __nv_bfloat16* __restrict__ sum_out, float* __restrict__ rstd_out, long long rows,
                        int H, float eps) {
  const int lane = threadIdx.x & 31;
  const int nvec = H >> 3;
  const long long warps = (long long)gridDim.x * 4;
  for (long long r = (long long)blockIdx.x * 4 + (threadIdx.x >> 5); r < rows; r += warps) {
    bf16x8 raw[VPT], raw_res[RES ? VPT : 1];
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = lane + j * 32;
      if (i < nvec) {
        raw[j] = ld8(x + r * H + i * 8);
        if (RES) raw_res[j] = ld8(res + r * H + i * 8);
      }
    }
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = lane + j * 32;
      if (i < nvec) {
        float f[8];
        unpack8(raw[j], f);
        if (RES) {
          float g[8];
          unpack8(raw_res[j], g);
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] += g[k];
          raw[j] = pack8(f);                       // the rounded sum is what gets stored and normalised
          if (sum_out != nullptr) st8(sum_out + r * H + i * 8, raw[j]);
          unpack8(raw[j], f);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) ss += f[k] * f[k];
      }
    }
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (lane == 0 && rstd_out != nullptr) rstd_out[r] = rstd;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = lane + j * 32;
      if (i < nvec) {
        float f[8], wv[8], o[8];
        unpack8(raw[j], f);
        unpack8(ld8(w + i * 8), wv);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = f[k] * rstd * wv[k];
        st8(y + r * H + i * 8, pack8(o));
      }
    }
  }
}

// One-pass form for rows that fit the block's registers (H <= THREADS * VPT * 8).  Persistent blocks
// walk rows blockIdx.x, +gridDim.x, ...; the loads of the next row are issued before the current row
// is reduced, scaled and stored, so that a block always has a row in flight (no shared-memory staging
// of the row; with the optional residual the rounded sum is written back and normalised).
template <int THREADS, int VPT>
__global__ void __launch_bounds__(THREADS)
rmsnorm_fwd_regs_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                        const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                        __nv_bfloat16* __restrict__ sum_out, float* __restrict__ rstd_out, long long rows,
                        int H, float eps) {
  __shared__ float red[2][32];
  const int nvec = H >> 3;
  bf16x8 cur[VPT], cur_res[VPT], nxt[VPT], nxt_res[VPT], wr[1];
  auto fetch = [&](long long r, bf16x8 (&dst)[VPT], bf16x8 (&dst_res)[VPT]) {
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = threadIdx.x + j * THREADS;
      if (i < nvec) {
        dst[j] = ld8(x + r * H + i * 8);
        if (res != nullptr) dst_res[j] = ld8(res + r * H + i * 8);
      }
    }
  };
  long long r = blockIdx.x;
  if (r < rows) fetch(r, cur, cur_res);
  if constexpr (VPT == 1) wr[0] = ld8(w + (threadIdx.x < nvec ? threadIdx.x : 0) * 8);   // ahead of the sum
  int flip = 0;
  for (; r < rows; r += gridDim.x, flip ^= 1) {
    const long long rn = r + gridDim.x;
    if (rn < rows) fetch(rn, nxt, nxt_res);          // in flight while this row is processed
    float f[VPT][8];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = threadIdx.x + j * THREADS;
      if (i < nvec) {
        unpack8(cur[j], f[j]);
        if (res != nullptr) {
          float g[8];
          unpack8(cur_res[j], g);
#pragma unroll
          for (int k = 0; k < 8; ++k) f[j][k] += g[k];
          if (sum_out != nullptr) {
            const bf16x8 s = pack8(f[j]);
            st8(sum_out + r * H + i * 8, s);
            unpack8(s, f[j]);  // normalise exactly what was stored
          }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) ss += f[j][k] * f[j][k];
      }
    }
    {   // block sum with alternating scratch: one barrier per row is enough
      const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
      ss = warp_sum(ss);
      if (lane == 0) red[flip][wid] = ss;
      __syncthreads();
      ss = warp_sum(lane < THREADS / 32 ? red[flip][lane] : 0.f);
    }
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (threadIdx.x == 0 && rstd_out != nullptr) rstd_out[r] = rstd;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = threadIdx.x + j * THREADS;
      if (i < nvec) {
        float wv[8], o[8];
        unpack8(VPT == 1 ? wr[0] : ld8(w + i * 8), wv);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = f[j][k] * rstd * wv[k];
        st8(y + r * H + i * 8, pack8(o));
      }
    }
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      cur[j] = nxt[j];
      cur_res[j] = nxt_res[j];
    }
  }
}

// RMSNorm backward, stage 1: each block walks rows blockIdx.x, +gridDim.x, ... and
//   dx = rstd * (dy*w) - x * rstd^3 * mean(dy*w*x)   (optionally dx += dres)
// while keeping partial sums of dw = sum_rows dy * x * rstd in registers; the partials go to
// `dw_partial[gridDim.x, H]` (scratch) and stage 2 reduces them over blocks.
// The loads of the next row are in flight while a row is summed, and one barrier a row is enough; bound by reading dy, x (and dres)
// and writing dx once.  Whole calls (with stage 2) from cold caches against loads in the row's turn and two barriers, with dres:
// 32768 x 3584 376 -> 196 us, 8416 x 3584 116 -> 65, 1481 x 4096 44 -> 28.  Above 4096 columns the prefetch takes 201 to 249 registers
// and one block of 256 threads an SM is resident where two were; the loads in flight are worth more: 32768 x 5120 513 -> 312, 32768 x
// 7168 663 -> 433, 1481 x 5120 48 -> 34, 1481 x 8192 65 -> 48, 16 x 7168 17.4 -> 15.4.
template <int THREADS, int VPT>
__global__ void __launch_bounds__(THREADS)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                   const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                   float* __restrict__ dw_partial, long long rows, int H) {
  __shared__ float red[2][32];
  const int nvec = H >> 3;
  float dw_acc[VPT][8];
  bf16x8 wv[VPT], cur_d[VPT], cur_x[VPT], cur_e[VPT], nxt_d[VPT], nxt_x[VPT], nxt_e[VPT];
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int i = threadIdx.x + j * THREADS;
    if (i < nvec) wv[j] = ld8(w + i * 8);
#pragma unroll
    for (int k = 0; k < 8; ++k) dw_acc[j][k] = 0.f;
  }
  auto fetch = [&](long long r, bf16x8 (&d)[VPT], bf16x8 (&xx)[VPT], bf16x8 (&e)[VPT]) {
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = threadIdx.x + j * THREADS;
      if (i < nvec) {
        d[j] = ld8(dy + r * H + i * 8);
        xx[j] = ld8(x + r * H + i * 8);
        if (dres != nullptr) e[j] = ld8(dres + r * H + i * 8);
      }
    }
  };
  long long r = blockIdx.x;
  float rs = 0.f, rs_next = 0.f;
  if (r < rows) {
    fetch(r, cur_d, cur_x, cur_e);
    rs = rstd[r];
  }
  int flip = 0;
  for (; r < rows; r += gridDim.x, flip ^= 1) {
    const long long rn = r + gridDim.x;
    if (rn < rows) {
      fetch(rn, nxt_d, nxt_x, nxt_e);
      rs_next = rstd[rn];
    }
    float g[VPT][8], xv[VPT][8];
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = threadIdx.x + j * THREADS;
      if (i < nvec) {
        float d[8], wf[8];
        unpack8(cur_d[j], d);
        unpack8(cur_x[j], xv[j]);
        unpack8(wv[j], wf);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          g[j][k] = d[k] * wf[k];
          dot += g[j][k] * xv[j][k];
          dw_acc[j][k] += d[k] * xv[j][k] * rs;
        }
      }
    }
    {   // block sum with alternating scratch
      const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
      dot = warp_sum(dot);
      if (lane == 0) red[flip][wid] = dot;
      __syncthreads();
      dot = warp_sum(lane < THREADS / 32 ? red[flip][lane] : 0.f);
    }
    const float c = dot * rs * rs * rs / (float)H;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int i = threadIdx.x + j * THREADS;
      if (i < nvec) {
        float o[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = g[j][k] * rs - xv[j][k] * c;
        if (dres != nullptr) {
          float e[8];
          unpack8(cur_e[j], e);
#pragma unroll
          for (int k = 0; k < 8; ++k) o[k] += e[k];
        }
        st8(dx + r * H + i * 8, pack8(o));
      }
    }
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      cur_d[j] = nxt_d[j];
      cur_x[j] = nxt_x[j];
      cur_e[j] = nxt_e[j];
    }
    rs = rs_next;
  }
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int i = threadIdx.x + j * THREADS;
    if (i < nvec) {
#pragma unroll
      for (int k = 0; k < 8; ++k) dw_partial[(long long)blockIdx.x * H + i * 8 + k] = dw_acc[j][k];
    }
  }
}

// Stage 2: dw[h] (+)= sum_b partial[b, h].  32 columns to a block, its warps share the rows and add up in their order: a chain of
// a few loads in place of one per row (4096 columns, 296 rows: 21.4 -> 3.6 us).
constexpr int COLSUM_WARPS = 16;
__global__ void __launch_bounds__(COLSUM_WARPS * 32)
colsum_partials_kernel(const float* __restrict__ partial, int nblocks, int H, float* __restrict__ out_f32,
                       __nv_bfloat16* __restrict__ out_bf16, int accumulate) {
  __shared__ float part[COLSUM_WARPS][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, h = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (h < H) {
#pragma unroll 8
    for (int b = warp; b < nblocks; b += COLSUM_WARPS) s += partial[(long long)b * H + h];
  }
  part[warp][lane] = s;
  __syncthreads();
  if (warp != 0 || h >= H) return;
#pragma unroll
  for (int w = 1; w < COLSUM_WARPS; ++w) s += part[w][lane];
  if (out_f32 != nullptr) out_f32[h] = accumulate ? out_f32[h] + s : s;
  if (out_bf16 != nullptr)
    out_bf16[h] = __float2bfloat16(accumulate ? __bfloat162float(out_bf16[h]) + s : s);
}

// --------------------------------------------------------------------------------------------
// Per-head RMSNorm (QK-norm), head_dim <= 256, in place capable.
// --------------------------------------------------------------------------------------------
// G lanes to a head (eight entries each), U heads a thread with their loads in flight together.  Bound by reading and writing the
// heads once (a warp to a head, half of it idle at 128 entries, and one load at a time before: 16384 tokens x 32 heads of 128
// 112 -> 49 us, 1481 tokens 11.9 -> 6.1).  A decode step has too few heads to put several in a thread.
template <int G, int U>
__global__ void __launch_bounds__(256)
headnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, HeadLayout L, const __nv_bfloat16* __restrict__ w,
                    __nv_bfloat16* __restrict__ y, float* __restrict__ rstd_out, unsigned heads, int nheads, int hd, float eps) {
  const int g = threadIdx.x % G;
  const bool act = g * 8 < hd;
  float wv[8];
  unpack8(ld8(w + (act ? g * 8 : 0)), wv);
  bf16x8 raw[U];
  long long off[U];
  const unsigned first = blockIdx.x * (U * 256 / G) + threadIdx.x / G;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const unsigned i = first + u * (256 / G);
    const unsigned t = i / (unsigned)nheads;
    off[u] = head_offset(L, t, (int)(i - t * (unsigned)nheads)) + g * 8;
    if (act && i < heads) raw[u] = ld8(x + off[u]);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const unsigned i = first + u * (256 / G);
    const bool on = act && i < heads;
    float f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (on) unpack8(raw[u], f);
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) ss += f[k] * f[k];
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float rs = rsqrtf(ss / (float)hd + eps);
    if (g == 0 && i < heads && rstd_out != nullptr) rstd_out[i] = rs;
    if (on) {
#pragma unroll
      for (int k = 0; k < 8; ++k) f[k] = f[k] * rs * wv[k];
      st8(y + off[u], pack8(f));
    }
  }
}

// Backward of the per-head norm. dx overwrites dy in place (same layout); dw partial sums are
// accumulated per block into dw_partial[gridDim.x, hd].
// The mapping of the forward, walked by persistent blocks (154 -> 68 us, 1481 tokens 15.0 -> 8.4).
template <int G>
__global__ void __launch_bounds__(256)
headnorm_bwd_kernel(__nv_bfloat16* __restrict__ dy_dx, const __nv_bfloat16* __restrict__ x, HeadLayout L,
                    const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd, float* __restrict__ dw_partial,
                    long long T, long long chunk, int nheads, int hd) {
  __shared__ float sdw[8][256];    // one row per warp (256 threads): summed in warp order, so that the
                                   // result does not depend on which warp finishes first
  constexpr int U = 2;
  const int lane = threadIdx.x & 31, g = threadIdx.x % G;
  const bool act = g * 8 < hd;
  float dw_acc[8] = {0, 0, 0, 0, 0, 0, 0, 0}, wv[8];
  unpack8(ld8(w + (act ? g * 8 : 0)), wv);
  for (long long t0 = 0; t0 < T; t0 += chunk, dy_dx += chunk * L.stride_t, x += chunk * L.stride_t, rstd += chunk * nheads) {
    const unsigned heads = (unsigned)(T - t0 < chunk ? T - t0 : chunk) * (unsigned)nheads;
    for (unsigned base = blockIdx.x * (U * 256 / G); base < heads; base += gridDim.x * (U * 256 / G)) {
      bf16x8 rd[U], rx[U];
      long long off[U];
      float rs[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned i = base + u * (256 / G) + threadIdx.x / G, t = i / (unsigned)nheads;
        off[u] = head_offset(L, t, (int)(i - t * (unsigned)nheads)) + g * 8;
        rs[u] = 0.f;
        if (act && i < heads) {
          rd[u] = ld8(dy_dx + off[u]);
          rx[u] = ld8(x + off[u]);
          rs[u] = rstd[i];
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool on = act && base + u * (256 / G) + threadIdx.x / G < heads;
        float d[8] = {0, 0, 0, 0, 0, 0, 0, 0}, xv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        float dot = 0.f;
        if (on) {
          unpack8(rd[u], d);
          unpack8(rx[u], xv);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            dw_acc[k] += d[k] * xv[k] * rs[u];
            d[k] *= wv[k];
            dot += d[k] * xv[k];
          }
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        const float c = dot * rs[u] * rs[u] * rs[u] / (float)hd;
        if (on) {
#pragma unroll
          for (int k = 0; k < 8; ++k) d[k] = d[k] * rs[u] - xv[k] * c;
          st8(dy_dx + off[u], pack8(d));
        }
      }
    }
  }
  // the groups of a warp
#pragma unroll
  for (int o = G; o < 32; o <<= 1)
#pragma unroll
    for (int k = 0; k < 8; ++k) dw_acc[k] += __shfl_xor_sync(0xffffffffu, dw_acc[k], o);
  const int warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (lane < G) sdw[warp][g * 8 + k] = act ? dw_acc[k] : 0.f;
  __syncthreads();
  for (int i = threadIdx.x; i < hd; i += blockDim.x) {
    float t = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sdw[w][i];
    dw_partial[(long long)blockIdx.x * hd + i] = t;
  }
}

// --------------------------------------------------------------------------------------------
// RoPE (rotate-half / "neox" pairing: element i pairs with i + hd/2), in place.
// cos_sin table: [max_pos, hd] fp32 = [cos(0..hd/2) | sin(0..hd/2)] per position.
// sign = +1 forward, -1 backward (the inverse rotation applied to gradients).
// --------------------------------------------------------------------------------------------
// A thread takes V pairs of a head, V = 8 with 16-byte accesses where base and strides allow, else 4; threads run over (token, head,
// vector) without regard to where a token ends, so that no count of heads leaves part of a block idle (a block to a token took 83 us
// for 16384 tokens of 32 + 4 heads of 128, 2.7 us for 48).  Bound by reading and writing the heads once; indices in 32 bits, two
// divisions a vector.  Before (V = 4, four 64-bit divisions) and now: 16384 tokens, 28 + 4 heads of 128 59 -> 49 us, 32 + 4
// 66 -> 54, 1481 tokens 7.5 -> 5.4; 32768 tokens, 12 + 12 heads of 72 (V = 4, at most eight blocks an SM) 60 -> 56.
template <int V>
__global__ void __launch_bounds__(256)
rope_kernel(__nv_bfloat16* __restrict__ q, HeadLayout Lq, unsigned nq, __nv_bfloat16* __restrict__ k, HeadLayout Lk, unsigned nk,
            const int* __restrict__ positions, const float* __restrict__ cos_sin, unsigned total, int hd, float sign) {
  const int half = hd >> 1;
  const unsigned per_head = half / V, nh = nq + nk;
  for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < total; i += gridDim.x * 256) {
    const unsigned th = i / per_head, t = th / nh, h = th - t * nh;
    const int c = (int)(i - th * per_head) * V;
    __nv_bfloat16* base = (h < nq ? q + head_offset(Lq, t, (int)h) : k + head_offset(Lk, t, (int)(h - nq))) + c;
    const float* cs = cos_sin + (long long)positions[t] * hd + c;
    alignas(16) float cc[V], sn[V];
    float a[V], b[V];
#pragma unroll
    for (int j = 0; j < V; j += 4) {
      *reinterpret_cast<float4*>(cc + j) = *reinterpret_cast<const float4*>(cs + j);
      *reinterpret_cast<float4*>(sn + j) = *reinterpret_cast<const float4*>(cs + half + j);
    }
    alignas(16) __nv_bfloat162 lo[V / 2], hi[V / 2];
    if constexpr (V == 8) {
      *reinterpret_cast<uint4*>(lo) = *reinterpret_cast<const uint4*>(base);
      *reinterpret_cast<uint4*>(hi) = *reinterpret_cast<const uint4*>(base + half);
    } else {
      *reinterpret_cast<uint2*>(lo) = *reinterpret_cast<const uint2*>(base);
      *reinterpret_cast<uint2*>(hi) = *reinterpret_cast<const uint2*>(base + half);
    }
#pragma unroll
    for (int j = 0; j < V / 2; ++j) {
      const float2 x = __bfloat1622float2(lo[j]), y = __bfloat1622float2(hi[j]);
      a[2 * j] = x.x, a[2 * j + 1] = x.y, b[2 * j] = y.x, b[2 * j + 1] = y.y;
    }
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const float s = sn[j] * sign, u = a[j] * cc[j] - b[j] * s;
      b[j] = b[j] * cc[j] + a[j] * s;
      a[j] = u;
    }
#pragma unroll
    for (int j = 0; j < V / 2; ++j) {
      lo[j] = __floats2bfloat162_rn(a[2 * j], a[2 * j + 1]);
      hi[j] = __floats2bfloat162_rn(b[2 * j], b[2 * j + 1]);
    }
    if constexpr (V == 8) {
      *reinterpret_cast<uint4*>(base) = *reinterpret_cast<const uint4*>(lo);
      *reinterpret_cast<uint4*>(base + half) = *reinterpret_cast<const uint4*>(hi);
    } else {
      *reinterpret_cast<uint2*>(base) = *reinterpret_cast<const uint2*>(lo);
      *reinterpret_cast<uint2*>(base + half) = *reinterpret_cast<const uint2*>(hi);
    }
  }
}

// --------------------------------------------------------------------------------------------
// SwiGLU: in [T, 2F] = [gate | up] -> out [T, F] = silu(gate) * up
// --------------------------------------------------------------------------------------------
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ in,
                                  __nv_bfloat16* __restrict__ out, long long T, int F) {
  const int nvec = F >> 3;
  const long long total = T * nvec;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long t = idx / nvec;
    const int i = (int)(idx % nvec);
    float g[8], u[8], o[8];
    unpack8(ld8(in + t * 2 * F + i * 8), g);
    unpack8(ld8(in + t * 2 * F + F + i * 8), u);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = silu_mul(g[k], u[k]);
    st8(out + t * F + i * 8, pack8(o));
  }
}

// dgate = dy * up * s * (1 + g*(1-s)),  dup = dy * g * s  with s = sigmoid(g); writes [T, 2F].
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ in,
                                  const __nv_bfloat16* __restrict__ dy,
                                  __nv_bfloat16* __restrict__ din, long long T, int F) {
  const int nvec = F >> 3;
  const long long total = T * nvec;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long t = idx / nvec;
    const int i = (int)(idx % nvec);
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(ld8(in + t * 2 * F + i * 8), g);
    unpack8(ld8(in + t * 2 * F + F + i * 8), u);
    unpack8(ld8(dy + t * F + i * 8), d);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float s = 1.f / (1.f + __expf(-g[k]));
      dg[k] = d[k] * u[k] * s * (1.f + g[k] * (1.f - s));
      du[k] = d[k] * g[k] * s;
    }
    st8(din + t * 2 * F + i * 8, pack8(dg));
    st8(din + t * 2 * F + F + i * 8, pack8(du));
  }
}

// out = a + b (bf16), n multiple of 8
__global__ void add_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                           __nv_bfloat16* __restrict__ out, long long nvec) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec;
       i += (long long)gridDim.x * blockDim.x) {
    float x[8], y[8];
    unpack8(ld8(a + i * 8), x);
    unpack8(ld8(b + i * 8), y);
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] += y[k];
    st8(out + i * 8, pack8(x));
  }
}

// Column sums of a [rows, C] bf16 matrix into partial[gridDim.y, C] (bias gradients).
__global__ void colsum_rows_kernel(const __nv_bfloat16* __restrict__ m, long long rows, int C,
                                   float* __restrict__ partial) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  float s = 0.f;
  for (long long r = blockIdx.y; r < rows; r += gridDim.y) s += __bfloat162float(m[r * C + c]);
  partial[(long long)blockIdx.y * C + c] = s;
}

// Embedding gradient: g[id] += sum of the rows d[t] with ids[t] == id, rows of one id added in fp32 in
// token order (no atomics: bit-reproducible).  `order` lists the tokens sorted by id (stable), segment s
// covers order[seg_start[s] .. seg_start[s + 1]) and belongs to row seg_id[s] of g.  One block per
// segment, 16-byte column vectors strided over the threads.
template <typename G>
__global__ void __launch_bounds__(128)
embedding_grad_kernel(const __nv_bfloat16* __restrict__ d, long long ldd, const long long* __restrict__ order,
                      const long long* __restrict__ seg_start, const long long* __restrict__ seg_id,
                      G* __restrict__ g, long long ldg, int H) {
  const long long s = blockIdx.x;
  const long long t0 = seg_start[s], t1 = seg_start[s + 1];
  G* row = g + seg_id[s] * ldg;
  for (int c = threadIdx.x * 8; c < H; c += 128 * 8) {
    float acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0.f;
    for (long long t = t0; t < t1; ++t) {
      float f[8];
      unpack8(ld8(d + order[t] * ldd + c), f);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += f[k];
    }
    if (sizeof(G) == 2) {
      __nv_bfloat16* r16 = reinterpret_cast<__nv_bfloat16*>(row);
      float cur[8];
      unpack8(ld8(r16 + c), cur);
#pragma unroll
      for (int k = 0; k < 8; ++k) cur[k] += acc[k];
      st8(r16 + c, pack8(cur));
    } else {
      float* r32 = reinterpret_cast<float*>(row);
#pragma unroll
      for (int k = 0; k < 8; ++k) r32[c + k] += acc[k];
    }
  }
}

}  // namespace msrl

using namespace msrl;

static inline int grid_for(long long work_items, int threads, int per_sm = 8) {
  long long b = ceil_div(work_items, threads);
  long long cap = (long long)sm_count() * per_sm;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

MSRL_API int msrl_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* sum_out,
                              float* rstd, long long rows, int H, float eps, cudaStream_t st) {
  if (rows == 0) return 0;
  if (H % 8 != 0 || H > 16384) return (int)cudaErrorInvalidValue;
  if (H <= 32 * 16 * 8 && rows >= 4LL * sm_count()) {        // the usual hidden sizes, enough rows: a warp per row
    const long long cap = (long long)sm_count() * 3;        // three blocks fit the registers of an SM
    const long long want = (rows + 3) / 4;
    const unsigned blocks = (unsigned)(want < cap ? want : cap);
#define MSRL_RMS_WARP(V, R)                                                                            \
    rmsnorm_fwd_warp_kernel<V, R><<<blocks, 128, 0, st>>>(                                             \
        (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w, (__nv_bfloat16*)y, \
        (__nv_bfloat16*)sum_out, rstd, rows, H, eps)
    if (res != nullptr) {
      if (H <= 32 * 8 * 8) MSRL_RMS_WARP(8, true);
      else if (H <= 32 * 14 * 8) MSRL_RMS_WARP(14, true);
      else MSRL_RMS_WARP(16, true);
    } else {
      if (H <= 32 * 8 * 8) MSRL_RMS_WARP(8, false);
      else if (H <= 32 * 14 * 8) MSRL_RMS_WARP(14, false);
      else MSRL_RMS_WARP(16, false);
    }
#undef MSRL_RMS_WARP
    MSRL_LAUNCH_CHECK();
  }
  if (H <= 256 * 4 * 8) {        // few rows (decode steps) or wider rows: a block per row, the row in registers
    // one wave of persistent blocks: four 128-thread (two 256-thread) blocks fit the registers of an SM
    const long long cap = (long long)sm_count() * (H <= 128 * 4 * 8 ? 4 : 2);
    const unsigned blocks = (unsigned)(rows < cap ? rows : cap);
    // Up to two rows to an SM a row takes its latency: one vector a thread and the weights ahead of the sum (3584 wide, residual: 1
    // row 3.0 -> 2.4 us, 48 x 2048 2.7 -> 2.2, 256 rows 3.75 -> 3.66; 500 rows 4.5 -> 5.7, which stay with four vectors).
    if (H <= 512 * 8 && rows <= 2LL * sm_count())
      rmsnorm_fwd_regs_kernel<512, 1><<<blocks, 512, 0, st>>>(
          (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w,
          (__nv_bfloat16*)y, (__nv_bfloat16*)sum_out, rstd, rows, H, eps);
    else if (H <= 128 * 4 * 8)
      rmsnorm_fwd_regs_kernel<128, 4><<<blocks, 128, 0, st>>>(
          (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w,
          (__nv_bfloat16*)y, (__nv_bfloat16*)sum_out, rstd, rows, H, eps);
    else
      rmsnorm_fwd_regs_kernel<256, 4><<<blocks, 256, 0, st>>>(
          (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w,
          (__nv_bfloat16*)y, (__nv_bfloat16*)sum_out, rstd, rows, H, eps);
    MSRL_LAUNCH_CHECK();
  }
  size_t smem = (size_t)H * sizeof(float);
  static bool attr_set = false;
  if (!attr_set) {
    cudaFuncSetAttribute(rmsnorm_fwd_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, 65536);
    attr_set = true;
  }
  rmsnorm_fwd_kernel<256><<<(unsigned)rows, 256, smem, st>>>(
      (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w,
      (__nv_bfloat16*)y, (__nv_bfloat16*)sum_out, rstd, H, eps);
  MSRL_LAUNCH_CHECK();
}

// Number of blocks (= rows of the dw scratch) the backward uses for a given problem.
MSRL_API int msrl_rmsnorm_bwd_blocks(long long rows) {
  // two blocks to an SM, kernel alone, 32768 x 3584: one 281 us, two 182, three 233, four 186 (the partial sums cost cap x H floats);
  // above 4096 columns one of the two is resident at a time, which is still the faster form (see the kernel)
  long long cap = (long long)sm_count() * 2;
  return (int)(rows < cap ? (rows < 1 ? 1 : rows) : cap);
}

// dw_partial: fp32 scratch of msrl_rmsnorm_bwd_blocks(rows) * H elements.
// dw_f32 / dw_bf16: either may be null; `accumulate` adds to the existing value.
MSRL_API int msrl_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd,
                              const void* dres, void* dx, float* dw_partial, float* dw_f32,
                              void* dw_bf16, int accumulate, long long rows, int H,
                              cudaStream_t st) {
  if (rows == 0) return 0;
  if (H % 8 != 0 || H > 8192) return (int)cudaErrorInvalidValue;
  const int nb = msrl_rmsnorm_bwd_blocks(rows);
  const int nvec = H / 8;
#define LAUNCH_BWD(VPT)                                                                        \
  rmsnorm_bwd_kernel<256, VPT><<<nb, 256, 0, st>>>(                                            \
      (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, rstd,        \
      (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx, dw_partial, rows, H)
  if (nvec <= 256) LAUNCH_BWD(1);
  else if (nvec <= 512) LAUNCH_BWD(2);
  else if (nvec <= 768) LAUNCH_BWD(3);
  else LAUNCH_BWD(4);
#undef LAUNCH_BWD
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  colsum_partials_kernel<<<(H + 31) / 32, COLSUM_WARPS * 32, 0, st>>>(dw_partial, nb, H, dw_f32,
                                                          (__nv_bfloat16*)dw_bf16, accumulate);
  MSRL_LAUNCH_CHECK();
}

// tokens whose heads count in 32 bits (with room for the last block's)
static long long head_chunk(int nheads) { return nheads <= 1 ? 1 << 30 : nheads >= (1 << 30) ? 1 : (1 << 30) / nheads; }

MSRL_API int msrl_headnorm_fwd(const void* x, long long stride_t, int group_stride, int hpg,
                               int head_stride, const void* w, void* y, float* rstd, long long T,
                               int nheads, int hd, float eps, cudaStream_t st) {
  if (T == 0) return 0;
  if (hd % 8 != 0 || hd > 256) return (int)cudaErrorInvalidValue;
  HeadLayout L{stride_t, group_stride, hpg, head_stride};
  const int g = hd <= 64 ? 8 : hd <= 128 ? 16 : 32;
  const int u = T * nheads <= 32LL * sm_count() ? 1 : 4;
  auto* kernel = g == 8    ? (u == 1 ? headnorm_fwd_kernel<8, 1> : headnorm_fwd_kernel<8, 4>)
                 : g == 16 ? (u == 1 ? headnorm_fwd_kernel<16, 1> : headnorm_fwd_kernel<16, 4>)
                           : (u == 1 ? headnorm_fwd_kernel<32, 1> : headnorm_fwd_kernel<32, 4>);
  const long long chunk = head_chunk(nheads);
  for (long long t0 = 0; t0 < T; t0 += chunk) {
    const unsigned heads = (unsigned)(T - t0 < chunk ? T - t0 : chunk) * (unsigned)nheads;
    kernel<<<(unsigned)ceil_div(heads, u * 256 / g), 256, 0, st>>>(
        (const __nv_bfloat16*)x + t0 * stride_t, L, (const __nv_bfloat16*)w, (__nv_bfloat16*)y + t0 * stride_t,
        rstd != nullptr ? rstd + t0 * nheads : nullptr, heads, nheads, hd, eps);
  }
  MSRL_LAUNCH_CHECK();
}

MSRL_API int msrl_headnorm_bwd_blocks() { return sm_count() * 4; }

MSRL_API int msrl_headnorm_bwd(void* dy_dx, const void* x, long long stride_t, int group_stride,
                               int hpg, int head_stride, const void* w, const float* rstd,
                               float* dw_partial, float* dw_f32, void* dw_bf16, int accumulate,
                               long long T, int nheads, int hd, cudaStream_t st) {
  if (T == 0) return 0;
  if (hd % 8 != 0 || hd > 256) return (int)cudaErrorInvalidValue;
  HeadLayout L{stride_t, group_stride, hpg, head_stride};
  const int nb = msrl_headnorm_bwd_blocks();
  auto* kernel = hd <= 64 ? headnorm_bwd_kernel<8> : hd <= 128 ? headnorm_bwd_kernel<16> : headnorm_bwd_kernel<32>;
  kernel<<<nb, 256, 0, st>>>((__nv_bfloat16*)dy_dx, (const __nv_bfloat16*)x, L, (const __nv_bfloat16*)w, rstd, dw_partial,
                             T, head_chunk(nheads), nheads, hd);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  colsum_partials_kernel<<<(hd + 31) / 32, COLSUM_WARPS * 32, 0, st>>>(dw_partial, nb, hd, dw_f32,
                                                           (__nv_bfloat16*)dw_bf16, accumulate);
  MSRL_LAUNCH_CHECK();
}

MSRL_API int msrl_rope(void* q, long long q_stride_t, int q_group_stride, int q_hpg,
                       int q_head_stride, int nq, void* k, long long k_stride_t, int k_group_stride,
                       int k_hpg, int k_head_stride, int nk, const int* positions,
                       const float* cos_sin, long long T, int hd, float sign, cudaStream_t st) {
  if (T == 0) return 0;
  if (hd % 8 != 0) return (int)cudaErrorInvalidValue;
  HeadLayout Lq{q_stride_t, q_group_stride, q_hpg, q_head_stride};
  HeadLayout Lk{k_stride_t, k_group_stride, k_hpg > 0 ? k_hpg : 1, k_head_stride};
  const bool wide = hd % 16 == 0 && ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k)) & 15) == 0 &&
                    (q_stride_t | k_stride_t | q_group_stride | k_group_stride | q_head_stride | k_head_stride) % 8 == 0;
  const long long per_token = (long long)(nq + nk) * (hd / (wide ? 16 : 8));
  if (per_token == 0) return 0;
  if (per_token > (1 << 30)) return (int)cudaErrorInvalidValue;
  const long long chunk = (1 << 30) / per_token;            // tokens whose vectors count in 32 bits
  for (long long t0 = 0; t0 < T; t0 += chunk) {
    const unsigned total = (unsigned)((T - t0 < chunk ? T - t0 : chunk) * per_token), all = (total + 255) / 256;
    const unsigned blocks = wide ? all : (unsigned)grid_for(total, 256);
    auto* kernel = wide ? rope_kernel<8> : rope_kernel<4>;
    kernel<<<blocks, 256, 0, st>>>((__nv_bfloat16*)q + t0 * q_stride_t, Lq, nq, (__nv_bfloat16*)k + t0 * k_stride_t, Lk, nk,
                                   positions + t0, cos_sin, total, hd, sign);
  }
  MSRL_LAUNCH_CHECK();
}

MSRL_API int msrl_swiglu_fwd(const void* in, void* out, long long T, int F, cudaStream_t st) {
  if (T == 0) return 0;
  if (F % 8 != 0) return (int)cudaErrorInvalidValue;
  swiglu_fwd_kernel<<<grid_for(T * (F / 8), 256), 256, 0, st>>>((const __nv_bfloat16*)in,
                                                                (__nv_bfloat16*)out, T, F);
  MSRL_LAUNCH_CHECK();
}

MSRL_API int msrl_swiglu_bwd(const void* in, const void* dy, void* din, long long T, int F,
                             cudaStream_t st) {
  if (T == 0) return 0;
  if (F % 8 != 0) return (int)cudaErrorInvalidValue;
  swiglu_bwd_kernel<<<grid_for(T * (F / 8), 256), 256, 0, st>>>(
      (const __nv_bfloat16*)in, (const __nv_bfloat16*)dy, (__nv_bfloat16*)din, T, F);
  MSRL_LAUNCH_CHECK();
}

MSRL_API int msrl_add(const void* a, const void* b, void* out, long long n, cudaStream_t st) {
  if (n == 0) return 0;
  if (n % 8 != 0) return (int)cudaErrorInvalidValue;
  add_kernel<<<grid_for(n / 8, 256), 256, 0, st>>>((const __nv_bfloat16*)a, (const __nv_bfloat16*)b,
                                                   (__nv_bfloat16*)out, n / 8);
  MSRL_LAUNCH_CHECK();
}

MSRL_API int msrl_colsum_blocks() { return 64; }

// Bias gradient: out[c] (+)= sum_r m[r, c]; partial is fp32 scratch [msrl_colsum_blocks(), C].
MSRL_API int msrl_colsum(const void* m, long long rows, int C, float* partial, float* out_f32,
                         void* out_bf16, int accumulate, cudaStream_t st) {
  if (rows == 0 || C == 0) return 0;
  const int nb = msrl_colsum_blocks();
  dim3 grid((C + 127) / 128, nb);
  colsum_rows_kernel<<<grid, 128, 0, st>>>((const __nv_bfloat16*)m, rows, C, partial);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  colsum_partials_kernel<<<(C + 31) / 32, COLSUM_WARPS * 32, 0, st>>>(partial, nb, C, out_f32,
                                                          (__nv_bfloat16*)out_bf16, accumulate);
  MSRL_LAUNCH_CHECK();
}

// g[seg_id[s]] += sum over t in [seg_start[s], seg_start[s+1]) of d[order[t]]   (see embedding_grad_kernel).
// d bf16 [T, H] (row pitch ldd), g bf16 or fp32 [V, H] (row pitch ldg); H a multiple of 8, rows 16-byte aligned.
MSRL_API int msrl_embedding_grad(const void* d, long long ldd, const long long* order, const long long* seg_start,
                                 const long long* seg_id, long long n_seg, void* g, long long ldg, int g_is_f32,
                                 int H, cudaStream_t st) {
  if (n_seg == 0) return 0;
  if (H % 8 != 0 || ldd % 8 != 0 || ldg % 8 != 0 || n_seg > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
  if (g_is_f32)
    embedding_grad_kernel<float><<<(unsigned)n_seg, 128, 0, st>>>((const __nv_bfloat16*)d, ldd, order, seg_start,
                                                                  seg_id, (float*)g, ldg, H);
  else
    embedding_grad_kernel<__nv_bfloat16><<<(unsigned)n_seg, 128, 0, st>>>((const __nv_bfloat16*)d, ldd, order,
                                                                          seg_start, seg_id, (__nv_bfloat16*)g, ldg, H);
  MSRL_LAUNCH_CHECK();
}
