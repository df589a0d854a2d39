// Flash attention backward for heads of 128 (included by attention_tcgen05.cu).  Two kernels without atomics, bit-reproducible:
//   fa_bwd_dkdv_kernel   block = 128 keys of one KV head, loop over the query heads of the group and their 128-row query tiles:
//                        S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q; dK and dV stay in TMEM;
//   fa_bwd_dq_kernel     block = 128 query rows of one head, loop over 128-key tiles: S = Q K^T, dP = dO V^T, dQ += dS K.
// P is recomputed from the saved log-sum-exp; delta = rowsum(dO o O) comes from a small kernel.
//
// P and dS (bf16) go back to TMEM over the scores they came from and are read there as the A operand; no tile of them passes
// through shared memory.  The 128 x 128 products read their operands from shared memory at just the rate of the tensor cores
// (the 128 x 64 ones of smaller tiles are bound by those reads), the ones with A in TMEM at half of it.  Eight soft-max warps:
// two threads to a TMEM lane, 64 columns each; a thread's P lies in the first 32 columns of its own scores, so that none is
// overwritten before its owner has read it.  (Sixteen warps with 32 columns each: the same.)
//
// Bound by: 2048 (dK/dV) and 1536 (dQ) tensor-core cycles per pair of tiles beside 1024 cycles of exponentials, at the clock the
// power limit leaves (1.62 GHz; the tensor pipe is busy 72 % of the time in dK/dV).  Both kernels and delta, causal, 28 heads over
// 4, before (64-key tiles, P and dS through shared memory) and now: 22528 + 7361 + 2879 tokens 15617 -> 12400 us, 1280 + 3072 +
// 1863 + 2201 tokens 836 -> 553 us, eight of 1024 483 -> 360 us.
#pragma once

namespace msrl {
namespace fa5 {

constexpr int BWD_WARPS = 8, BWD_TMA = 8, BWD_MMA = 9, BWD_THREADS = 320;      // warps 0-7 soft-max, 8 TMA, 9 MMA
constexpr int NC = 64;                                 // columns of a soft-max thread: 128 over two warpgroups
// Two resident tiles (K, V or Q, dO) and stages of the two that stream by.
constexpr uint32_t BWD_A = 0, BWD_B = TILE_BYTES, BWD_X = 2 * TILE_BYTES, DKDV_Y = 4 * TILE_BYTES, DKDV_SMEM = 6 * TILE_BYTES;
// dQ: three stages of K, which the last product of a step frees and the next but one step reads first (with two, every step waited
// for its K: 666 us against 528 for one sequence of 8192, 28 heads over 4).
constexpr uint32_t DQ_Y = 5 * TILE_BYTES, DQ_SMEM = 7 * TILE_BYTES;
constexpr float LOG2E = 1.4426950408889634f;

struct BwdParams {
  const __nv_bfloat16* o;
  const __nv_bfloat16* dout;
  long long o_stride_t;
  const float* lse;      // [nh, Tq], natural log
  float* delta;          // [nh, Tq]
  __nv_bfloat16* dq;
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  long long q_stride_t, k_stride_t, v_stride_t;
  const int* cu_q;
  const int* cu_k;
  int nh, nkv, batch;
  long long Tq;
  float scale, scale_log2;
  int causal;
  int q_group_stride, q_hpg, q_head_stride;
  int k_group_stride, k_hpg, k_head_stride;
  int v_group_stride, v_hpg, v_head_stride;
  int* error;
};

// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d]; one warp per (t, h), head size 128.
__global__ void fa_delta128_kernel(const BwdParams p) {
  const long long w = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= p.Tq * p.nh) return;
  const long long t = w / p.nh;
  const int h = (int)(w % p.nh);
  const long long base = t * p.o_stride_t + (long long)h * D + lane * 4;
  const uint2 a = *reinterpret_cast<const uint2*>(p.o + base);
  const uint2 b = *reinterpret_cast<const uint2*>(p.dout + base);
  const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&a);
  const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&b);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float2 x = __bfloat1622float2(a2[i]), y = __bfloat1622float2(b2[i]);
    s += x.x * y.x + x.y * y.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) p.delta[(long long)h * p.Tq + t] = s;
}

// One warp's 32 TMEM lanes x 64 accumulator columns -> bf16, through a shared-memory patch, stored
// as whole 128-byte row segments.  `dst` points at (first row of the warp, first of the 64 columns).
__device__ __forceinline__ void store_half_tile(uint32_t taddr, float scale, bool zero, unsigned char* patch, int lane,
                                                __nv_bfloat16* dst, long long row_stride, int rows_valid) {
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    float v[32];
    if (!zero) {
      tmem_ld32(taddr + hh * 32, v);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] *= scale;
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = 0.f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<bf16x8*>(patch + lane * OUT_PITCH + hh * 64 + q * 16) = pack8(v + q * 8);
  }
  __syncwarp();
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int r = it * 4 + (lane >> 3);
    if (r < rows_valid)
      st8(dst + (long long)r * row_stride + (lane & 7) * 8,
          *reinterpret_cast<const bf16x8*>(patch + r * OUT_PITCH + (lane & 7) * 16));
  }
  __syncwarp();
}

// tmem_c (+)= A B^T over a head of 128, both tiles [128 rows, 128] K-major in shared memory
__device__ __forceinline__ void tile_product(uint32_t tmem_c, uint32_t a, uint32_t b) {
  constexpr uint32_t id = idesc_bf16(BM, 128, false);
#pragma unroll
  for (int kk = 0; kk < 8; ++kk)
    umma(tmem_c, desc_sw128(a + (kk >> 2) * TILE_HALF + (kk & 3) * 32, 16, 1024),
         desc_sw128(b + (kk >> 2) * TILE_HALF + (kk & 3) * 32, 16, 1024), id, kk > 0 ? 1u : 0u);
}
// tmem_c (+)= A B for 16 of the 128 inner rows: A bf16 in TMEM (NC to a soft-max thread, in the first half of its columns),
// B [128 inner rows, 128] MN-major in shared memory
__device__ __forceinline__ void tmem_step(uint32_t tmem_c, uint32_t tmem_a, uint32_t b, int kk, bool add) {
  constexpr uint32_t id = idesc_bf16(BM, D, true);
  umma_ts(tmem_c, tmem_a + kk * 16 / NC * NC + kk * 16 % NC / 2, desc_sw128(b + kk * 2048, TILE_HALF, 1024), id, add ? 1u : 0u);
}

__device__ __forceinline__ uint32_t pack_bf16(float2 v) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// SPLITS blocks of one cluster (or one block alone) share a key tile, each with a contiguous part of its (query head, query tile)
// list; their dK and dV meet in shared memory at the end, added in rank order.
template <int SPLITS>
__global__ void __launch_bounds__(BWD_THREADS, 1)
fa_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                   const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                   const __grid_constant__ BwdParams p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ uint64_t kv_full, q_full[2], q_empty[2], do_full[2], do_empty[2], s_full, dp_full, p_part[2], ds_ready, done;
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(16) float stat[2][2][128];        // per stage: -lse (exp2 domain) and -delta of its query rows

  const int rank = blockIdx.x % SPLITS, work = blockIdx.x / SPLITS;
  const int hk = work % p.nkv, b = work / p.nkv % p.batch, kb = work / p.nkv / p.batch * BM;   // first key of this block
  const int q0 = p.cu_q[b], qlen = p.cu_q[b + 1] - q0;
  const int k0 = p.cu_k[b], klen = p.cu_k[b + 1] - k0;
  if (kb >= klen) return;                                 // the whole cluster
  const int rep = p.nh / p.nkv, off = klen - qlen;
  // query tiles that see any of these keys: rows r with r + off >= kb (causal), r < qlen
  const int i_start = p.causal ? max(0, kb - off) / BM : 0;
  const int nq = max(0, (qlen + BM - 1) / BM - i_start), all = nq * rep;
  const int first = (int)((long long)all * rank / SPLITS), n_it = (int)((long long)all * (rank + 1) / SPLITS) - first;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(&kv_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&do_full[i], 1);
      mbar_init(&do_empty[i], 1);
      mbar_init(&p_part[i], BWD_WARPS);
    }
    mbar_init(&s_full, 1);
    mbar_init(&dp_full, 1);
    mbar_init(&ds_ready, BWD_WARPS);
    mbar_init(&done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == BWD_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;                        // S^T (P^T), dP^T (dS^T), dV, dK: 128 columns each
  const uint32_t tm_dp = tmem + 128, tm_dv = tmem + 256, tm_dk = tmem + 384;
  bool ok = true;

  if (warp == BWD_TMA) {
    // one lane issues the loads; all lanes bring the per-query statistics, which are read before the wait for their place
    const int kc = head_col(0, p.k_group_stride, p.k_hpg, p.k_head_stride, hk);
    const int vc = head_col(0, p.v_group_stride, p.v_hpg, p.v_head_stride, hk);
    for (int n = 0; n < n_it; ++n) {
      const int st = n & 1;
      const uint32_t use = n >> 1;
      const int hq = hk * rep + (first + n) / nq, qr = (i_start + (first + n) % nq) * BM;
      float l[4], d[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int q = qr + i * 32 + lane;
        const long long at = (long long)hq * p.Tq + q0 + q;
        l[i] = q < qlen ? -__ldg(p.lse + at) * LOG2E : -INFINITY;      // P is exactly 0
        d[i] = q < qlen ? -__ldg(p.delta + at) : 0.f;
      }
      if (use > 0 && !mbar_wait_warp(&q_empty[st], (use - 1) & 1, p.error, ERR_EMPTY)) break;   // all lanes or none
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        stat[st][0][i * 32 + lane] = l[i];
        stat[st][1][i * 32 + lane] = d[i];
      }
      __syncwarp();
      if (lane == 0) {
        if (n == 0) {
          mbar_expect_tx(&kv_full, 2 * TILE_BYTES);
          for (int i = 0; i < 2; ++i) tma_load_2d(smem + BWD_A + i * TILE_HALF, &map_k, &kv_full, kc + i * 64, k0 + kb);
        }
        const int qc = head_col(0, p.q_group_stride, p.q_hpg, p.q_head_stride, hq);
        mbar_expect_tx(&q_full[st], TILE_BYTES);
        for (int i = 0; i < 2; ++i)
          tma_load_2d(smem + BWD_X + st * TILE_BYTES + i * TILE_HALF, &map_q, &q_full[st], qc + i * 64, q0 + qr);
        if (n == 0)
          for (int i = 0; i < 2; ++i) tma_load_2d(smem + BWD_B + i * TILE_HALF, &map_v, &kv_full, vc + i * 64, k0 + kb);
        if (use > 0) ok = mbar_wait(&do_empty[st], (use - 1) & 1, p.error, ERR_EMPTY);
        if (ok) {
          mbar_expect_tx(&do_full[st], TILE_BYTES);
          for (int i = 0; i < 2; ++i)
            tma_load_2d(smem + DKDV_Y + st * TILE_BYTES + i * TILE_HALF, &map_do, &do_full[st], hq * D + i * 64, q0 + qr);
        }
      }
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
      if (!ok) break;
    }
  } else if (warp == BWD_MMA) {
    if (elect_one() && n_it > 0) {
      const uint32_t base = smem_u32(smem);
      auto scores = [&](int n) {                           // S^T[keys, q]
        ok = ok && mbar_wait(&q_full[n & 1], (n >> 1) & 1, p.error, ERR_Q);
        if (!ok) return;
        fence_after();
        tile_product(tmem, base + BWD_A, base + BWD_X + (n & 1) * TILE_BYTES);
        commit(&s_full);
      };
      auto dprobs = [&](int n) {                           // dP^T[keys, q]
        ok = ok && mbar_wait(&do_full[n & 1], (n >> 1) & 1, p.error, ERR_Q);
        if (!ok) return;
        fence_after();
        tile_product(tm_dp, base + BWD_B, base + DKDV_Y + (n & 1) * TILE_BYTES);
        commit(&dp_full);
      };
      ok = mbar_wait(&kv_full, 0, p.error, ERR_K);
      scores(0);
      dprobs(0);
      for (int n = 0; n < n_it && ok; ++n) {
        const int st = n & 1;
        const uint32_t q_addr = base + BWD_X + st * TILE_BYTES, do_addr = base + DKDV_Y + st * TILE_BYTES;
        // Sixteens of queries that see none of the keys are left out: their P and dS are 0, but 0 times an inf or nan of dO or Q
        // would reach dV and dK.  Tested once a tile, in front of steps without a branch.
        const int qr = (i_start + (first + n) % nq) * BM, from = (p.causal ? max(kb - off - qr, 0) : 0) - 15, to = qlen - qr;
        const bool whole = from <= 0 && to > 112;
        bool add = n > 0;
        // dV += P^T dO, the first half of each thread's columns as soon as it is there
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          ok = ok && mbar_wait(&p_part[part], n & 1, p.error, ERR_P);
          if (!ok) break;
          fence_after();
          if (whole) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              tmem_step(tm_dv, tmem, do_addr, (i >> 1) * 4 + part * 2 + (i & 1), n > 0 || part > 0 || i > 0);
          } else {
#pragma unroll 1
            for (int i = 0; i < 4; ++i) {
              const int kk = (i >> 1) * 4 + part * 2 + (i & 1);
              if (kk * 16 < from || kk * 16 >= to) continue;
              tmem_step(tm_dv, tmem, do_addr, kk, add);
              add = true;
            }
          }
        }
        if (!ok) break;
        commit(&do_empty[st]);                             // dP of this tile is older
        if (n + 1 < n_it) scores(n + 1);                   // over P, which the products before it have read
        ok = ok && mbar_wait(&ds_ready, n & 1, p.error, ERR_P);
        if (!ok) break;
        fence_after();
        // dK += dS^T Q
        if (whole) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) tmem_step(tm_dk, tm_dp, q_addr, kk, n > 0 || kk > 0);
        } else {
#pragma unroll 1
          for (int kk = 0; kk < 8; ++kk)
            if (kk * 16 >= from && kk * 16 < to) tmem_step(tm_dk, tm_dp, q_addr, kk, n > 0 || kk * 16 >= from + 16);
        }
        commit(&q_empty[st]);
        if (n + 1 < n_it) dprobs(n + 1);
      }
      if (ok) commit(&done);
    }
  } else if (warp < BWD_WARPS) {
    const int wg = warp >> 2, quarter = warp & 3;
    const int key = kb + quarter * 32 + lane;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    const uint32_t ts = tmem + lanes + wg * 64, tdp = tm_dp + lanes + wg * 64;
    const f2 scale2 = pack2(p.scale_log2, p.scale_log2);
    for (int n = 0; n < n_it; ++n) {
      const int st = n & 1, qr = (i_start + (first + n) % nq) * BM;
      // the statistics were written before the arrival on this barrier
      ok = mbar_wait_warp(&q_full[st], (n >> 1) & 1, p.error, ERR_Q) && mbar_wait_warp(&s_full, n & 1, p.error, ERR_S);
      if (!ok) break;
      fence_after();
      float s[64];
      tmem_ld_cols<64>(ts, s);
      const float* nl = &stat[st][0][wg * 64];
      const float* nd = &stat[st][1][wg * 64];
      // query column i (of this thread) sees this key iff key <= qr + wg * 64 + i + off
      const bool masked = p.causal && kb + BM - 1 - off > qr;
      const int from = masked ? key - off - qr - wg * 64 : 0;
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const int c = part * 32 + 2 * i;
          const float4 l = *reinterpret_cast<const float4*>(nl + c);
          float2 a = unpack2(fma2(pack2(s[c], s[c + 1]), scale2, pack2(l.x, l.y)));
          float2 e = unpack2(fma2(pack2(s[c + 2], s[c + 3]), scale2, pack2(l.z, l.w)));
          a = make_float2(ex2(a.x), ex2(a.y));
          e = make_float2(ex2(e.x), ex2(e.y));
          if (masked) {
            a.x = c >= from ? a.x : 0.f;
            a.y = c + 1 >= from ? a.y : 0.f;
            e.x = c + 2 >= from ? e.x : 0.f;
            e.y = c + 3 >= from ? e.y : 0.f;
          }
          s[c] = a.x, s[c + 1] = a.y, s[c + 2] = e.x, s[c + 3] = e.y;
          packed[i] = pack_bf16(a);
          packed[i + 1] = pack_bf16(e);
        }
        tmem_st_cols(ts + part * 16, packed);
        tmem_wait_st();
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_part[part]);
      }
      ok = mbar_wait_warp(&dp_full, n & 1, p.error, ERR_S);
      if (!ok) break;
      fence_after();
      float dp[64];
      tmem_ld_cols<64>(tdp, dp);
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const int c = part * 32 + 2 * i;
          const float4 d = *reinterpret_cast<const float4*>(nd + c);
          packed[i] = pack_bf16(unpack2(mul2(pack2(s[c], s[c + 1]), add2(pack2(dp[c], dp[c + 1]), pack2(d.x, d.y)))));
          packed[i + 1] =
              pack_bf16(unpack2(mul2(pack2(s[c + 2], s[c + 3]), add2(pack2(dp[c + 2], dp[c + 3]), pack2(d.z, d.w)))));
        }
        tmem_st_cols(tdp + part * 16, packed);
      }
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ds_ready);
    }
    if (ok && n_it > 0) ok = mbar_wait_warp(&done, 0, p.error, ERR_PV);
    if (ok && n_it > 0) fence_after();
    const int kc = head_col(0, p.k_group_stride, p.k_hpg, p.k_head_stride, hk);
    const int vc = head_col(0, p.v_group_stride, p.v_hpg, p.v_head_stride, hk);
    if constexpr (SPLITS == 1) {
      if (ok) {
        unsigned char* patch = smem + warp * (32 * OUT_PITCH);
        const int rows_valid = klen - (kb + quarter * 32);
        const long long row = k0 + kb + quarter * 32;
        store_half_tile(tm_dv + lanes + wg * 64, 1.f, n_it == 0, patch, lane, p.dv + row * p.v_stride_t + vc + wg * 64,
                        p.v_stride_t, rows_valid);
        store_half_tile(tm_dk + lanes + wg * 64, p.scale, n_it == 0, patch, lane, p.dk + row * p.k_stride_t + kc + wg * 64,
                        p.k_stride_t, rows_valid);
      }
    } else {
      // this block's sums in fp32, rows of 512 bytes, chunks of 16 bytes XORed with the row
      const int row = quarter * 32 + lane;
#pragma unroll
      for (int which = 0; which < 2; ++which) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float v[32];
          if (n_it > 0 && ok) {
            tmem_ld32((which ? tm_dk : tm_dv) + lanes + wg * 64 + c * 32, v);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0.f;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i)
            *reinterpret_cast<float4*>(smem + which * 65536 + row * 512 + (((wg * 16 + c * 8 + i) ^ lane) << 4)) =
                make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
      }
    }
  }
  if constexpr (SPLITS > 1) {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    // rank r adds up and stores its share of the rows; 16 threads to a row, 8 columns each
    constexpr int per = BM / SPLITS;
    const int col = threadIdx.x & 15;
    const uint32_t base = smem_u32(smem);
    for (int i = threadIdx.x >> 4; i < 2 * per; i += BWD_THREADS / 16) {
      const int which = i / per, row = rank * per + i % per;
      if (kb + row >= klen) continue;
      float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int r = 0; r < SPLITS; ++r) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t at;
          const uint32_t mine = base + which * 65536 + row * 512 + (((col * 2 + c) ^ (row & 31)) << 4);
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(mine), "r"(r));
          float4 x;
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                       : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(at) : "memory");
          v[4 * c] += x.x, v[4 * c + 1] += x.y, v[4 * c + 2] += x.z, v[4 * c + 3] += x.w;
        }
      }
      const long long t = k0 + kb + row;
      if (which) {
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] *= p.scale;
        st8(p.dk + t * p.k_stride_t + head_col(0, p.k_group_stride, p.k_hpg, p.k_head_stride, hk) + col * 8, pack8(v));
      } else {
        st8(p.dv + t * p.v_stride_t + head_col(0, p.v_group_stride, p.v_hpg, p.v_head_stride, hk) + col * 8, pack8(v));
      }
    }
    __syncwarp();
    // no block leaves while others read its sums
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  }
  fence_before();
  __syncthreads();
  if (warp == BWD_MMA) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
  }
}

__global__ void __launch_bounds__(BWD_THREADS, 1)
fa_bwd_dq_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                 const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                 const __grid_constant__ BwdParams p, const int tiles) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ uint64_t qdo_full, k_full[3], k_empty[3], v_full[2], v_empty[2], s_full[2], dp_full, dp_free, ds_ready, done;
  __shared__ uint32_t tmem_slot;

  // longest key ranges first
  const int h = blockIdx.x % p.nh, b = blockIdx.x / p.nh % p.batch, m0 = (tiles - 1 - blockIdx.x / p.nh / p.batch) * BM;
  const int q0 = p.cu_q[b], qlen = p.cu_q[b + 1] - q0;
  const int k0 = p.cu_k[b], klen = p.cu_k[b + 1] - k0;
  if (m0 >= qlen) return;
  const int hk = h / (p.nh / p.nkv), off = klen - qlen;
  const int kmax = p.causal ? min(klen, m0 + BM + off) : klen;
  const int n_tiles = (max(kmax, 0) + 127) / 128;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(&qdo_full, 1);
    for (int i = 0; i < 3; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
    }
    mbar_init(&dp_full, 1);
    mbar_init(&dp_free, BWD_WARPS);
    mbar_init(&ds_ready, BWD_WARPS);
    mbar_init(&done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == BWD_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;                        // S (dS) in turn at 0 and 128, dP 256, dQ 384
  const uint32_t tm_dp = tmem + 256, tm_dq = tmem + 384;

  if (warp == BWD_TMA) {
    if (elect_one() && n_tiles > 0) {
      const int qc = head_col(0, p.q_group_stride, p.q_hpg, p.q_head_stride, h);
      const int kc = head_col(0, p.k_group_stride, p.k_hpg, p.k_head_stride, hk);
      const int vc = head_col(0, p.v_group_stride, p.v_hpg, p.v_head_stride, hk);
      mbar_expect_tx(&qdo_full, 2 * TILE_BYTES);
      for (int i = 0; i < 2; ++i) tma_load_2d(smem + BWD_A + i * TILE_HALF, &map_q, &qdo_full, qc + i * 64, q0 + m0);
      for (int i = 0; i < 2; ++i) tma_load_2d(smem + BWD_B + i * TILE_HALF, &map_do, &qdo_full, h * D + i * 64, q0 + m0);
      for (int j = 0; j < n_tiles; ++j) {
        const int sk = j % 3, sv = j & 1;
        if (j >= 3 && !mbar_wait(&k_empty[sk], (j / 3 - 1) & 1, p.error, ERR_EMPTY)) break;
        mbar_expect_tx(&k_full[sk], TILE_BYTES);
        for (int i = 0; i < 2; ++i)
          tma_load_2d(smem + BWD_X + sk * TILE_BYTES + i * TILE_HALF, &map_k, &k_full[sk], kc + i * 64, k0 + j * 128);
        if (j >= 2 && !mbar_wait(&v_empty[sv], ((j >> 1) - 1) & 1, p.error, ERR_EMPTY)) break;
        mbar_expect_tx(&v_full[sv], TILE_BYTES);
        for (int i = 0; i < 2; ++i)
          tma_load_2d(smem + DQ_Y + sv * TILE_BYTES + i * TILE_HALF, &map_v, &v_full[sv], vc + i * 64, k0 + j * 128);
      }
    }
  } else if (warp == BWD_MMA) {
    if (elect_one() && n_tiles > 0) {
      const uint32_t base = smem_u32(smem);
      bool ok = mbar_wait(&qdo_full, 0, p.error, ERR_Q);
      auto scores = [&](int j) {                           // over dS of tile j - 2, which the product with K has read
        ok = ok && mbar_wait(&k_full[j % 3], (j / 3) & 1, p.error, ERR_K);
        if (!ok) return;
        fence_after();
        tile_product(tmem + (j & 1) * 128, base + BWD_A, base + BWD_X + j % 3 * TILE_BYTES);
        commit(&s_full[j & 1]);
      };
      auto dprobs = [&](int j) {
        ok = ok && mbar_wait(&v_full[j & 1], (j >> 1) & 1, p.error, ERR_V);
        if (ok && j > 0) ok = mbar_wait(&dp_free, (j - 1) & 1, p.error, ERR_S);
        if (!ok) return;
        fence_after();
        tile_product(tm_dp, base + BWD_B, base + DQ_Y + (j & 1) * TILE_BYTES);
        commit(&dp_full);
        commit(&v_empty[j & 1]);
      };
      scores(0);
      dprobs(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles) {
          scores(j + 1);
          dprobs(j + 1);
        }
        ok = ok && mbar_wait(&ds_ready, j & 1, p.error, ERR_P);
        if (!ok) break;
        fence_after();
        const uint32_t k_addr = base + BWD_X + j % 3 * TILE_BYTES;
        // dQ += dS K, sixteens of keys that no row sees left out as in dK/dV
        if (j * 128 + 112 < kmax) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) tmem_step(tm_dq, tmem + (j & 1) * 128, k_addr, kk, j > 0 || kk > 0);
        } else {
#pragma unroll 1
          for (int kk = 0; j * 128 + kk * 16 < kmax; ++kk) tmem_step(tm_dq, tmem + (j & 1) * 128, k_addr, kk, j > 0 || kk > 0);
        }
        commit(&k_empty[j % 3]);
      }
      if (ok) commit(&done);
    }
  } else if (warp < BWD_WARPS) {
    const int wg = warp >> 2, quarter = warp & 3;
    const int grow = m0 + quarter * 32 + lane;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    const bool row_ok = grow < qlen;
    // a row outside the sequence gets lse = +inf, so that its P is exactly 0
    const float nl = row_ok ? -p.lse[(long long)h * p.Tq + q0 + grow] * LOG2E : -INFINITY;
    const float nd = row_ok ? -p.delta[(long long)h * p.Tq + q0 + grow] : 0.f;
    const f2 scale2 = pack2(p.scale_log2, p.scale_log2), nl2 = pack2(nl, nl), nd2 = pack2(nd, nd);
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      const uint32_t ts = tmem + (j & 1) * 128 + lanes + wg * NC;
      ok = mbar_wait_warp(&s_full[j & 1], (j >> 1) & 1, p.error, ERR_S);
      if (!ok) break;
      fence_after();
      float s[NC];
      tmem_ld_cols<NC>(ts, s);
      const bool masked = j * 128 + 128 > klen || (p.causal && j * 128 + 127 > m0 + off);
      const int limit = masked ? min(klen, p.causal ? grow + off + 1 : klen) - j * 128 - wg * NC : NC;   // valid columns
#pragma unroll
      for (int c = 0; c < NC; c += 2) {
        float2 a = unpack2(fma2(pack2(s[c], s[c + 1]), scale2, nl2));
        a = make_float2(ex2(a.x), ex2(a.y));
        if (masked) {
          a.x = c < limit ? a.x : 0.f;
          a.y = c + 1 < limit ? a.y : 0.f;
        }
        s[c] = a.x, s[c + 1] = a.y;
      }
      ok = mbar_wait_warp(&dp_full, j & 1, p.error, ERR_S);
      if (!ok) break;
      fence_after();
      float dp[NC];
      tmem_ld_cols<NC>(tm_dp + lanes + wg * NC, dp);
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&dp_free);
#pragma unroll
      for (int c = 0; c < NC; c += 32) {
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int e = c + 2 * i;
          packed[i] = pack_bf16(unpack2(mul2(pack2(s[e], s[e + 1]), add2(pack2(dp[e], dp[e + 1]), nd2))));
        }
        tmem_st_cols(ts + c / 2, packed);
      }
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ds_ready);
    }
    if (ok && n_tiles > 0) ok = mbar_wait_warp(&done, 0, p.error, ERR_PV);
    if (ok) {
      if (n_tiles > 0) fence_after();
      const int qc = head_col(0, p.q_group_stride, p.q_hpg, p.q_head_stride, h);
      store_half_tile(tm_dq + lanes + wg * 64, p.scale, n_tiles == 0, smem + warp * (32 * OUT_PITCH), lane,
                      p.dq + (long long)(q0 + m0 + quarter * 32) * p.q_stride_t + qc + wg * 64, p.q_stride_t,
                      qlen - (m0 + quarter * 32));
    }
  }
  fence_before();
  __syncthreads();
  if (warp == BWD_MMA) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
  }
}

}  // namespace fa5
}  // namespace msrl
