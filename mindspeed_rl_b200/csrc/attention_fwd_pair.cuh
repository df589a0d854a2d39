// Flash attention forward for heads of 128, two query tiles to a block (included by attention_tcgen05.cu).
//
// A block takes two 128-row query tiles of one KV head and walks the keys in tiles of 128; both query tiles use each K and V
// tile once it is in shared memory.  The query tiles of a KV head are numbered row tile by row tile and, inside one, query head
// by query head, so that a pair shares its key range (or differs by one tile) with grouped heads and without.  Per tile:
//   S = Q K^T        tcgen05.mma 128 x 128 x 16, both operands from shared memory, into TMEM;
//   soft-max         one warpgroup to a query tile, one thread to a row: the row in registers, running maximum and sum in the
//                    exp2 domain, P (bf16) back to TMEM over the first half of its own scores;
//   O += P V         tcgen05.mma with P read from TMEM and V as an MN-major operand; starts on the first 64 keys while the
//                    exponentials of the other 64 are computed.
// While one tile's soft-max runs, the tensor cores work on the other tile: PV and the next scores of a tile are issued together,
// in turn for the two tiles.  O moves to a new running maximum only when a row's maximum passed it by more than 2^8.
//
// What bounds it: 16384 exponentials and 1024 tensor-core cycles per tile of 128 x 128 (both units are full at about the same
// rate on an SM), and the soft-max of one tile plus its own two products in a row.  Before: 64-key tiles, whose 128 x 64 products
// are bound by shared-memory reads, with P through shared memory and each score read twice from TMEM.  Causal, 28 heads over 4:
// one sequence of 22528, 7361 and 2879 tokens each 6261 -> 3273 us (653 -> 1248 TFLOP/s), 1280 + 3072 + 1863 + 2201 tokens
// 334 -> 186 us, eight of 1024 184 -> 127 us.
#pragma once

namespace msrl {
namespace fa5 {

constexpr int PAIR_THREADS = 384;                     // warps 0-3, 4-7: soft-max of tile 0, 1; warp 8: TMA; warp 9: MMA
constexpr int PAIR_TMA = 8, PAIR_MMA = 9;
constexpr uint32_t PAIR_Q = 0, PAIR_K = 2 * TILE_BYTES, PAIR_V = PAIR_K + 2 * TILE_BYTES, PAIR_SMEM = PAIR_V + 2 * TILE_BYTES;

// max of three (one instruction)
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float ex2(float x) {
  float d;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(d) : "f"(x));
  return d;
}

// Query tile `item` of KV head hk: row tile item / rep, query head item % rep, the keys [k0, k1) that its rows see and the key tiles
// [t0, t1) they lie in.
struct QueryTile {
  int m0, h, k0, k1, t0, t1;
  __device__ __forceinline__ QueryTile(const Params& p, int item, int hk, int rep, int qlen, int klen) {
    m0 = item / rep * BM;
    h = hk * rep + item % rep;
    const int off = klen - qlen;
    k0 = p.window > 0 ? max(m0 + off - p.window + 1, 0) : 0;
    k1 = max(p.causal ? min(klen, m0 + BM + off) : klen, 0);
    t0 = k0 / 128;
    t1 = m0 < qlen ? max((k1 + 127) / 128, t0) : t0;
  }
};

template <bool CAP>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
fa_fwd_pair_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const __grid_constant__ Params p, const int batch, const int groups,
                   const int width) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ uint64_t q_full[2], k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_part[2][2], o_full[2];
  __shared__ uint32_t tmem_slot;

  // longest key ranges first: the last row tiles of every (sequence, KV head)
  const int hk = blockIdx.x % p.nkv, b = blockIdx.x / p.nkv % batch, grp = groups - 1 - blockIdx.x / p.nkv / batch;
  const int q0 = p.cu_q[b], qlen = p.cu_q[b + 1] - q0;
  const int k0 = p.cu_k[b], klen = p.cu_k[b + 1] - k0;
  const int rep = p.nh / p.nkv;
  const int items = (qlen + BM - 1) / BM * rep;
  if (grp * width >= items) return;                    // uniform for the block, before any allocation
  const QueryTile tile0(p, grp * width, hk, rep, qlen, klen);
  const bool second = width == 2 && grp * 2 + 1 < items;
  const QueryTile tile1(p, second ? grp * 2 + 1 : items, hk, rep, qlen, klen);
  const bool empty0 = tile0.t0 == tile0.t1, empty1 = !second || tile1.t0 == tile1.t1;
  int j0 = 0, j1 = 0;
  if (!empty0) j0 = tile0.t0, j1 = tile0.t1;
  if (!empty1) j0 = empty0 ? tile1.t0 : min(j0, tile1.t0), j1 = max(j1, tile1.t1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_part[i][0], 4);
      mbar_init(&p_part[i][1], 4);
      mbar_init(&o_full[i], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == PAIR_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;                     // scores (and P) of the two tiles: 0, 128; O: 256, 384

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;\n");   // 56 + 2 x 224 = 3 x 168, what the block was launched with
    if (warp == PAIR_TMA && elect_one()) {
      const int kc = head_col(p.k_col0, p.k_group_stride, p.k_hpg, p.k_head_stride, hk);
      const int vc = head_col(p.v_col0, p.v_group_stride, p.v_hpg, p.v_head_stride, hk);
      auto load_q = [&](int x, const QueryTile& t) {
        const int qc = head_col(p.q_col0, p.q_group_stride, p.q_hpg, p.q_head_stride, t.h);
        mbar_expect_tx(&q_full[x], TILE_BYTES);
        for (int i = 0; i < 2; ++i)
          tma_load_2d(smem + PAIR_Q + x * TILE_BYTES + i * TILE_HALF, &map_q, &q_full[x], qc + i * 64, q0 + t.m0);
      };
      if (!empty0) load_q(0, tile0);
      for (int j = j0; j < j1; ++j) {
        const int st = (j - j0) & 1;
        const uint32_t use = (j - j0) >> 1;
        if (use > 0 && !mbar_wait(&k_empty[st], (use - 1) & 1, p.error, ERR_EMPTY)) break;
        mbar_expect_tx(&k_full[st], TILE_BYTES);
        for (int i = 0; i < 2; ++i)
          tma_load_2d(smem + PAIR_K + st * TILE_BYTES + i * TILE_HALF, &map_k, &k_full[st], kc + i * 64, k0 + j * 128);
        if (j == j0 && !empty1) load_q(1, tile1);
        if (use > 0 && !mbar_wait(&v_empty[st], (use - 1) & 1, p.error, ERR_EMPTY)) break;
        mbar_expect_tx(&v_full[st], TILE_BYTES);
        for (int i = 0; i < 2; ++i)
          tma_load_2d(smem + PAIR_V + st * TILE_BYTES + i * TILE_HALF, &map_v, &v_full[st], vc + i * 64, k0 + j * 128);
      }
    } else if (warp == PAIR_MMA && elect_one()) {
      constexpr uint32_t id_s = idesc_bf16(BM, 128, false), id_o = idesc_bf16(BM, D, true);
      const uint32_t base = smem_u32(smem);
      uint32_t turn[2] = {0, 0};                       // tiles whose P was taken, per query tile
      bool ok = true;
      auto pv = [&](int x, int j, const QueryTile& t) {  // O_x += P_x V_j
        const int st = (j - j0) & 1;
        const uint32_t v_addr = base + PAIR_V + st * TILE_BYTES;
        // Sixteens of keys that no row sees are left out: their P is 0, but 0 times an inf or nan of V would reach the rows.  Tested
        // once a tile, in front of steps without a branch (a branch a step cost prompts 0.7 to 0.9 %).
        const int from = t.k0 - j * 128 - 15, to = t.k1 - j * 128;
        const bool whole = from <= 0 && to > 112;
        ok = mbar_wait(&v_full[st], ((j - j0) >> 1) & 1, p.error, ERR_V);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          ok = ok && mbar_wait(&p_part[x][half], turn[x] & 1, p.error, ERR_P);
          if (!ok) return;
          fence_after();
          auto step = [&](int kk, bool add) {
            umma_ts(tmem + 256 + x * 128, tmem + x * 128 + kk * 8, desc_sw128(v_addr + kk * 2048, TILE_HALF, 1024), id_o,
                    add ? 1u : 0u);
          };
          if (whole) {
#pragma unroll
            for (int kk = half * 4; kk < half * 4 + 4; ++kk) step(kk, j > t.t0 || kk > 0);
          } else {
#pragma unroll 1
            for (int kk = half * 4; kk < half * 4 + 4; ++kk)
              if (kk * 16 >= from && kk * 16 < to) step(kk, j > t.t0 || kk * 16 >= from + 16);
          }
        }
        ++turn[x];
      };
      auto scores = [&](int x, int j, const QueryTile& t) {  // S_x = Q_x K_j^T
        const int st = (j - j0) & 1;
        const uint32_t q_addr = base + PAIR_Q + x * TILE_BYTES, k_addr = base + PAIR_K + st * TILE_BYTES;
        ok = mbar_wait(&k_full[st], ((j - j0) >> 1) & 1, p.error, ERR_K);
        if (ok && j == t.t0) ok = mbar_wait(&q_full[x], 0, p.error, ERR_Q);
        if (!ok) return;
        fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma(tmem + x * 128, desc_sw128(q_addr + (kk >> 2) * TILE_HALF + (kk & 3) * 32, 16, 1024),
               desc_sw128(k_addr + (kk >> 2) * TILE_HALF + (kk & 3) * 32, 16, 1024), id_s, kk > 0 ? 1u : 0u);
        commit(&s_full[x]);
      };
      auto in = [](int j, const QueryTile& t) { return j >= t.t0 && j < t.t1; };
      // step j: the products with V of key tile j - 1 and the scores of key tile j; a commit covers everything issued before
      // it, so full scores also say that the earlier P of this query tile has been read
      for (int j = j0; j <= j1 && j1 > j0; ++j) {
        if (!empty0) {
          if (in(j - 1, tile0)) pv(0, j - 1, tile0);
          if (ok && j == tile0.t1) commit(&o_full[0]);
          if (ok && in(j, tile0)) scores(0, j, tile0);
        }
        if (ok && !empty1 && in(j - 1, tile1)) pv(1, j - 1, tile1);
        if (!ok) break;
        if (j > j0) commit(&v_empty[(j - 1 - j0) & 1]);
        if (!empty1) {
          if (j == tile1.t1) commit(&o_full[1]);
          if (in(j, tile1)) scores(1, j, tile1);
        }
        if (!ok) break;
        if (j < j1) commit(&k_empty[(j - j0) & 1]);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;\n");
    const int x = warp >> 2, quarter = warp & 3;
    if (x == 0 || second) {
      const QueryTile& t = x == 0 ? tile0 : tile1;
      const int row = quarter * 32 + lane, grow = t.m0 + row;   // row of the tile, of the sequence
      const int off = klen - qlen;
      const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
      const uint32_t tm_s = tmem + lanes + x * 128, tm_o = tmem + lanes + 256 + x * 128;
      const f2 scale2 = pack2(p.scale_log2, p.scale_log2);
      const SoftCap2 cap(CAP ? p.softcap : 1.f);
      float m_run = -INFINITY, l_run = 0.f;
      bool ok = true;
      for (int j = t.t0; j < t.t1; ++j) {
        ok = mbar_wait_warp(&s_full[x], (j - t.t0) & 1, p.error, ERR_S);
        if (!ok) break;
        fence_after();
        float s[128];
        tmem_ld_cols<128>(tm_s, s);
        const int kbase = j * 128;
        if ((kbase + 128 > klen) || (p.causal && kbase + 127 > t.m0 + off) ||
            (p.window > 0 && kbase <= t.m0 + BM - 1 + off - p.window)) {
          const int limit = min(klen, p.causal ? grow + off + 1 : klen) - kbase;   // this row sees [from, limit)
          const int from = p.window > 0 ? grow + off + 1 - p.window - kbase : 0;
#pragma unroll
          for (int i = 0; i < 128; ++i) s[i] = (i < limit && i >= from) ? s[i] : -INFINITY;
        }
        float m4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) m4[i] = fmaxf(s[i], s[i + 4]);
#pragma unroll
        for (int i = 8; i < 128; i += 8)
#pragma unroll
          for (int c = 0; c < 4; ++c) m4[c] = max3(m4[c], s[i + c], s[i + c + 4]);
        float mx = fmaxf(max3(m4[0], m4[1], m4[2]), m4[3]) * p.scale_log2;         // scale > 0
        if (CAP && mx != -INFINITY) mx = cap(mx);
        float m_new = fmaxf(m_run, mx);
        if (m_run != -INFINITY && m_new - m_run <= 8.f) m_new = m_run;
        const float m_use = m_new == -INFINITY ? 0.f : m_new;
        const float corr = exp2f(m_run - m_use);
        // full scores say that the product with the previous V is finished, so O stands still here
        if (j > t.t0 && __any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            float o[32];
            tmem_ld32(tm_o + c * 32, o);
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] *= corr;
            tmem_st32(tm_o + c * 32, o);
          }
        }
        const f2 neg = pack2(-m_use, -m_use);
        f2 sum[4] = {0, 0, 0, 0};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t packed[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int e = c * 32 + 2 * i;
            float2 v;
            if constexpr (CAP) {
              v = make_float2(s[e] == -INFINITY ? -INFINITY : cap(s[e] * p.scale_log2) - m_use,
                              s[e + 1] == -INFINITY ? -INFINITY : cap(s[e + 1] * p.scale_log2) - m_use);
            } else {
              v = unpack2(fma2(pack2(s[e], s[e + 1]), scale2, neg));
            }
            v.x = ex2(v.x);
            v.y = ex2(v.y);
            sum[i & 3] = add2(sum[i & 3], pack2(v.x, v.y));
            const __nv_bfloat162 h2 = __floats2bfloat162_rn(v.x, v.y);
            packed[i] = *reinterpret_cast<const uint32_t*>(&h2);
          }
          tmem_st_cols(tm_s + c * 16, packed);
          if (c & 1) {
            tmem_wait_st();
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_part[x][c >> 1]);
          }
        }
        const float2 a = unpack2(add2(add2(sum[0], sum[1]), add2(sum[2], sum[3])));
        l_run = l_run * corr + (a.x + a.y);
        m_run = m_new;
      }
      const bool none = t.t0 == t.t1;
      if (ok && !none) ok = mbar_wait_warp(&o_full[x], 0, p.error, ERR_PV);
      if (ok) {
        fence_after();
        const float factor = grow < qlen ? p.tail.scale2(q0 + grow, t.h, m_run, l_run) : 0.f;
        // 32 rows of 256 bytes through this warp's quarter of the query tile, which every product has read by now; chunks of
        // 16 bytes are XORed with the row
        unsigned char* patch = smem + PAIR_Q + x * TILE_BYTES + quarter * 8192;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float v[32];
          if (!none) {
            tmem_ld32(tm_o + c * 32, v);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] *= factor;
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0.f;
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
            *reinterpret_cast<bf16x8*>(patch + lane * 256 + (((c * 4 + q) ^ (lane & 7)) << 4)) = pack8(v + q * 8);
        }
        __syncwarp();
        __nv_bfloat16* dst = p.o + (long long)(q0 + t.m0 + quarter * 32) * p.o_stride_t + (long long)t.h * D;
        const int rows = qlen - (t.m0 + quarter * 32), chunk = lane & 15;
#pragma unroll
        for (int it = 0; it < 16; ++it) {
          const int r = it * 2 + (lane >> 4);
          if (r < rows)
            st8(dst + (long long)r * p.o_stride_t + chunk * 8,
                *reinterpret_cast<const bf16x8*>(patch + r * 256 + ((chunk ^ (r & 7)) << 4)));
        }
        if (grow < qlen) p.lse[(long long)t.h * p.Tq + q0 + grow] = (m_run + log2f(l_run)) * 0.6931471805599453f;
      }
    }
  }
  fence_before();
  __syncthreads();
  if (warp == PAIR_MMA) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
  }
}

}  // namespace fa5
}  // namespace msrl
