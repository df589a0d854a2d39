// The log-softmax record of one row over (a part of) the vocabulary: written by the statistics kernel of logprob.cu and by the
// epilogues of the two LM-head GEMMs, combined by logprob_finish_kernel.
#pragma once
#include <cstddef>

#include "common.cuh"

namespace msrl {

struct RowStat {
  float m;    // max of z
  float s;    // sum exp(z - m)
  float zy;   // z[label] if the label lies in this part, else 0
  float spz;  // sum exp(z - m) * z
};
static_assert(sizeof(RowStat) == 16 && offsetof(RowStat, m) == 0 && offsetof(RowStat, s) == 4 && offsetof(RowStat, zy) == 8 &&
              offsetof(RowStat, spz) == 12);   // logprob_finish_kernel takes a record as a float4, other readers as four columns

// Record of a row over COLS accumulator columns: `load(c, v)` fetches columns [32 c, 32 c + 32) of this thread's row.  Columns from
// `N` on do not count; `col0` is the column of the first, `label` relative to column 0 of the matrix.
template <int COLS, typename Load>
__device__ __forceinline__ RowStat tile_row_stat(Load load, int col0, int N, long long label, float inv_temp) {
  RowStat r{-INFINITY, 0.f, 0.f, 0.f};
#pragma unroll 1
  for (int c = 0; c < COLS / 32; ++c) {
    float v[32];
    load(c, v);
    const int col = col0 + c * 32;
    float cm = -INFINITY;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      // logits take the bf16 rounding the un-fused path would apply before the soft-max
      v[j] = (col + j < N) ? __bfloat162float(__float2bfloat16(v[j])) * inv_temp : -INFINITY;
      cm = fmaxf(cm, v[j]);
    }
    if (cm > r.m) {
      const float corr = __expf(r.m - cm);
      r.s *= corr;
      r.spz *= corr;
      r.m = cm;
    }
    if (r.m > -INFINITY) {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        if (col + j < N) {
          const float e = __expf(v[j] - r.m);
          r.s += e;
          r.spz += e * v[j];
        }
      }
    }
    if (label >= col && label < col + 32 && label < N) {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (label == col + j) r.zy = v[j];
    }
  }
  return r;
}

}  // namespace msrl
