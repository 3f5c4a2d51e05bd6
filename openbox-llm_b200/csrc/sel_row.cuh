// Selection attention of single rows in scalar fp32, for the rows and key tiles that the three-term tcgen05 kernels
// cannot finish: a product of a masked probability (zero) with a value that is infinite or NaN is NaN, so where such a
// value sits in a tile every row of the tile would carry it.  What comes out non-finite there is computed
// again here from the row's own list, key by key, and stays with what attends the value.  Speed does not matter.
#pragma once

#include "common.cuh"

namespace nsa {
namespace tc {

// How often a list of S blocks names block `blk`.
__device__ __forceinline__ int times_listed(const int32_t* __restrict__ row, int S, int blk) {
  int n = 0;
#pragma unroll 1
  for (int s = 0; s < S; ++s) n += __ldg(row + s) == blk;
  return n;
}

template <int D>
__device__ __forceinline__ float dot_rows(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b) {
  float acc = 0.f;
#pragma unroll 1
  for (int d = 0; d < D; d += 2) {
    const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(a + d));
    const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(b + d));
    acc = fmaf(x.x, y.x, acc);
    acc = fmaf(x.y, y.y, acc);
  }
  return acc;
}

// Output and LSE of one row, 32 columns at a time; k and v are those of its unit.
template <int D>
__device__ __noinline__ void sel_row_forward(const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v,
                                             const int32_t* list, int S, int block_size, int t, float scale_log2,
                                             __nv_bfloat16* o, float* lse) {
  float m = -INFINITY;
#pragma unroll 1
  for (int pass = 0; pass <= D / 32; ++pass) {           // pass 0: the maximum
    float acc[32], l = 0.f;
#pragma unroll
    for (int e = 0; e < 32; ++e) acc[e] = 0.f;
#pragma unroll 1
    for (int s = 0; s < S; ++s) {
      const int blk = __ldg(list + s);
      if (blk < 0 || (long long)blk * block_size > t) continue;
      const int last = min(t, (blk + 1) * block_size - 1);
#pragma unroll 1
      for (int key = blk * block_size; key <= last; ++key) {
        const float x = dot_rows<D>(q, k + (size_t)key * D) * scale_log2;
        if (pass == 0) {
          m = fmaxf(m, x);
          continue;
        }
        const float p = exp2f(x - m);
        l += p;
        const __nv_bfloat16* vr = v + (size_t)key * D + (pass - 1) * 32;
#pragma unroll
        for (int e = 0; e < 32; ++e) acc[e] = fmaf(p, to_float(vr[e]), acc[e]);
      }
    }
    if (pass == 0) continue;
    const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
    for (int e = 0; e < 32; ++e) o[(pass - 1) * 32 + e] = __float2bfloat16_rn(acc[e] * inv);
    *lse = l > 0.f ? (m + log2f(l)) * kLn2 : kLseEmpty;
  }
}

}  // namespace tc
}  // namespace nsa
