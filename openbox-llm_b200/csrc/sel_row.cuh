// Selection attention of single rows in scalar fp32, for the rows and key tiles that the three-term tcgen05 kernels
// cannot finish: a product of a masked probability (zero) with a value that is infinite or NaN is NaN, so where such a
// value sits in a tile every row of the tile would carry it.  What comes out non-finite there is computed
// again here from the row's own list, key by key, and stays with what attends the value.
//
// The other roles of a CTA wait meanwhile, each wait for about a second at most.  What a wait covers is one row's list in
// the forward, 13 us a key at D = 128 on a full SM, which is why longer lists than 32768 keys stay on the CUDA cores, and
// one row tile against one key tile in the backward, a tenth of a millisecond.  A value that every query attends, at
// 8192 tokens of 4 heads of 128 and 8 blocks of 16 a list: forward 2.0 ms, backward 27 (CUDA cores 0.28 and 0.92; 9
// and 151 by elements of 2 bytes and with the sums of a key tile in shared memory).
#pragma once

#include "common.cuh"

namespace nsa {
namespace tc {

// How often a list of S blocks names block `blk`.
__device__ __forceinline__ int times_listed(const int32_t* row, int S, int blk) {
  int n = 0;
#pragma unroll 1
  for (int s = 0; s < S; ++s) n += ld_plain(row + s) == blk;
  return n;
}

// eight bf16 of an aligned row as floats
__device__ __forceinline__ void load8_row(const __nv_bfloat16* p, float* f) {
  const uint4 u = ld_plain(reinterpret_cast<const uint4*>(p));
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    f[2 * e] = __uint_as_float(w[e] << 16);
    f[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
  }
}

template <int D>
__device__ __forceinline__ float dot_rows(const __nv_bfloat16* a, const __nv_bfloat16* b) {
  float acc[2] = {0.f, 0.f};
#pragma unroll 2
  for (int d = 0; d < D; d += 8) {
    float x[8], y[8];
    load8_row(a + d, x);
    load8_row(b + d, y);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e & 1] = fmaf(x[e], y[e], acc[e & 1]);
  }
  return acc[0] + acc[1];
}

// acc += w * (32 columns of a row)
__device__ __forceinline__ void add32_row(float w, const __nv_bfloat16* row, float* acc) {
#pragma unroll
  for (int c = 0; c < 32; c += 8) {
    float x[8];
    load8_row(row + c, x);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[c + e] = fmaf(w, x[e], acc[c + e]);
  }
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
      const int blk = ld_plain(list + s);
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
        add32_row(p, v + (size_t)key * D + (pass - 1) * 32, acc);
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
