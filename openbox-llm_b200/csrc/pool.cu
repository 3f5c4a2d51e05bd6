// Pooling of the compression branch: learned pooling (nsa_model.py:118-123) and mean pooling
// (nsa_fused_kernel.py:549-554), forward and backward, for bf16 rows of 16, 32, 64 or 128 columns
// (and mean pooling of fp32).  Every kernel takes the K and the V tensor of the branch in one
// launch (blockIdx.y).  All of them are bound by the one pass over x (and dx); at 2 x 16 units of
// 32768 x 128 the learned forward takes 0.11 ms (0.18 ms as two launches with their loads one
// window row at a time) and its backward 0.18 ms (0.25 ms with the projection's gradient in scalar atomics; 0.63 ms when it read x
// twice more and had that gradient in a kernel of its own); at 4 units of 512 x 64 the forward takes 5 us
// (2 x 14 us).  In short calls the backward's end counts: D x D atomics of every CTA, and the last CTA's copy of their sums;
// as vectors of four, and with the copy's loads all in flight, 2 x 1024 tokens of 4 heads of 128 in windows of 16 take 30 us, 63 before.
#include "pool.cuh"

namespace nsa {
namespace {

constexpr int kThreads = 256;
constexpr int kLoads = 4;        // 16-byte loads of one summary row a thread has in flight

__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {                         // bf16 -> fp32 is a shift
    f[2 * e] = __uint_as_float(w[e] << 16);
    f[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ void cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_commit_wait() { asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory"); }

// softmax over the window positions into w[len]; e[len] is scratch.  One exponential per position
// and thread; the sum runs in position order in every thread, so w is the same whatever the
// number of threads.  Ends with a barrier.
__device__ __forceinline__ void pool_weights(const float* __restrict__ logits, float* w, float* e, int len) {
  for (int r = threadIdx.x; r < len; r += blockDim.x) e[r] = __ldg(logits + r);
  __syncthreads();
  float mx = -INFINITY;
  for (int r = 0; r < len; ++r) mx = fmaxf(mx, e[r]);
  __syncthreads();
  for (int r = threadIdx.x; r < len; r += blockDim.x) e[r] = expf(e[r] - mx);
  __syncthreads();
  float den = 0.f;
  for (int r = 0; r < len; ++r) den += e[r];
  for (int r = threadIdx.x; r < len; r += blockDim.x) w[r] = e[r] / den;
  __syncthreads();
}

// Forward.  A CTA takes R consecutive summary rows: D/8 threads per token row with 16-byte loads,
// 256/(D/8) token rows at a time, all loads of two summary rows in flight together; the
// projection matrix travels into shared memory (cp.async, padded rows) meanwhile.  R = 8, or 4, where
// that still gives every SM a CTA, else 2: a short sequence has a few dozen rows in all, and the
// latency of one CTA's chain is what counts.  512 rows of 128 in windows of 16: R = 8 14.5 us, 4 14.5, 2 18.8 (more CTAs than fit at once);
// 552 rows of 64 in windows of 64: 14.6, 13.4, 16.7.  Over the range of R = 4 (K and V, R = 2 | 4), windows of 64: 296 rows of 64 10.5 | 10.3, 400
// 12.5 | 11.5, 584 16.6 | 12.5; 296 rows of 128 13.0 | 12.5, 400 18.6 | 14.8, 584 20.7 | 16.7; windows of 16: 8.7 | 8.6 to 16.7 | 12.7.
template <int D, int R>
struct PoolFwdSmem {
  static constexpr int kProjLd = D + 4;                 // float4 reads of 8 lanes cover all banks
  static constexpr int kFloats = D /*cvec*/ + R * D /*pooled*/ + R * 8 * D /*partials*/ + D * kProjLd;
};

template <int D, int R>
__global__ void __launch_bounds__(kThreads, 2)
pool_fwd_kernel(const PoolSides s, int T_, int len, int stride, int n_sum, int rows) {
  extern __shared__ float4 sm4[];
  chain_go();
  float* sm = reinterpret_cast<float*>(sm4);
  constexpr int VL = D / 8, RG = kThreads / VL, kLd = PoolFwdSmem<D, R>::kProjLd;
  float* projS = sm;
  float* cvec = projS + D * kLd;
  float* pooled = cvec + D;
  float* part = pooled + R * D;
  float* w = part + R * 8 * D;
  float* e = w + len;
  const int side = blockIdx.y;
  const __nv_bfloat16* __restrict__ x = (const __nv_bfloat16*)s.x[side];
  const float* __restrict__ intra = s.intra[side];
  __nv_bfloat16* out = (__nv_bfloat16*)s.out[side];
  float* pooled_out = s.pooled[side];
  const int tid = threadIdx.x, warp = tid >> 5;
  const int vl = tid % VL, rg = tid / VL;
  const int row0 = blockIdx.x * R;
  if (out)
    for (int i = tid; i < D * D / 4; i += kThreads)
      cp16(projS + (i / (D / 4)) * kLd + (i % (D / 4)) * 4, s.proj[side] + (size_t)i * 4);
  asm volatile("cp.async.commit_group;" ::: "memory");
  pool_weights(s.logits[side], w, e, len);
  // the row-independent part: sum_r w[r] * intra[r][:]
  {
    float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int r = rg; r < len; r += RG) {
      const float4 lo = __ldg(reinterpret_cast<const float4*>(intra + (size_t)r * D + vl * 8));
      const float4 hi = __ldg(reinterpret_cast<const float4*>(intra + (size_t)r * D + vl * 8 + 4));
      const float wr = w[r];
      a[0] = fmaf(wr, lo.x, a[0]); a[1] = fmaf(wr, lo.y, a[1]); a[2] = fmaf(wr, lo.z, a[2]); a[3] = fmaf(wr, lo.w, a[3]);
      a[4] = fmaf(wr, hi.x, a[4]); a[5] = fmaf(wr, hi.y, a[5]); a[6] = fmaf(wr, hi.z, a[6]); a[7] = fmaf(wr, hi.w, a[7]);
    }
    // threads of a warp that hold the same columns (VL apart) meet by shuffles
#pragma unroll
    for (int o = 16; o >= VL; o >>= 1)
#pragma unroll
      for (int k = 0; k < 8; ++k) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
    if ((tid & 31) < VL)
#pragma unroll
      for (int k = 0; k < 8; ++k) part[warp * D + vl * 8 + k] = a[k];
  }
  __syncthreads();
  if (tid < D) {
    float c = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) c += part[k * D + tid];
    cvec[tid] = c;
  }
  __syncthreads();
#pragma unroll
  for (int b0 = 0; b0 < R; b0 += 2) {
    float a[2][8];
    const __nv_bfloat16* xb[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int row = min(row0 + b0 + k, rows - 1);      // rows past the end repeat the last one and are dropped
      xb[k] = x + ((size_t)(row / n_sum) * T_ + (size_t)(row % n_sum) * stride) * D + vl * 8;
#pragma unroll
      for (int q = 0; q < 8; ++q) a[k][q] = 0.f;
    }
    for (int r0 = rg; r0 < len; r0 += RG * kLoads) {
      uint4 u[2][kLoads];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < kLoads; ++j) {
          const int r = r0 + j * RG;
          u[k][j] = r < len ? __ldg(reinterpret_cast<const uint4*>(xb[k] + (size_t)r * D)) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < kLoads; ++j) {
          const int r = r0 + j * RG;
          const float wr = r < len ? w[r] : 0.f;
          float f[8];
          unpack8(u[k][j], f);
#pragma unroll
          for (int q = 0; q < 8; ++q) a[k][q] = fmaf(wr, f[q], a[k][q]);
        }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
#pragma unroll
      for (int o = 16; o >= VL; o >>= 1)
#pragma unroll
        for (int q = 0; q < 8; ++q) a[k][q] += __shfl_xor_sync(0xffffffffu, a[k][q], o);
      if ((tid & 31) < VL) {
        float4* dst = reinterpret_cast<float4*>(part + ((b0 + k) * 8 + warp) * D + vl * 8);
        dst[0] = make_float4(a[k][0], a[k][1], a[k][2], a[k][3]);
        dst[1] = make_float4(a[k][4], a[k][5], a[k][6], a[k][7]);
      }
    }
  }
  __syncthreads();
  for (int idx = tid; idx < R * D; idx += kThreads) {
    const int b = idx / D, d = idx % D;
    float v = cvec[d];
#pragma unroll
    for (int k = 0; k < 8; ++k) v += part[(b * 8 + k) * D + d];
    pooled[idx] = v;
    if (pooled_out && row0 + b < rows) pooled_out[(size_t)(row0 + b) * D + d] = v;
  }
  if (!out) return;
  cp_commit_wait();
  __syncthreads();
  // out[row][o] = sum_i proj[o][i] * pooled[row][i], in the order of i; up to four rows per thread
  constexpr int RP = R < 4 ? R : 4;
  for (int idx = tid; idx < (R / RP) * D; idx += kThreads) {
    const int b0 = (idx / D) * RP, o = idx % D;
    float acc[RP];
#pragma unroll
    for (int k = 0; k < RP; ++k) acc[k] = 0.f;
#pragma unroll 4
    for (int i = 0; i < D; i += 4) {
      const float4 pv = *reinterpret_cast<const float4*>(projS + o * kLd + i);
#pragma unroll
      for (int k = 0; k < RP; ++k) {
        const float4 pl = *reinterpret_cast<const float4*>(pooled + (b0 + k) * D + i);
        acc[k] = fmaf(pv.x, pl.x, acc[k]); acc[k] = fmaf(pv.y, pl.y, acc[k]);
        acc[k] = fmaf(pv.z, pl.z, acc[k]); acc[k] = fmaf(pv.w, pl.w, acc[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < RP; ++k)
      if (row0 + b0 + k < rows) out[(size_t)(row0 + b0 + k) * D + o] = __float2bfloat16(acc[k]);
  }
}

// Backward of the same, persistent: a CTA walks groups of R summary rows.
//   d_pooled = d_out @ W                       (W stays in shared memory)
//   dx       = w[pos] * d_pooled               (windows that do not overlap; else pool_dx_kernel)
//   d_w[pos] += sum_d d_pooled[d] * x[pos][d],  sum_dp += d_pooled,  d_proj += d_out^T pooled
// The sums stay in registers over all groups of the CTA and meet by atomics once at its end; the
// last CTA to arrive turns them into d_intra, d_logits and d_proj.  One pass over x and one over
// dx is all the traffic there is.
template <int D> struct PoolBwdSmem {
  static constexpr int R = 8;
  static constexpr int kFloats = D * D + 3 * R * D;
};

template <int D>
__global__ void __launch_bounds__(kThreads, 2)
pool_bwd_kernel(const PoolSides s, int T_, int len, int stride, int n_sum, int rows) {
  extern __shared__ float4 sm4[];
  float* sm = reinterpret_cast<float*>(sm4);
  constexpr int VL = D / 8, RG = kThreads / VL, R = PoolBwdSmem<D>::R;
  constexpr int kTile = D >= 64 ? D / 16 : D / 8;       // d_proj: each thread owns kTile x kTile entries
  constexpr int kSide = D / kTile;                      // of a kSide x kSide grid of threads
  constexpr int kVec = kTile >= 4 ? 4 : 2;              // entries an atomic
  float* pj = sm;                 // [D][D]
  float* go = pj + D * D;         // [R][D] d_out
  float* dp = go + R * D;         // [R][D] d_pooled
  float* pl = dp + R * D;         // [R][D] pooled
  float* w = pl + R * D;          // [len]
  float* dw = w + len;            // [len]
  __shared__ int s_last;
  const int side = blockIdx.y;
  const __nv_bfloat16* __restrict__ x = (const __nv_bfloat16*)s.x[side];
  const __nv_bfloat16* __restrict__ d_out = (const __nv_bfloat16*)s.d_out[side];
  const float* __restrict__ pooled = s.pooled[side];
  __nv_bfloat16* __restrict__ dx = (__nv_bfloat16*)s.dx[side];
  const bool write_dx = stride == len;
  float* acc_dp = s.acc[side];            // [D]
  float* acc_proj = acc_dp + D;           // [D][D]
  float* acc_w = acc_proj + D * D;        // [len]
  unsigned* arrived = reinterpret_cast<unsigned*>(acc_w + len);
  const int tid = threadIdx.x;
  const int vl = tid % VL, rg = tid / VL;
  for (int i = tid; i < D * D / 4; i += kThreads) cp16(pj + i * 4, s.proj[side] + (size_t)i * 4);
  asm volatile("cp.async.commit_group;" ::: "memory");
  pool_weights(s.logits[side], w, dw, len);
  for (int r = tid; r < len; r += kThreads) dw[r] = 0.f;

  const int ti = tid % kSide, to = tid / kSide;
  const bool owns = to < kSide;
  float pacc[kTile][kTile];
#pragma unroll
  for (int a = 0; a < kTile; ++a)
#pragma unroll
    for (int b = 0; b < kTile; ++b) pacc[a][b] = 0.f;
  float dwacc[kLoads];
#pragma unroll
  for (int j = 0; j < kLoads; ++j) dwacc[j] = 0.f;
  float sdp = 0.f;
  const int tail = write_dx ? T_ - n_sum * len : 0;     // tokens past the last complete window: zero gradient
  cp_commit_wait();

  for (int row0 = blockIdx.x * R; row0 < rows; row0 += gridDim.x * R) {
    __syncthreads();
    for (int idx = tid; idx < R * D / 8; idx += kThreads) {
      const int b = idx / (D / 8), c = (idx % (D / 8)) * 8;
      float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      float4 p0 = make_float4(0.f, 0.f, 0.f, 0.f), p1 = p0;
      if (row0 + b < rows) {
        const size_t off = (size_t)(row0 + b) * D + c;
        unpack8(__ldg(reinterpret_cast<const uint4*>(d_out + off)), f);
        p0 = __ldg(reinterpret_cast<const float4*>(pooled + off));
        p1 = __ldg(reinterpret_cast<const float4*>(pooled + off + 4));
      }
      *reinterpret_cast<float4*>(go + b * D + c) = make_float4(f[0], f[1], f[2], f[3]);
      *reinterpret_cast<float4*>(go + b * D + c + 4) = make_float4(f[4], f[5], f[6], f[7]);
      *reinterpret_cast<float4*>(pl + b * D + c) = p0;
      *reinterpret_cast<float4*>(pl + b * D + c + 4) = p1;
    }
    __syncthreads();
    for (int idx = tid; idx < (R / 4) * D; idx += kThreads) {
      const int b0 = (idx / D) * 4, d = idx % D;
      float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
      for (int o = 0; o < D; o += 4) {
        float pv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) pv[q] = pj[(o + q) * D + d];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float4 g = *reinterpret_cast<const float4*>(go + (b0 + k) * D + o);
          a[k] = fmaf(g.x, pv[0], a[k]); a[k] = fmaf(g.y, pv[1], a[k]);
          a[k] = fmaf(g.z, pv[2], a[k]); a[k] = fmaf(g.w, pv[3], a[k]);
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        dp[(b0 + k) * D + d] = a[k];
        if (!write_dx && row0 + b0 + k < rows) s.d_pooled[side][(size_t)(row0 + b0 + k) * D + d] = a[k];
      }
    }
    __syncthreads();
    if (tid < D) {
#pragma unroll
      for (int b = 0; b < R; ++b) sdp += dp[b * D + tid];        // rows past the end hold zeros
    }
    if (owns) {
#pragma unroll 2
      for (int b = 0; b < R; ++b) {
        float gv[kTile], pv[kTile];
#pragma unroll
        for (int a = 0; a < kTile; ++a) { gv[a] = go[b * D + to * kTile + a]; pv[a] = pl[b * D + ti * kTile + a]; }
#pragma unroll
        for (int a = 0; a < kTile; ++a)
#pragma unroll
          for (int c = 0; c < kTile; ++c) pacc[a][c] = fmaf(gv[a], pv[c], pacc[a][c]);
      }
    }
#pragma unroll 1
    for (int b = 0; b < R; b += 2) {
      if (row0 + b >= rows) break;
      size_t base[2];
      bool live[2];
      float g[2][8];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int row = row0 + b + k;
        live[k] = row < rows;
        const int rc = live[k] ? row : rows - 1;
        base[k] = ((size_t)(rc / n_sum) * T_ + (size_t)(rc % n_sum) * stride) * D + vl * 8;
#pragma unroll
        for (int q = 0; q < 8; ++q) g[k][q] = dp[(b + k) * D + vl * 8 + q];   // zero for rows past the end
      }
      for (int r0 = rg, chunk = 0; r0 - rg < len; r0 += RG * kLoads, ++chunk) {
        uint4 u[2][kLoads];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int j = 0; j < kLoads; ++j) {
            const int r = r0 + j * RG;
            u[k][j] = r < len ? __ldg(reinterpret_cast<const uint4*>(x + base[k] + (size_t)r * D)) : make_uint4(0, 0, 0, 0);
          }
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int j = 0; j < kLoads; ++j) {
            const int r = r0 + j * RG;
            float f[8], dot = 0.f;
            unpack8(u[k][j], f);
#pragma unroll
            for (int q = 0; q < 8; ++q) dot = fmaf(g[k][q], f[q], dot);
            if (chunk == 0) dwacc[j] += dot;
            else if (r < len) atomicAdd(dw + r, dot);
            if (write_dx && live[k] && r < len) {
              const float wr = w[r];
              uint4 o;
              o.x = pack2(wr * g[k][0], wr * g[k][1]); o.y = pack2(wr * g[k][2], wr * g[k][3]);
              o.z = pack2(wr * g[k][4], wr * g[k][5]); o.w = pack2(wr * g[k][6], wr * g[k][7]);
              *reinterpret_cast<uint4*>(dx + base[k] + (size_t)r * D) = o;
            }
          }
      }
    }
    if (tail > 0) {       // the group that holds the last window of a (b, h) clears the tokens after it
      for (int b = 0; b < R && row0 + b < rows; ++b)
        if ((row0 + b) % n_sum == n_sum - 1) {
          uint4* dst = reinterpret_cast<uint4*>(dx + ((size_t)((row0 + b) / n_sum) * T_ + (size_t)n_sum * len) * D);
          for (int i = tid; i < tail * D / 8; i += kThreads) dst[i] = make_uint4(0, 0, 0, 0);
        }
    }
  }
  // ---- the CTA's sums -------------------------------------------------------------------------
#pragma unroll
  for (int j = 0; j < kLoads; ++j) {
    float v = dwacc[j];
#pragma unroll
    for (int o = VL >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int r = rg + j * RG;
    if (vl == 0 && r < len) atomicAdd(dw + r, v);
  }
  if (tid < D) atomicAdd(acc_dp + tid, sdp);
  if (owns) {
#pragma unroll
    for (int a = 0; a < kTile; ++a)
#pragma unroll
      for (int c = 0; c < kTile; c += kVec) {
        float* at = acc_proj + (size_t)(to * kTile + a) * D + ti * kTile + c;
        if constexpr (kVec == 4)
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(at), "f"(pacc[a][c]), "f"(pacc[a][c + 1]), "f"(pacc[a][c + 2]),
                       "f"(pacc[a][c + 3]) : "memory");
        else
          asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(at), "f"(pacc[a][c]), "f"(pacc[a][c + 1]) : "memory");
      }
  }
  __syncthreads();
  for (int r = tid; r < len; r += kThreads) atomicAdd(acc_w + r, dw[r]);
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(arrived, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // ---- d_intra[pos][d] = w[pos] * sum_dp[d];  d_logits = w * (d_w - sum(d_w * w)), where d_w also
  // takes the share of intra_pos: sum_d sum_dp[d] * intra_pos[pos][d] -------------------------------
  float* sdps = go;
  if (tid < D) sdps[tid] = __ldcg(acc_dp + tid);
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31;
  for (int r = warp; r < len; r += kThreads / 32) {
    float v = 0.f;
    for (int d = lane; d < D; d += 32) v = fmaf(sdps[d], __ldg(s.intra[side] + (size_t)r * D + d), v);
    v = warp_sum(v);
    if (lane == 0) dw[r] = __ldcg(acc_w + r) + v;
  }
  __syncthreads();
  float dot = 0.f;
  for (int r = 0; r < len; ++r) dot = fmaf(dw[r], w[r], dot);
  for (int r = tid; r < len; r += kThreads) s.d_logits[side][r] = w[r] * (dw[r] - dot);
  for (int i = tid; i < len * D; i += kThreads) s.d_intra[side][i] = w[i / D] * sdps[i % D];
  // (several vectors in flight: one at a time, this copy was half of a short call)
  constexpr int kCopy = (D * D / 4 + kThreads - 1) / kThreads;
  float4 out[kCopy];
#pragma unroll
  for (int k = 0; k < kCopy; ++k) {
    const int i = tid + k * kThreads;
    if (i < D * D / 4) out[k] = __ldcg(reinterpret_cast<const float4*>(acc_proj) + i);
  }
  const bool vec = (reinterpret_cast<uintptr_t>(s.d_proj[side]) & 15) == 0;
#pragma unroll
  for (int k = 0; k < kCopy; ++k) {
    const int i = tid + k * kThreads;
    if (i >= D * D / 4) continue;
    float* dst = s.d_proj[side] + 4 * i;
    if (vec) {
      *reinterpret_cast<float4*>(dst) = out[k];
    } else {
      dst[0] = out[k].x; dst[1] = out[k].y; dst[2] = out[k].z; dst[3] = out[k].w;
    }
  }
}

// dx of overlapping windows (stride < len): token pos of (b, h) collects w[pos - j*stride] *
// d_pooled[j] from every window j that holds it; one thread per 8 columns.
__global__ void pool_dx_kernel(const PoolSides s, int T_, int D, int len, int stride, int n_sum, size_t n_vec) {
  extern __shared__ float4 sm4[];
  float* w = reinterpret_cast<float*>(sm4);
  const int side = blockIdx.y;
  pool_weights(s.logits[side], w, w + len, len);
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_vec) return;
  const float* __restrict__ d_pooled = s.d_pooled[side];
  const int VL = D >> 3;
  const int vl = (int)(i % VL);
  const int pos = (int)((i / VL) % T_);
  const size_t bh = i / ((size_t)VL * T_);
  const int j_hi = min(n_sum - 1, pos / stride);
  const int j_lo = max(0, (pos - len + stride) / stride);   // ceil((pos - len + 1) / stride) for pos >= len - 1
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int j = j_lo; j <= j_hi; ++j) {
    const float wj = w[pos - j * stride];
    const float4 lo = __ldg(reinterpret_cast<const float4*>(d_pooled + (bh * n_sum + j) * D + vl * 8));
    const float4 hi = __ldg(reinterpret_cast<const float4*>(d_pooled + (bh * n_sum + j) * D + vl * 8 + 4));
    acc[0] = fmaf(wj, lo.x, acc[0]); acc[1] = fmaf(wj, lo.y, acc[1]); acc[2] = fmaf(wj, lo.z, acc[2]); acc[3] = fmaf(wj, lo.w, acc[3]);
    acc[4] = fmaf(wj, hi.x, acc[4]); acc[5] = fmaf(wj, hi.y, acc[5]); acc[6] = fmaf(wj, hi.z, acc[6]); acc[7] = fmaf(wj, hi.w, acc[7]);
  }
  uint4 o;
  o.x = pack2(acc[0], acc[1]); o.y = pack2(acc[2], acc[3]); o.z = pack2(acc[4], acc[5]); o.w = pack2(acc[6], acc[7]);
  *reinterpret_cast<uint4*>((__nv_bfloat16*)s.dx[side] + i * 8) = o;
}

// ---- mean pooling: 16 bytes of columns per thread, the window's tokens added in order ----------
template <typename T> struct Vec;
template <> struct Vec<__nv_bfloat16> {
  static constexpr int N = 8;
  static __device__ __forceinline__ void unpack(const uint4& u, float* f) { unpack8(u, f); }
  static __device__ __forceinline__ uint4 pack(const float* f) {
    return make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
  }
};
template <> struct Vec<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void unpack(const uint4& u, float* f) {
    f[0] = __uint_as_float(u.x); f[1] = __uint_as_float(u.y); f[2] = __uint_as_float(u.z); f[3] = __uint_as_float(u.w);
  }
  static __device__ __forceinline__ uint4 pack(const float* f) {
    return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
  }
};

// A warp to a summary: Dv lanes side by side on a token's 16-byte vectors, 32 / Dv tokens at a time, whose sums meet by
// shuffles.  A thread that walked all tokens of its columns waited for one load chain of 64 in four: 21 us for
// 2 x 4 x 4096 tokens of 64 bf16, 5 so.
template <typename T>
__global__ void mean_fwd_kernel(const PoolSides s, int T_, int Dv, int len, int n_sum, size_t rows) {
  chain_go();
  constexpr int N = Vec<T>::N;
  const size_t row = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31, d = lane & (Dv - 1), step = 32 / Dv;      // Dv: a power of two up to 32 (pool_mean_ok)
  const size_t bh = row / n_sum, j = row % n_sum;
  const uint4* p = reinterpret_cast<const uint4*>(s.x[blockIdx.y]) + (bh * T_ + j * len) * Dv + d;
  float a[N];
#pragma unroll
  for (int e = 0; e < N; ++e) a[e] = 0.f;
#pragma unroll 8
  for (int r = lane / Dv; r < len; r += step) {
    float f[N];
    Vec<T>::unpack(__ldg(p + (size_t)r * Dv), f);
#pragma unroll
    for (int e = 0; e < N; ++e) a[e] += f[e];
  }
  for (int o = Dv; o < 32; o <<= 1)
#pragma unroll
    for (int e = 0; e < N; ++e) a[e] += __shfl_xor_sync(0xffffffffu, a[e], o);
#pragma unroll
  for (int e = 0; e < N; ++e) a[e] /= (float)len;
  if (lane < Dv) reinterpret_cast<uint4*>(s.out[blockIdx.y])[row * Dv + d] = Vec<T>::pack(a);
}

template <typename T>
__global__ void mean_bwd_kernel(const PoolSides s, int T_, int Dv, int len, int n_sum, size_t n_in) {
  constexpr int N = Vec<T>::N;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_in) return;
  const int d = (int)(i % Dv);
  const size_t row = i / Dv;
  const size_t bh = row / T_;
  const int j = (int)(row % T_) / len;
  float g[N];
#pragma unroll
  for (int e = 0; e < N; ++e) g[e] = 0.f;
  if (j < n_sum) {
    Vec<T>::unpack(__ldg(reinterpret_cast<const uint4*>(s.d_out[blockIdx.y]) + (bh * n_sum + j) * Dv + d), g);
#pragma unroll
    for (int e = 0; e < N; ++e) g[e] /= (float)len;
  }
  reinterpret_cast<uint4*>(s.dx[blockIdx.y])[i] = Vec<T>::pack(g);
}

// an argument error where a side's rows or matrices do not start on a 16-byte boundary
int check_vectors(const PoolSides& s) {
  for (int k = 0; k < s.n; ++k)
    NSA_CHECK_ARG(aligned16(s.x[k], s.intra[k], s.proj[k], s.out[k], s.pooled[k], s.d_out[k], s.dx[k], s.d_pooled[k]),
                  "pooling: K, V and the pooling parameters must start on a 16-byte boundary");
  return NSA_OK;
}

template <int D, int R>
int launch_pool_fwd(const PoolSides& s, int T, int len, int stride, int n_sum, int rows, cudaStream_t st) {
  const size_t smem = (PoolFwdSmem<D, R>::kFloats + 2 * (size_t)len) * sizeof(float);
  NSA_CUDA_OK(func_smem((const void*)pool_fwd_kernel<D, R>, smem));
  KernelScope ks("pool_fwd_kernel", st);
  pool_fwd_kernel<D, R><<<dim3((unsigned)((rows + R - 1) / R), s.n), kThreads, smem, st>>>(s, T, len, stride, n_sum, rows);
  return NSA_OK;
}
template <int D>
int launch_pool_fwd(const PoolSides& s, int T, int len, int stride, int n_sum, int rows, cudaStream_t st) {
  if ((long long)s.n * ((rows + 7) / 8) >= sm_count()) return launch_pool_fwd<D, 8>(s, T, len, stride, n_sum, rows, st);
  if ((long long)s.n * ((rows + 3) / 4) >= sm_count()) return launch_pool_fwd<D, 4>(s, T, len, stride, n_sum, rows, st);
  return launch_pool_fwd<D, 2>(s, T, len, stride, n_sum, rows, st);
}
template <int D>
int launch_pool_bwd(const PoolSides& s, int T, int len, int stride, int n_sum, int rows, cudaStream_t st) {
  const size_t smem = (PoolBwdSmem<D>::kFloats + 2 * (size_t)len) * sizeof(float);
  NSA_CUDA_OK(func_smem((const void*)pool_bwd_kernel<D>, smem));
  const int groups = (rows + PoolBwdSmem<D>::R - 1) / PoolBwdSmem<D>::R;
  // a CTA ends with D*D + D + len atomics: as few CTAs as keep the SMs busy (two each over both sides)
  const int grid = min(groups, max(1, 2 * sm_count() / s.n));
  KernelScope ks("pool_bwd_kernel", st);
  pool_bwd_kernel<D><<<dim3(grid, s.n), kThreads, smem, st>>>(s, T, len, stride, n_sum, rows);
  return NSA_OK;
}

}  // namespace

bool pool_learned_ok(int D, int len, int dtype) {
  return dtype == NSA_DTYPE_BF16 && (D == 16 || D == 32 || D == 64 || D == 128) && len >= 1 && len <= 1024;
}
size_t pool_acc_floats(int D, int len) { return ((size_t)D * D + D + len + 1 + 63) / 64 * 64; }

int pool_learned_fwd(const PoolSides& s, int B, int H, int T, int D, int len, int stride, cudaStream_t st) {
  if (int bad = check_vectors(s)) return bad;
  const int n_sum = pool_count(T, len, stride);
  const size_t rows = (size_t)B * H * n_sum;
  if (rows == 0) return NSA_OK;
  NSA_CHECK_ARG(rows < (1u << 30), "too many summaries");
  int rc = NSA_ERR_UNSUPPORTED;
  switch (D) {
    case 16: rc = launch_pool_fwd<16>(s, T, len, stride, n_sum, (int)rows, st); break;
    case 32: rc = launch_pool_fwd<32>(s, T, len, stride, n_sum, (int)rows, st); break;
    case 64: rc = launch_pool_fwd<64>(s, T, len, stride, n_sum, (int)rows, st); break;
    case 128: rc = launch_pool_fwd<128>(s, T, len, stride, n_sum, (int)rows, st); break;
    default: break;
  }
  if (rc != NSA_OK) return rc;
  NSA_LAUNCH_OK("pool_fwd_kernel");
  return NSA_OK;
}

int pool_learned_bwd(const PoolSides& s, int B, int H, int T, int D, int len, int stride, cudaStream_t st) {
  if (int bad = check_vectors(s)) return bad;
  const int n_sum = pool_count(T, len, stride);
  const size_t rows = (size_t)B * H * n_sum;
  NSA_CHECK_ARG(rows < (1u << 30), "too many summaries");
  const size_t n_x = (size_t)B * H * T * D;
  if (rows == 0) {
    for (int k = 0; k < s.n; ++k) {
      if (n_x) NSA_CUDA_OK(cudaMemsetAsync(s.dx[k], 0, n_x * 2, st));
      NSA_CUDA_OK(cudaMemsetAsync(s.d_intra[k], 0, (size_t)len * D * sizeof(float), st));
      NSA_CUDA_OK(cudaMemsetAsync(s.d_logits[k], 0, (size_t)len * sizeof(float), st));
      NSA_CUDA_OK(cudaMemsetAsync(s.d_proj[k], 0, (size_t)D * D * sizeof(float), st));
    }
    return NSA_OK;
  }
  int rc = NSA_ERR_UNSUPPORTED;
  switch (D) {
    case 16: rc = launch_pool_bwd<16>(s, T, len, stride, n_sum, (int)rows, st); break;
    case 32: rc = launch_pool_bwd<32>(s, T, len, stride, n_sum, (int)rows, st); break;
    case 64: rc = launch_pool_bwd<64>(s, T, len, stride, n_sum, (int)rows, st); break;
    case 128: rc = launch_pool_bwd<128>(s, T, len, stride, n_sum, (int)rows, st); break;
    default: break;
  }
  if (rc != NSA_OK) return rc;
  NSA_LAUNCH_OK("pool_bwd_kernel");
  if (stride < len) {
    KernelScope ks("pool_dx_kernel", st);
    pool_dx_kernel<<<dim3((unsigned)((n_x / 8 + 255) / 256), s.n), 256, 2 * (size_t)len * sizeof(float), st>>>(
        s, T, D, len, stride, n_sum, n_x / 8);
    NSA_LAUNCH_OK("pool_dx_kernel");
  }
  return NSA_OK;
}

// Rows of 1, 2, 4 ... 32 vectors of 16 bytes, which is how mean_fwd_kernel lays a token over the lanes of a warp.
bool pool_mean_ok(int D, int dtype) {
  const int per = dtype == NSA_DTYPE_BF16 ? 8 : 4;
  const int Dv = D / per;
  return D > 0 && D % per == 0 && Dv <= 32 && (Dv & (Dv - 1)) == 0;
}

int pool_mean_fwd(const PoolSides& s, int B, int H, int T, int D, int len, int dtype, cudaStream_t st) {
  if (int bad = check_vectors(s)) return bad;
  NSA_CHECK_ARG(pool_mean_ok(D, dtype), "mean pooling by warps: rows have to be 1, 2, 4 ... 32 vectors of 16 bytes");
  const int n_sum = T / len;
  const size_t rows = (size_t)B * H * n_sum;
  if (rows == 0) return NSA_OK;
  const int Dv = dtype == NSA_DTYPE_BF16 ? D / 8 : D / 4;
  KernelScope ks("mean_pool_fwd_kernel", st);
  const dim3 grid((unsigned)((rows + 3) / 4), s.n);
  if (dtype == NSA_DTYPE_BF16) mean_fwd_kernel<__nv_bfloat16><<<grid, 128, 0, st>>>(s, T, Dv, len, n_sum, rows);
  else mean_fwd_kernel<float><<<grid, 128, 0, st>>>(s, T, Dv, len, n_sum, rows);
  NSA_LAUNCH_OK("mean_pool_fwd_kernel");
  return NSA_OK;
}

int pool_mean_bwd(const PoolSides& s, int B, int H, int T, int D, int len, int dtype, cudaStream_t st) {
  if (int bad = check_vectors(s)) return bad;
  const int n_sum = T / len;
  const int Dv = dtype == NSA_DTYPE_BF16 ? D / 8 : D / 4;
  const size_t n = (size_t)B * H * T * Dv;
  if (n == 0) return NSA_OK;
  KernelScope ks("mean_pool_bwd_kernel", st);
  const dim3 grid((unsigned)((n + 255) / 256), s.n);
  if (dtype == NSA_DTYPE_BF16) mean_bwd_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(s, T, Dv, len, n_sum, n);
  else mean_bwd_kernel<float><<<grid, 256, 0, st>>>(s, T, Dv, len, n_sum, n);
  NSA_LAUNCH_OK("mean_pool_bwd_kernel");
  return NSA_OK;
}

}  // namespace nsa
