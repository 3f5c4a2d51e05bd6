// CUDA-core attention on tiles of 64 rows x 64 keys, fp32 arithmetic throughout: the fp32 path (D of 64: f32_tile.cu, by the
// same rules, unless the caller asks for the CUDA cores), and bf16 shapes the tcgen05 kernels do not take (D of 16 / 32, one query head per kv head, other
// block sizes).  A row is one (query token, query head); the rows of a unit are numbered token-major
// (row = t * G + head), so a tile's rows share their K / V tiles whatever the group size.
//   window, compression   the tile walks the keys its rows can see, 64 at a time
//   selection             the union of the blocks its queries list, as one run of keys, with a
//                         64-bit membership word (bit: query of the tile) per block
// These kernels are bound by the FFMA pipes: a thread holds an 8 x 4 (forward) or 4 x 4 (backward)
// patch of every product and reads its operands from shared memory as 16-byte vectors, 5 to 10 FFMAs
// per word.  The row-per-warp kernels of simt.cu re-read K and V from L1 for every row and, in
// backward, add every key's gradient by its own atomics; here one vector atomic per (row tile, key)
// does, and window / compression / selection at B=1, T=2048, 8 heads of 64 in fp32 went from
// 1.6 / 3.8 ms (forward / backward, three branches) to 0.42 / 0.68 ms.
// A row tile is one chain through its key tiles: where tiles are few a cluster of 2 or 4 CTAs shares
// it, every CTA its key tiles, and adds up O (by its maximum) or dQ through distributed shared memory in
// rank order; at that size selection goes from 299 / 453 us to 187 / 353.
#include "cluster.cuh"
#include "simt_tile.cuh"

namespace nsa {
namespace {

constexpr int kPad = 4;          // floats: 16-byte reads of 8 neighbouring rows cover all banks
constexpr int kPLd = kK + kPad;
const char* const kFwdNames[3] = {"simt_tile_fwd_win", "simt_tile_fwd_cmp", "simt_tile_fwd_slc"};
const char* const kBwdNames[3] = {"simt_tile_bwd_win", "simt_tile_bwd_cmp", "simt_tile_bwd_slc"};

// eight consecutive elements of a row as floats
__device__ __forceinline__ void load8(const float* p, float* f) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float* f) {
  const uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    f[2 * e] = __uint_as_float(w[e] << 16);
    f[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
  }
}
__device__ __forceinline__ void put8(float* dst, const float* f) {
  *reinterpret_cast<float4*>(dst) = make_float4(f[0], f[1], f[2], f[3]);
  *reinterpret_cast<float4*>(dst + 4) = make_float4(f[4], f[5], f[6], f[7]);
}
__device__ __forceinline__ void cp16(float* dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A thread's C = D / 16 columns of a row: one scalar, one float2, or float4s 64 columns apart.
template <int C> __device__ __forceinline__ int col_of(int tx, int v) { return C >= 4 ? tx * 4 + (v >> 2) * 64 + (v & 3) : tx * C + v; }
template <int C> __device__ __forceinline__ void load_cols(const float* row, int tx, float* f) {
  if constexpr (C == 1) f[0] = row[tx];
  else if constexpr (C == 2) { const float2 a = *reinterpret_cast<const float2*>(row + tx * 2); f[0] = a.x; f[1] = a.y; }
  else
#pragma unroll
    for (int k = 0; k < C / 4; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(row + tx * 4 + k * 64);
      f[4 * k] = a.x; f[4 * k + 1] = a.y; f[4 * k + 2] = a.z; f[4 * k + 3] = a.w;
    }
}
template <int C> __device__ __forceinline__ void red_cols(float* row, int tx, const float* f) {
  if constexpr (C == 1) atomicAdd(row + tx, f[0]);
  else if constexpr (C == 2)
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(row + tx * 2), "f"(f[0]), "f"(f[1]) : "memory");
  else
#pragma unroll
    for (int k = 0; k < C / 4; ++k)
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(row + tx * 4 + k * 64), "f"(f[4 * k]),
                   "f"(f[4 * k + 1]), "f"(f[4 * k + 2]), "f"(f[4 * k + 3])
                   : "memory");
}
__device__ __forceinline__ void store_val(float* p, float v) { *p = v; }
__device__ __forceinline__ void store_val(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
template <int C, typename T> __device__ __forceinline__ void store_cols(T* row, int tx, const float* f) {
#pragma unroll
  for (int v = 0; v < C; ++v) store_val(row + col_of<C>(tx, v), f[v]);
}

// one K or V tile into shared memory [64][D + 4]; keys that do not exist read as zero
template <typename T, int D, int kThreads>
__device__ __forceinline__ void load_keys(float* dst, const T* __restrict__ base, const int* tok) {
  constexpr int LD = D + kPad;
  if constexpr (sizeof(T) == 4) {
    constexpr int kPer = D / 4;
#pragma unroll
    for (int i = threadIdx.x; i < kK * kPer; i += kThreads) {
      const int r = i / kPer, c = (i % kPer) * 4, t = tok[r];
      cp16(dst + r * LD + c, reinterpret_cast<const float*>(base) + (size_t)max(t, 0) * D + c, t >= 0);
    }
  } else {
    constexpr int kPer = D / 8;
#pragma unroll
    for (int i = threadIdx.x; i < kK * kPer; i += kThreads) {
      const int r = i / kPer, c = (i % kPer) * 8, t = tok[r];
      float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (t >= 0) load8(base + (size_t)t * D + c, f);
      put8(dst + r * LD + c, f);
    }
  }
}

// Whether a value of the tile that this thread has put into shared memory is infinite or NaN; the loop is load_keys'.
template <typename T, int D, int kThreads>
__device__ __forceinline__ bool non_finite(const float* tile) {
  constexpr int LD = D + kPad, kPer = D / (sizeof(T) == 4 ? 4 : 8), kVec = sizeof(T) == 4 ? 1 : 2;
  float z = 0.f;                                         // x * 0: 0 or NaN
#pragma unroll
  for (int i = threadIdx.x; i < kK * kPer; i += kThreads) {
#pragma unroll
    for (int k = 0; k < kVec; ++k) {
      const float4 v = *reinterpret_cast<const float4*>(tile + (i / kPer) * LD + (i % kPer) * 4 * kVec + 4 * k);
      z = fmaf(v.x, 0.f, z); z = fmaf(v.y, 0.f, z); z = fmaf(v.z, 0.f, z); z = fmaf(v.w, 0.f, z);
    }
  }
  return z != 0.f;
}

template <int D> constexpr size_t fwd_floats() { return (size_t)3 * kR * (D + kPad) + (size_t)kR * kPLd; }
template <int D> constexpr size_t bwd_floats() { return (size_t)4 * kR * (D + kPad) + (size_t)2 * kR * kPLd; }

constexpr int kFwdThreads = 128;
constexpr int kBwdThreads = 256;

// Forward.  Thread (tx, ty) = (tid % 16, tid / 16) owns rows ty + 8 i (i < 8), keys tx + 16 j (j < 4) of
// S and D / 16 columns of O.  V travels while S is computed, the next K while O is.
template <typename T, int D>
__global__ void __launch_bounds__(kFwdThreads)
simt_tile_fwd_kernel(const AttnArgs a, const int csize) {
  constexpr int LD = D + kPad, C = D / 16;
  extern __shared__ float4 sm4[];
  float* sQ = reinterpret_cast<float*>(sm4);
  float* sK = sQ + kR * LD;
  float* sV = sK + kK * LD;
  float* sP = sV + kK * LD;
  KeyInfo* ki = reinterpret_cast<KeyInfo*>(sP + kR * kPLd);
  const SelList sl = sel_list(a, ki + 1);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int G = a.Hq / a.Hkv, n_rows = a.T * G, tiles = (n_rows + kR - 1) / kR;
  const int rank = (int)blockIdx.x & (csize - 1), work = (int)blockIdx.x / csize;    // the cluster's CTAs take its key tiles in turn
  const int bh = work / tiles, b = bh / a.Hkv, hkv = bh % a.Hkv;
  const int row0 = (tiles - 1 - work % tiles) * kR;                  // long rows first
  const int t_first = row0 / G, t_last = (min(row0 + kR, n_rows) - 1) / G;
  auto row_ptr = [&](int r) -> size_t {                              // row r of the tile in [B, Hq, T]
    const int f = row0 + r;
    return ((size_t)b * a.Hq + hkv * G + f % G) * a.T + f / G;
  };
  const TileKeys tk = tile_keys<kFwdThreads>(a, bh, t_first, t_last, sl);
  const bool repeats = a.kind == 2 && *sl.repeats;
  const int n_kt = (tk.n + kK - 1) / kK;
  const T* kbase = reinterpret_cast<const T*>(a.k) + (size_t)bh * a.Lk * D;
  const T* vbase = reinterpret_cast<const T*>(a.v) + (size_t)bh * a.Lk * D;
  for (int i = tid; i < kR * D / 8; i += kFwdThreads) {
    const int r = i / (D / 8), c = (i % (D / 8)) * 8;
    float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (row0 + r < n_rows) load8(reinterpret_cast<const T*>(a.q) + row_ptr(r) * D + c, f);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= a.scale;
    put8(sQ + r * LD + c, f);
  }
  int lo[8], hi[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int f = row0 + ty + 8 * i;
    lo[i] = 0; hi[i] = -1;
    if (f < n_rows) row_range(a, f / G, lo[i], hi[i]);
  }
  float m[8], l[8], o[8][C];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < C; ++c) o[i][c] = 0.f;
  }
  if (rank < n_kt) {
    fill_keys<true>(a, tk, sl, ki, 0, rank);
    __syncthreads();
    load_keys<T, D, kFwdThreads>(sK, kbase, ki->tok[0]);
    cp_commit();
    load_keys<T, D, kFwdThreads>(sV, vbase, ki->tok[0]);
    cp_commit();
  }
  int buf = 0;
  for (int kt = rank; kt < n_kt; kt += csize, buf ^= 1) {
    const bool more = kt + csize < n_kt;
    cp_wait<1>();
    __syncthreads();
    float s[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
      float4 kv[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(sK + (tx + 16 * j) * LD + d);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 qv = *reinterpret_cast<const float4*>(sQ + (ty + 8 * i) * LD + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[i][j] = fmaf(qv.x, kv[j].x, s[i][j]); s[i][j] = fmaf(qv.y, kv[j].y, s[i][j]);
          s[i][j] = fmaf(qv.z, kv[j].z, s[i][j]); s[i][j] = fmaf(qv.w, kv[j].w, s[i][j]);
        }
      }
    }
    int tok[4];
    unsigned long long mk[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) { tok[j] = ki->tok[buf][tx + 16 * j]; mk[j] = ki->mask[buf][tx + 16 * j]; }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int ql = (row0 + ty + 8 * i) / G - t_first;
      float mx = -INFINITY;
      bool ok[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        ok[j] = tok[j] >= lo[i] && tok[j] <= hi[i];
        if (a.kind == 2) ok[j] = ok[j] && ((mk[j] >> ql) & 1ull);
        s[i][j] = ok[j] ? s[i][j] : -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int w = 8; w >= 1; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
      const float m_new = fmaxf(m[i], mx);
      const float ms = m_new == -INFINITY ? 0.f : m_new;
      const float alpha = expf(m[i] - ms);               // m = -inf: 0
      m[i] = m_new;
      l[i] *= alpha;
#pragma unroll
      for (int c = 0; c < C; ++c) o[i][c] *= alpha;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float e = expf(s[i][j] - m_new);           // for all: a select below, not a branch around it
        const float p = ok[j] ? e : kMasked;
        l[i] += p;
        sP[(ty + 8 * i) * kPLd + tx + 16 * j] = p;
      }
    }
    if (repeats) {                        // this thread's places once more
#pragma unroll
      for (int i = 0; i < 8; ++i) {
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
          float* p = sP + (ty + 8 * i) * kPLd + tx + 16 * j;
          const float one = *p;
          const int n = attended(one) ? times_listed(a, bh, (row0 + ty + 8 * i) / G, ki->tok[buf][tx + 16 * j]) : 1;
          if (n > 1) {
            *p = one * (float)n;
            l[i] += one * (float)(n - 1);
          }
        }
      }
    }
    if (more) fill_keys<true>(a, tk, sl, ki, buf ^ 1, kt + csize);
    __syncthreads();
    if (more) load_keys<T, D, kFwdThreads>(sK, kbase, ki->tok[buf ^ 1]);
    cp_commit();
    cp_wait<1>();
    if (__syncthreads_or(non_finite<T, D, kFwdThreads>(sV))) {
#pragma unroll 1
      for (int k = 0; k < kK; ++k) {
        float v[C];
        load_cols<C>(sV + k * LD, tx, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float p = sP[(ty + 8 * i) * kPLd + k];
          if (attended(p))
#pragma unroll
            for (int c = 0; c < C; ++c) o[i][c] = fmaf(p, v[c], o[i][c]);
        }
      }
    } else
#pragma unroll 2
    for (int k = 0; k < kK; k += 4) {
      float v[4][C];
#pragma unroll
      for (int e = 0; e < 4; ++e) load_cols<C>(sV + (k + e) * LD, tx, v[e]);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 p = *reinterpret_cast<const float4*>(sP + (ty + 8 * i) * kPLd + k);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          o[i][c] = fmaf(p.x, v[0][c], o[i][c]); o[i][c] = fmaf(p.y, v[1][c], o[i][c]);
          o[i][c] = fmaf(p.z, v[2][c], o[i][c]); o[i][c] = fmaf(p.w, v[3][c], o[i][c]);
        }
      }
    }
    __syncthreads();
    if (more) load_keys<T, D, kFwdThreads>(sV, vbase, ki->tok[buf ^ 1]);
    cp_commit();
  }
  cp_wait<0>();
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int w = 8; w >= 1; w >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], w);
  if (csize > 1) {
    // every CTA leaves what its keys gave (O over the K tile; m and l over P); the rows are dealt out for the sum
    float* sO = sK;
    float* sM = sP;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int c = 0; c < C; ++c) sO[(ty + 8 * i) * LD + col_of<C>(tx, c)] = o[i][c];
      if (tx == 0) { sM[ty + 8 * i] = m[i]; sM[kR + ty + 8 * i] = l[i]; }
    }
    cluster_sync();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if ((i & (csize - 1)) != rank) continue;
      const int r = ty + 8 * i;
      float mx = -INFINITY;
      for (int k = 0; k < csize; ++k) mx = fmaxf(mx, ld_peer_f32(sM + r, k));
      const float ms = mx == -INFINITY ? 0.f : mx;
      l[i] = 0.f;
#pragma unroll
      for (int c = 0; c < C; ++c) o[i][c] = 0.f;
      for (int k = 0; k < csize; ++k) {
        const float w = expf(ld_peer_f32(sM + r, k) - ms);
        l[i] = fmaf(w, ld_peer_f32(sM + kR + r, k), l[i]);
#pragma unroll
        for (int c = 0; c < C; ++c) o[i][c] = fmaf(w, ld_peer_f32(sO + r * LD + col_of<C>(tx, c), k), o[i][c]);
      }
      m[i] = mx;
    }
    cluster_sync();                       // nobody leaves while its memory is read
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if ((i & (csize - 1)) != rank) continue;
    if (row0 + ty + 8 * i < n_rows) {
      const size_t row = row_ptr(ty + 8 * i);
      const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
#pragma unroll
      for (int c = 0; c < C; ++c) o[i][c] *= inv;
      store_cols<C>(reinterpret_cast<T*>(a.o) + row * D, tx, o[i]);
      if (tx == 0 && a.lse) a.lse[row] = l[i] > 0.f ? m[i] + logf(l[i]) : kLseEmpty;
    }
  }
}

// Backward.  Thread (tx, ty) = (tid % 16, tid / 16) owns rows ty + 16 i, keys tx + 16 j of S and dP, and D / 16
// columns of dQ (rows ty + 16 i) and of dK / dV (keys 4 ty + e), which leave by vector atomics.
template <typename T, int D>
__global__ void __launch_bounds__(kBwdThreads, D <= 64 ? 2 : 1)
simt_tile_bwd_kernel(const AttnArgs a, const int csize) {
  constexpr int LD = D + kPad, C = D / 16;
  extern __shared__ float4 sm4[];
  float* sQ = reinterpret_cast<float*>(sm4);
  float* sDO = sQ + kR * LD;
  float* sK = sDO + kR * LD;
  float* sV = sK + kK * LD;
  float* sP = sV + kK * LD;
  float* sDS = sP + kR * kPLd;
  KeyInfo* ki = reinterpret_cast<KeyInfo*>(sDS + kR * kPLd);
  const SelList sl = sel_list(a, ki + 1);
  __shared__ float s_lse[kR], s_delta[kR];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int G = a.Hq / a.Hkv, n_rows = a.T * G, tiles = (n_rows + kR - 1) / kR;
  const int rank = (int)blockIdx.x & (csize - 1), work = (int)blockIdx.x / csize;
  const int bh = work / tiles, b = bh / a.Hkv, hkv = bh % a.Hkv;
  const int row0 = (tiles - 1 - work % tiles) * kR;
  const int t_first = row0 / G, t_last = (min(row0 + kR, n_rows) - 1) / G;
  auto row_ptr = [&](int r) -> size_t {
    const int f = row0 + r;
    return ((size_t)b * a.Hq + hkv * G + f % G) * a.T + f / G;
  };
  const TileKeys tk = tile_keys<kBwdThreads>(a, bh, t_first, t_last, sl);
  const bool repeats = a.kind == 2 && *sl.repeats;
  const int n_kt = (tk.n + kK - 1) / kK;
  const size_t kvoff = (size_t)bh * a.Lk * D;
  const T* kbase = reinterpret_cast<const T*>(a.k) + kvoff;
  const T* vbase = reinterpret_cast<const T*>(a.v) + kvoff;
  float* dkb = a.dk_acc + kvoff;
  float* dvb = a.dv_acc + kvoff;
  if (rank < n_kt) fill_keys<true>(a, tk, sl, ki, 0, rank);
  // Q (scaled), dO (times the gate of a gated branch), lse and delta; four threads per row
  bool rows_bad;                        // a value of Q or dO is infinite or NaN
  {
    const int r = tid >> 2, part = tid & 3;
    const bool in = row0 + r < n_rows;
    const size_t row = in ? row_ptr(r) : 0;
    const float rs = in && a.row_scale ? a.row_scale[row] : 1.f;
    float dot = 0.f, z = 0.f;
    for (int c = part * 8; c < D; c += 32) {
      float q[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, g[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (in) {
        load8(reinterpret_cast<const T*>(a.q) + row * D + c, q);
        load8(reinterpret_cast<const T*>(a.d_o) + row * D + c, g);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        q[e] *= a.scale; g[e] *= rs;
        z = fmaf(q[e], 0.f, z); z = fmaf(g[e], 0.f, z);
      }
      if (in && !a.row_dot) {
        float o[8];
        load8(reinterpret_cast<const T*>(a.o) + row * D + c, o);
#pragma unroll
        for (int e = 0; e < 8; ++e) dot = fmaf(g[e], o[e], dot);
      }
      put8(sQ + r * LD + c, q);
      put8(sDO + r * LD + c, g);
    }
    dot += __shfl_xor_sync(0xffffffffu, dot, 1);
    dot += __shfl_xor_sync(0xffffffffu, dot, 2);
    if (part == 0) {
      s_lse[r] = in ? a.lse[row] : 0.f;
      s_delta[r] = in ? (a.row_dot ? rs * a.row_dot[row] : dot) : 0.f;
    }
    rows_bad = z != 0.f;
  }
  rows_bad = __syncthreads_or(rows_bad);
  int lo[4], hi[4];
  float lse[4], delta[4], dq[4][C];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int f = row0 + ty + 16 * i;
    lo[i] = 0; hi[i] = -1;
    if (f < n_rows) row_range(a, f / G, lo[i], hi[i]);
    lse[i] = s_lse[ty + 16 * i];
    delta[i] = s_delta[ty + 16 * i];
#pragma unroll
    for (int c = 0; c < C; ++c) dq[i][c] = 0.f;
  }
  if (rank < n_kt) {
    load_keys<T, D, kBwdThreads>(sV, vbase, ki->tok[0]);
    load_keys<T, D, kBwdThreads>(sK, kbase, ki->tok[0]);
    cp_commit();
  }
  int buf = 0;
  for (int kt = rank; kt < n_kt; kt += csize, buf ^= 1) {
    const bool more = kt + csize < n_kt;
    cp_wait<0>();
    const bool bad = __syncthreads_or(non_finite<T, D, kBwdThreads>(sK) || non_finite<T, D, kBwdThreads>(sV)) || rows_bad;
    float s[4][4], dp[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) { s[i][j] = 0.f; dp[i][j] = 0.f; }
#pragma unroll 2
    for (int d = 0; d < D; d += 4) {
      float4 kv[4], vv[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        kv[j] = *reinterpret_cast<const float4*>(sK + (tx + 16 * j) * LD + d);
        vv[j] = *reinterpret_cast<const float4*>(sV + (tx + 16 * j) * LD + d);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 qv = *reinterpret_cast<const float4*>(sQ + (ty + 16 * i) * LD + d);
        const float4 gv = *reinterpret_cast<const float4*>(sDO + (ty + 16 * i) * LD + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[i][j] = fmaf(qv.x, kv[j].x, s[i][j]); s[i][j] = fmaf(qv.y, kv[j].y, s[i][j]);
          s[i][j] = fmaf(qv.z, kv[j].z, s[i][j]); s[i][j] = fmaf(qv.w, kv[j].w, s[i][j]);
          dp[i][j] = fmaf(gv.x, vv[j].x, dp[i][j]); dp[i][j] = fmaf(gv.y, vv[j].y, dp[i][j]);
          dp[i][j] = fmaf(gv.z, vv[j].z, dp[i][j]); dp[i][j] = fmaf(gv.w, vv[j].w, dp[i][j]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int tok = ki->tok[buf][tx + 16 * j];
      const unsigned long long mk = ki->mask[buf][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        bool ok = tok >= lo[i] && tok <= hi[i];
        if (a.kind == 2) ok = ok && ((mk >> ((row0 + ty + 16 * i) / G - t_first)) & 1ull);
        const float e = expf(s[i][j] - lse[i]);          // for all: a select below, not a branch around it
        const float p = ok ? e : kMasked;
        sP[(ty + 16 * i) * kPLd + tx + 16 * j] = p;
        sDS[(ty + 16 * i) * kPLd + tx + 16 * j] = ok ? p * (dp[i][j] - delta[i]) : 0.f;
      }
    }
    if (repeats) {                        // this thread's places once more
#pragma unroll 1
      for (int e = 0; e < 16; ++e) {
        const int at = (ty + 16 * (e >> 2)) * kPLd + tx + 16 * (e & 3);
        const int n = attended(sP[at]) ? times_listed(a, bh, (row0 + ty + 16 * (e >> 2)) / G, ki->tok[buf][tx + 16 * (e & 3)]) : 1;
        if (n > 1) { sP[at] *= (float)n; sDS[at] *= (float)n; }
      }
    }
    if (more) fill_keys<true>(a, tk, sl, ki, buf ^ 1, kt + csize);
    __syncthreads();
    if (more) load_keys<T, D, kBwdThreads>(sV, vbase, ki->tok[buf ^ 1]);
    // dQ += dS K
    if (bad) {
#pragma unroll 1
      for (int k = 0; k < kK; ++k) {
        float v[C];
        load_cols<C>(sK + k * LD, tx, v);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float ds = sDS[(ty + 16 * i) * kPLd + k];
          if (attended(sP[(ty + 16 * i) * kPLd + k]))
#pragma unroll
            for (int c = 0; c < C; ++c) dq[i][c] = fmaf(ds, v[c], dq[i][c]);
        }
      }
    } else
#pragma unroll 2
    for (int k = 0; k < kK; k += 4) {
      float v[4][C];
#pragma unroll
      for (int e = 0; e < 4; ++e) load_cols<C>(sK + (k + e) * LD, tx, v[e]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 p = *reinterpret_cast<const float4*>(sDS + (ty + 16 * i) * kPLd + k);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          dq[i][c] = fmaf(p.x, v[0][c], dq[i][c]); dq[i][c] = fmaf(p.y, v[1][c], dq[i][c]);
          dq[i][c] = fmaf(p.z, v[2][c], dq[i][c]); dq[i][c] = fmaf(p.w, v[3][c], dq[i][c]);
        }
      }
    }
    __syncthreads();
    if (more) load_keys<T, D, kBwdThreads>(sK, kbase, ki->tok[buf ^ 1]);
    cp_commit();
    // dV += P^T dO and dK += dS^T Q (Q carries the scale), one after the other to spare registers
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      const float* w = which ? sDS : sP;
      const float* x = which ? sQ : sDO;
      float acc[4][C];
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int c = 0; c < C; ++c) acc[e][c] = 0.f;
      if (bad) {
#pragma unroll 1
        for (int r = 0; r < kR; ++r) {
          float v[C];
          load_cols<C>(x + r * LD, tx, v);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float we = w[r * kPLd + ty * 4 + e];
            if (attended(sP[r * kPLd + ty * 4 + e]))
#pragma unroll
              for (int c = 0; c < C; ++c) acc[e][c] = fmaf(we, v[c], acc[e][c]);
          }
        }
      } else
#pragma unroll 4
      for (int r = 0; r < kR; ++r) {
        const float4 p = *reinterpret_cast<const float4*>(w + r * kPLd + ty * 4);
        float v[C];
        load_cols<C>(x + r * LD, tx, v);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          acc[0][c] = fmaf(p.x, v[c], acc[0][c]); acc[1][c] = fmaf(p.y, v[c], acc[1][c]);
          acc[2][c] = fmaf(p.z, v[c], acc[2][c]); acc[3][c] = fmaf(p.w, v[c], acc[3][c]);
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int tok = ki->tok[buf][ty * 4 + e];
        if (tok >= 0) red_cols<C>((which ? dkb : dvb) + (size_t)tok * D, tx, acc[e]);
      }
    }
  }
  if (csize > 1) {                        // dQ of the cluster's CTAs, over their K tiles, in rank order
    float* sD = sK;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < C; ++c) sD[(ty + 16 * i) * LD + col_of<C>(tx, c)] = dq[i][c];
    cluster_sync();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if ((i & (csize - 1)) != rank) continue;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        dq[i][c] = 0.f;
        for (int k = 0; k < csize; ++k) dq[i][c] += ld_peer_f32(sD + (ty + 16 * i) * LD + col_of<C>(tx, c), k);
      }
    }
    cluster_sync();                       // nobody leaves while its memory is read
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if ((i & (csize - 1)) == rank && row0 + ty + 16 * i < n_rows) {
#pragma unroll
      for (int c = 0; c < C; ++c) dq[i][c] *= a.scale;
      store_cols<C>(reinterpret_cast<T*>(a.dq) + row_ptr(ty + 16 * i) * D, tx, dq[i]);
    }
}

// CTAs that share a row tile, each taking every csize-th key tile.  A row tile is one long chain; with few of them the
// longest is what the call waits for.  The lines, in row tiles per SM (fp32, D = 64, 8 heads on 2; alone | 2 | 4 CTAs a
// tile, us): selection at 0.86 forward 132 | 93 | 66, backward 232 | 180 | 125; at 1.7 310 | 189 | 182 and
// 640 | 355 | 399; at 6.9 650 | 615 | 678 and 1507 | 1345 | 1499; at 21 1648 | 1691 | 2021 and 3935 | 3994 | 4467.
// Window (chains of 9 key tiles) at 0.4 69 | 44 | 37 and 109 | 64 | 55; at 1.3 101 | 78 | 90 and 196 | 145 | 159; at 1.7
// 103 | 98 | 121 and 199 | 215 | 225.  At D = 128 a tile has an SM to itself: sharing only fills idle SMs.
int cluster_size(const AttnArgs& a) {
  const long long tiles = n_tiles(a), sms = sm_count();
  const long long n_kt = ((a.kind == 0 ? (long long)a.window + kR / (a.Hq / a.Hkv) : a.Lk) + kK - 1) / kK;    // (any window)
  int csize = 1;
  if (a.D > 64) csize = 4 * tiles <= sms ? 4 : 2 * tiles <= sms ? 2 : 1;
  else if (a.kind == 2) csize = tiles <= sms ? 4 : tiles <= 7 * sms ? 2 : 1;
  else csize = 2 * tiles <= sms ? 4 : 3 * tiles <= 4 * sms ? 2 : 1;
  while (csize > 1 && n_kt < 2 * csize) csize >>= 1;
  return csize;
}

template <typename T, int D>
int launch(const AttnArgs& a, bool bwd, cudaStream_t st) {
  const int csize = cluster_size(a);
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)csize;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)n_tiles(a) * csize);   // in x, which takes any number of units
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = csize > 1 ? 1 : 0;
  if (!bwd) {
    const size_t smem = fwd_floats<D>() * sizeof(float) + extra_smem(a);
    NSA_CUDA_OK(func_smem((const void*)simt_tile_fwd_kernel<T, D>, smem));
    KernelScope ks(branch_name(kFwdNames, a.kind), st);
    cfg.blockDim = dim3(kFwdThreads);
    cfg.dynamicSmemBytes = smem;
    NSA_CUDA_OK(cudaLaunchKernelEx(&cfg, simt_tile_fwd_kernel<T, D>, a, csize));
  } else {
    const size_t smem = bwd_floats<D>() * sizeof(float) + extra_smem(a);
    NSA_CUDA_OK(func_smem((const void*)simt_tile_bwd_kernel<T, D>, smem));
    KernelScope ks(branch_name(kBwdNames, a.kind), st);
    cfg.blockDim = dim3(kBwdThreads);
    cfg.dynamicSmemBytes = smem;
    NSA_CUDA_OK(cudaLaunchKernelEx(&cfg, simt_tile_bwd_kernel<T, D>, a, csize));
  }
  NSA_LAUNCH_OK("simt_tile kernel");
  return NSA_OK;
}
template <typename T>
int launch_d(const AttnArgs& a, bool bwd, cudaStream_t st) {
  switch (a.D) {
    case 16: return launch<T, 16>(a, bwd, st);
    case 32: return launch<T, 32>(a, bwd, st);
    case 64:
      if (sizeof(T) == 4 && !a.cuda_cores) return f32_tile_launch(a, bwd, st);       // on the tensor cores
      return launch<T, 64>(a, bwd, st);
    case 128: return launch<T, 128>(a, bwd, st);
    default: set_error("head dim %d not in {16,32,64,128}", a.D); return NSA_ERR_UNSUPPORTED;
  }
}

}  // namespace

// Whether a tile beats a row at a time.  Window and compression: always.  Selection: a tile of 64 / G
// queries works through the union of their lists, at most every block there is (half of them on
// average over a causal sequence), where a row at a time goes through its own blocks only.  At 64
// blocks of 16 tokens, 8 list slots, D = 128 and lists that share little (B=2, T=1024, 16 heads) the
// forward tile took 0.62 ms against 0.36, the backward tile 0.81 against 0.91: the lines are drawn at 4
// and 8 blocks per list slot.  And a tile is a chain through its keys, which four CTAs share
// at most, while the row kernels spread its work over 64 warps: with few tiles the rows end sooner.  In
// row tiles per SM (8 heads on 2, tile | rows, us): fp32, D = 64, blocks of 64, at 0.11 forward 29 | 27 and backward 41 | 33,
// at 0.22 33 | 42 and 44 | 73, at 0.43 39 | 125 and 62 | 251; fp32, blocks of 32, 4 listed, at 0.43 38 | 50 and 63 | 101;
// bf16, blocks of 16, 4 listed, at 0.22 34 | 25 and 47 | 31; blocks of 32, 8 listed, at 0.65 57 | 86 and 84 | 165.
// Rows must be whole 16-byte vectors.
bool simt_tile_ok(const AttnArgs& a, int dtype, bool bwd) {
  const uintptr_t p = (uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.o | (uintptr_t)a.d_o |
                      (uintptr_t)a.dq | (uintptr_t)a.dk_acc | (uintptr_t)a.dv_acc;
  if (p & 15) return false;
  if ((long long)a.T * (a.Hq / a.Hkv) >= (1LL << 31) - kR || n_tiles(a) >= (1LL << 31)) return false;
  if (a.kind != 2) return true;
  const int n_blk = (a.T + a.block_size - 1) / a.block_size;
  return n_blk <= kMaxBlocks && n_blk <= (bwd ? 8LL : 4LL) * a.S && (dtype == NSA_DTYPE_BF16 ? 2 : 5) * n_tiles(a) >= sm_count();
}

int simt_tile_fwd(const AttnArgs& a, int dtype, cudaStream_t st) {
  return dtype == NSA_DTYPE_BF16 ? launch_d<__nv_bfloat16>(a, false, st) : launch_d<float>(a, false, st);
}
int simt_tile_bwd(const AttnArgs& a, int dtype, cudaStream_t st) {
  return dtype == NSA_DTYPE_BF16 ? launch_d<__nv_bfloat16>(a, true, st) : launch_d<float>(a, true, st);
}

}  // namespace nsa
