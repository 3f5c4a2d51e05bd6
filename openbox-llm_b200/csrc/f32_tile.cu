// fp32 attention at D = 64 on the tensor cores: tiles of 64 rows x 64 keys as in simt_tile.cu, every product as six
// products of bf16 terms.
//
// An fp32 value is the sum of three bf16 terms, each what the ones before it leave of it (24 bits in all, down to values of 2^-109: below,
// the last terms fall under bf16's smallest, and NSA_IMPL_SIMT keeps what these tiles drop).  Of the nine
// products of two such sums the six largest are formed: what is left out is below 2^-26 of the product.  The tensor cores cut
// the bits that fall out of a sum off, instead of rounding, so the five small products (2^-8 of the large one and less) have
// an accumulator of their own, neither goes over more than 64 places of the contraction (320 products in the small one), and both are
// added up in fp32.  Measured over dot
// products of N(0, 1): 64 terms 0.7e-7 off the 64-bit value (a chain of 64 FFMAs 1.4e-7), 512 terms 0.9e-7 (4.1e-7), 2048
// terms 1.3e-7 (8.0e-7); with one accumulator, small products first, 3.9e-7 at 64 terms.
//
// What bounds them: mma.sync issues 1019 products a clock and SM, 170 of fp32, where FFMA does 128 at best and did
// 58 here, with both operands from shared memory.  A tile takes 3.1 k cycles of them forward and 7.7 k backward, the operands' loads from
// shared memory 2.9 k and 6 k, splits, masks and exponentials 2.6 k and 4 k issue slots; two CTAs of eight warps an SM overlap that to 6.1 k
// and 12.6 k (selection and window: tensor pipe active 46 to 49 % of the time forward, 61 to 62 % backward; compression, one key tile a CTA,
// 24 and 52 %; CUDA-core tiles 9.3 k and 21 k).  128 registers a thread, 140 bytes spilled forward and 72 backward.  Three branches of 2048 tokens, 8 heads of 64, forward and
// backward: selection 188 + 351 -> 117 + 239 us, window 100 + 195 -> 66 + 134, the pass 850 -> 550.  Slower than the CUDA-core tiles, which fit three
// CTAs an SM, is compression forward of one key tile on two to three row tiles per SM: 26.5 -> 29 us at 384 row tiles.  Tried: four warps of 16 x 64 with 168
// and 255 registers (forward 139, backward 225: the same work an SM, but a tile takes twice as long, which is what few
// tiles wait for); K and V of the next tile, or of the first, brought into L1 ahead (3 % slower, no change).  tcgen05.mma has three times this
// rate; it is not tried: each 64 places its sums would come back from tensor memory for the adds in fp32, and P and dS go there in three terms.
//
// Values that the split cannot carry (infinite, NaN, or from 2^60 on, where its products could overflow) are zeros in the products,
// eight neighbouring columns at a time, and noted by row and columns; what attends them is put right by FFMAs.  Rows that
// do not keep their bits.
#include "cluster.cuh"
#include "simt_tile.cuh"

namespace nsa {
namespace {

constexpr int D = 64;
constexpr int kThreads = 256;                     // eight warps
constexpr int kTermBytes = kR * D * 2;            // one term of a tile: 64 rows of 128 bytes, 16-byte chunks swizzled by the row
constexpr int kTileBytes = 3 * kTermBytes;
constexpr uint32_t kTooLarge = 0x5d80u;           // 2^60 in bf16
constexpr int kLd = D + 4;
const char* const kFwdNames[3] = {"f32_tile_fwd_win", "f32_tile_fwd_cmp", "f32_tile_fwd_slc"};
const char* const kBwdNames[3] = {"f32_tile_bwd_win", "f32_tile_bwd_cmp", "f32_tile_bwd_slc"};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// the three terms of two values
__device__ __forceinline__ void split2(float x, float y, uint32_t& t0, uint32_t& t1, uint32_t& t2) {
  t0 = pack2(x, y);
  x -= __uint_as_float(t0 << 16); y -= __uint_as_float(t0 & 0xffff0000u);
  t1 = pack2(x, y);
  x -= __uint_as_float(t1 << 16); y -= __uint_as_float(t1 & 0xffff0000u);
  t2 = pack2(x, y);
}
// Eight values of row r, columns 8 c ..., as terms into a tile.  Values that cannot be split: zeros, a bit in bad[r], and true.
__device__ __forceinline__ bool put_terms(uint32_t tile, uint32_t* bad, int r, int c, const float* f) {
  uint32_t t[3][4], big = 0u;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    split2(f[2 * e], f[2 * e + 1], t[0][e], t[1][e], t[2][e]);
    big = __vmaxu2(big, t[0][e] & 0x7fff7fffu);
  }
  const bool too_large = max(big & 0xffffu, big >> 16) >= kTooLarge;
  if (too_large) {
    atomicOr(bad + r, 1u << c);
#pragma unroll
    for (int e = 0; e < 4; ++e) t[0][e] = t[1][e] = t[2][e] = 0u;
  }
  const uint32_t at = tile + r * 128 + ((c ^ (r & 7)) << 4);
#pragma unroll
  for (int m = 0; m < 3; ++m)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + m * kTermBytes), "r"(t[m][0]), "r"(t[m][1]), "r"(t[m][2]),
                 "r"(t[m][3]) : "memory");
  return too_large;
}
__device__ __forceinline__ void load8(const float* p, float* f) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
// a K or V tile as terms; keys that do not exist read as zero
__device__ __forceinline__ bool load_terms(uint32_t tile, uint32_t* bad, const float* __restrict__ base, const int* tok) {
  bool any = false;
#pragma unroll
  for (int k = 0; k < kK * (D / 8) / kThreads; ++k) {
    const int i = threadIdx.x + k * kThreads, r = i >> 3, c = i & 7, t = tok[r];
    float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (t >= 0) load8(base + (size_t)t * D + 8 * c, f);
    any |= put_terms(tile, bad, r, c, f);
  }
  return any;
}
// the value at a place of a tile of terms
__device__ __forceinline__ float of_terms(const uint8_t* tile, int r, int c) {
  const uint8_t* at = tile + r * 128 + (((c >> 3) ^ (r & 7)) << 4) + (c & 7) * 2;
  float x = 0.f;
#pragma unroll
  for (int m = 2; m >= 0; --m) x += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(at + m * kTermBytes));
  return x;
}
// a dot product of two rows, the first times a factor
__device__ __noinline__ float dot_row(const float* x, float times, const float* y) {
  float s = 0.f;
#pragma unroll 4
  for (int d = 0; d < D; ++d) s = fmaf(x[d] * times, y[d], s);
  return s;
}

__device__ __forceinline__ void ldsm4(uint32_t at, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t at, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void mma(float* d, const uint32_t* a, const uint32_t* b) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// Where a lane's 16 bytes of an operand lie in a term.  A by rows (16 rows from r0, 16 columns from chunk c), or B of a tile whose
// rows are the contraction, transposed as it is read:
__device__ __forceinline__ uint32_t at_a(int lane, int r0, int c) {
  const int r = r0 + (lane & 15);
  return r * 128 + (((c + (lane >> 4)) ^ (r & 7)) << 4);
}
// B of a tile whose rows are its columns (16 of them from r0), or A of one whose rows are the contraction:
__device__ __forceinline__ uint32_t at_b(int lane, int r0, int c) {
  const int r = r0 + (lane & 7) + ((lane >> 4) << 3);
  return r * 128 + (((c + ((lane >> 3) & 1)) ^ (r & 7)) << 4);
}

// out[4][4], 16 x 32, = A B over 16 KK places: load_a(kk, a) brings the terms of A, load_b(m, kk, j, b) those of columns 8 j ... 8 j + 15
// of B.  Four accumulators in turn: one is ready again after some 35 cycles, the time of four MMAs.
template <int KK, typename LA, typename LB>
__device__ __forceinline__ void product(float (*out)[4], LA load_a, LB load_b) {
  float small[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) out[j][e] = small[j][e] = 0.f;
#pragma unroll
  for (int kk = 0; kk < KK; ++kk) {
    uint32_t a[3][4];
    load_a(kk, a);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      uint32_t b[2][4];
      load_b(m, kk, 0, b[0]);
      load_b(m, kk, 2, b[1]);
#pragma unroll
      for (int n = 2 - m; n >= 0; --n)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma(m + n ? small[j] : out[j], a[n], b[j >> 1] + 2 * (j & 1));
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) out[j][e] += small[j][e];
}
__device__ __forceinline__ void ldsm_terms(uint32_t at, uint32_t (*a)[4]) {
#pragma unroll
  for (int m = 0; m < 3; ++m) ldsm4(at + m * kTermBytes, a[m]);
}

// What a row attends of a key tile: its keys by position and, for selection, by its query's list, a bit per key.
struct RowKeys {
  int lo, hi, ql;
  __device__ __forceinline__ RowKeys(const AttnArgs& a, int f, int n_rows, int G, int t_first) : lo(0), hi(-1), ql(0) {
    if (f < n_rows) {
      ql = f / G - t_first;
      row_range(a, f / G, lo, hi);
    }
  }
  // Run by run: a tile is one run of tokens, or of selection one for each block that reaches into it.  (Key by key where blocks are not
  // multiples of 16, as it was, took longer than the products: 1000 tokens of 8 heads, 8 blocks of 40, forward 122 -> 54 us, backward 143 -> 82;
  // CUDA-core tiles 63 and 121.)
  __device__ __forceinline__ unsigned long long of_tile(const AttnArgs& a, const TileKeys& tk, const SelList& sl, int i) const {
    unsigned long long bits = 0ull;
    int slot = a.kind == 2 ? i * kK / a.block_size : 0;
    int in = a.kind == 2 ? i * kK - slot * a.block_size : 0;         // the run's first key in its block
    const int n = min(kK, tk.n - i * kK);
#pragma unroll 1
    for (int c = 0; c < n;) {
      int step = n - c, tok = tk.first + i * kK;
      bool listed = true;
      if (a.kind == 2) {
        const int b = sl.list[slot++];
        step = min(step, a.block_size - in);
        tok = b * a.block_size + in;
        in = 0;
        listed = (sl.mask[b] >> ql) & 1ull;
      }
      // (past the sequence's last token, the tokens are above hi)
      const int l = min(max(lo - tok, 0), step), h = min(max(hi - tok + 1, 0), step);
      if (listed && l < h) bits |= ((h - l == 64 ? 0ull : 1ull << (h - l)) - 1ull) << (c + l);
      c += step;
    }
    return bits;
  }
};
// bookkeeping of key tile i: its keys (threads 0 .. 63), and what each row attends of it (64 .. 127), as two words of 32 keys
__device__ __forceinline__ void fill_tile(const AttnArgs& a, const TileKeys& tk, const SelList& sl, KeyInfo* ki, uint32_t (*att)[2][kR],
                                          const RowKeys& rk, int buf, int i) {
  fill_keys<false>(a, tk, sl, ki, buf, i);
  const int r = (int)threadIdx.x - kK;
  if (r < 0 || r >= kR) return;
  const unsigned long long bits = rk.of_tile(a, tk, sl, i);
  att[buf][0][r] = (uint32_t)bits;
  att[buf][1][r] = (uint32_t)(bits >> 32);
}

// A lane holds rows lane / 4 and 8 more of its warp's 16, and of each eight columns the two from 2 (lane % 4) on.  Warps w and w + 4
// share 16 rows: they take 32 columns each.

constexpr int kFwdBytes = 3 * kTileBytes;         // Q, K, V
constexpr int kBwdBytes = 4 * kTileBytes;         // Q, dO, K, V (then dS)

__global__ void __launch_bounds__(kThreads, 2)
f32_tile_fwd_kernel(const AttnArgs a, const int csize) {
  extern __shared__ float4 sm4[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(sm4);
  const uint32_t sQ = smem_addr(smem), sK = sQ + kTileBytes, sV = sK + kTileBytes;
  KeyInfo* ki = reinterpret_cast<KeyInfo*>(smem + kFwdBytes);
  const SelList sl = sel_list(a, ki + 1);
  __shared__ uint32_t s_att[2][2][kR], s_bad[3][kR];             // (K, V, Q)
  const int tid = threadIdx.x, warp = (tid >> 5) & 3, half = tid >> 7, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int G = a.Hq / a.Hkv, n_rows = a.T * G, tiles = (n_rows + kR - 1) / kR;
  const int rank = (int)blockIdx.x & (csize - 1), work = (int)blockIdx.x / csize;    // the cluster's CTAs take its key tiles in turn
  const int units = a.B * a.Hkv, bh = work % units, b = bh / a.Hkv, hkv = bh % a.Hkv;
  const int row0 = (tiles - 1 - work / units) * kR;                  // long rows first
  const int t_first = row0 / G, t_last = (min(row0 + kR, n_rows) - 1) / G;
  auto row_ptr = [&](int r) -> size_t {                              // row r of the tile in [B, Hq, T]
    const int f = row0 + r;
    return ((size_t)b * a.Hq + hkv * G + f % G) * a.T + f / G;
  };
  const float* q = reinterpret_cast<const float*>(a.q);
  const float* kbase = reinterpret_cast<const float*>(a.k) + (size_t)bh * a.Lk * D;
  const float* vbase = reinterpret_cast<const float*>(a.v) + (size_t)bh * a.Lk * D;
  for (int i = tid; i < 3 * kR; i += kThreads) s_bad[i / kR][i % kR] = 0u;
  __syncthreads();
  const TileKeys tk = tile_keys<kThreads>(a, bh, t_first, t_last, sl);
  const bool repeats = a.kind == 2 && *sl.repeats;
  const int n_kt = (tk.n + kK - 1) / kK;
  const RowKeys rk(a, row0 + (tid & (kR - 1)), n_rows, G, t_first);
  if (rank < n_kt) fill_tile(a, tk, sl, ki, s_att, rk, 0, rank);
  bool q_bad = false;
  for (int i = tid; i < kR * D / 8; i += kThreads) {
    const int r = i >> 3, c = i & 7;
    float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (row0 + r < n_rows) load8(q + row_ptr(r) * D + 8 * c, f);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= a.scale;
    q_bad |= put_terms(sQ, s_bad[2], r, c, f);
  }
  const int row[2] = {16 * warp + g, 16 * warp + g + 8};             // this lane's two rows
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
  int buf = 0;
  for (int kt = rank; kt < n_kt; kt += csize, buf ^= 1) {
    __syncthreads();                      // the last tile is done with; this one's keys are known
    bool bad = load_terms(sK, s_bad[0], kbase, ki->tok[buf]);
    bad |= load_terms(sV, s_bad[1], vbase, ki->tok[buf]);
    bad = __syncthreads_or(bad || q_bad);
    if (kt + csize < n_kt) fill_tile(a, tk, sl, ki, s_att, rk, buf ^ 1, kt + csize);
    const int key0 = 32 * half + 2 * t4;             // this lane's keys: key0 + 8 j and the next
    float s[4][4];
    product<D / 16>(s, [&](int kk, uint32_t (*x)[4]) { ldsm_terms(sQ + at_a(lane, 16 * warp, 2 * kk), x); },
                    [&](int t, int kk, int j, uint32_t* y) { ldsm4(sK + t * kTermBytes + at_b(lane, 32 * half + 8 * j, 2 * kk), y); });
    float mx[2] = {-INFINITY, -INFINITY};
    const uint32_t in[2] = {s_att[buf][half][row[0]] >> (2 * t4), s_att[buf][half][row[1]] >> (2 * t4)};
    if (bad) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if ((in[e >> 1] & (1u << (8 * j + (e & 1)))) && (s_bad[0][key0 + 8 * j + (e & 1)] | s_bad[2][row[e >> 1]]))
            s[j][e] = dot_row(q + row_ptr(row[e >> 1]) * D, a.scale, kbase + (size_t)ki->tok[buf][key0 + 8 * j + (e & 1)] * D);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (!(in[e >> 1] & (1u << (8 * j + (e & 1))))) s[j][e] = -INFINITY;
        mx[e >> 1] = fmaxf(mx[e >> 1], s[j][e]);
      }
    float alpha[2], m_new[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
      m_new[i] = fmaxf(m[i], mx[i]);
      alpha[i] = expf(m[i] - (m_new[i] == -INFINITY ? 0.f : m_new[i]));        // m = -inf: 0
      m[i] = m_new[i];
      l[i] *= alpha[i];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x = expf(s[j][e] - m_new[e >> 1]);        // for all: a select below, not a branch around it
        const float p = in[e >> 1] & (1u << (8 * j + (e & 1))) ? x : kMasked;
        l[e >> 1] += p;
        s[j][e] = p;
      }
    if (repeats) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int n = attended(s[j][e]) ? times_listed(a, bh, (row0 + row[e >> 1]) / G, ki->tok[buf][key0 + 8 * j + (e & 1)]) : 1;
          if (n > 1) {
            l[e >> 1] += s[j][e] * (float)(n - 1);
            s[j][e] *= (float)n;
          }
        }
    }
    {
      uint32_t p[2][3][4];
#pragma unroll
      for (int kk = 0; kk < 2; ++kk)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          split2(s[2 * kk + (e >> 1)][2 * (e & 1)], s[2 * kk + (e >> 1)][2 * (e & 1) + 1], p[kk][0][e], p[kk][1][e], p[kk][2][e]);
#pragma unroll
      for (int dh = 0; dh < 2; ++dh) {
        float pv[4][4];
        product<2>(pv, [&](int kk, uint32_t (*x)[4]) {
#pragma unroll
                     for (int t = 0; t < 3; ++t)
#pragma unroll
                       for (int e = 0; e < 4; ++e) x[t][e] = p[kk][t][e];
                   },
                   [&](int t, int kk, int j, uint32_t* y) { ldsm4t(sV + t * kTermBytes + at_a(lane, 32 * half + 16 * kk, 4 * dh + j), y); });
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[4 * dh + j][e] = fmaf(o[4 * dh + j][e], alpha[e >> 1], pv[j][e]);
      }
    }
    if (bad) {
#pragma unroll
      for (int k4 = 0; k4 < 8; ++k4)                                 // columns k4 / 2 of eight, and their first or second key
#pragma unroll 1
        for (int t = 0; t < 4; ++t) {
          const int src = (lane & ~3) | t, k = 32 * half + 8 * (k4 >> 1) + 2 * t + (k4 & 1);
          const float p[2] = {__shfl_sync(0xffffffffu, s[k4 >> 1][k4 & 1], src), __shfl_sync(0xffffffffu, s[k4 >> 1][2 + (k4 & 1)], src)};
          const uint32_t chunks = s_bad[1][k];
          if (!chunks) continue;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (!((chunks >> j) & 1u)) continue;
            const float2 v = __ldg(reinterpret_cast<const float2*>(vbase + (size_t)ki->tok[buf][k] * D + 8 * j + 2 * t4));
            if (attended(p[0])) { o[j][0] = fmaf(p[0], v.x, o[j][0]); o[j][1] = fmaf(p[0], v.y, o[j][1]); }
            if (attended(p[1])) { o[j][2] = fmaf(p[1], v.x, o[j][2]); o[j][3] = fmaf(p[1], v.y, o[j][3]); }
          }
        }
      __syncthreads();                    // the notes have been read: clean for the next tile
      if (tid < 2 * kK) s_bad[tid / kK][tid % kK] = 0u;
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
  }
  // both warps of 16 rows, of every CTA of the cluster, leave what their keys gave (O over K and V; m and l over Q); the rows are dealt
  // out for the sum
  float* sO = reinterpret_cast<float*>(smem + kTileBytes);       // [half][row][kLd]
  float* sM = reinterpret_cast<float*>(smem);                    // [half][m, l][row]
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      *reinterpret_cast<float2*>(sO + (half * kR + row[i]) * kLd + 8 * j + 2 * t4) = make_float2(o[j][2 * i], o[j][2 * i + 1]);
    if (t4 == 0) { sM[half * 2 * kR + row[i]] = m[i]; sM[half * 2 * kR + kR + row[i]] = l[i]; }
  }
  if (csize > 1) cluster_sync(); else __syncthreads();
  auto get = [&](const float* p, int k) -> float { return csize > 1 ? ld_peer_f32(p, k >> 1) : *p; };
  for (int i = tid; i < kR / csize * (D / 4); i += kThreads) {
    const int r = (i / (D / 4)) * csize + rank, c = (i % (D / 4)) * 4;
    if (row0 + r >= n_rows) continue;
    float mm = -INFINITY, ll = 0.f;
    for (int k = 0; k < 2 * csize; ++k) mm = fmaxf(mm, get(sM + (k & 1) * 2 * kR + r, k));
    const float ms = mm == -INFINITY ? 0.f : mm;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < 2 * csize; ++k) {
      const float w = expf(get(sM + (k & 1) * 2 * kR + r, k) - ms);
      const float* at = sO + ((k & 1) * kR + r) * kLd + c;
      const float4 v = csize > 1 ? ld_peer_f32x4(at, k >> 1) : *reinterpret_cast<const float4*>(at);
      ll = fmaf(w, get(sM + (k & 1) * 2 * kR + kR + r, k), ll);
      acc.x = fmaf(w, v.x, acc.x); acc.y = fmaf(w, v.y, acc.y); acc.z = fmaf(w, v.z, acc.z); acc.w = fmaf(w, v.w, acc.w);
    }
    const size_t at = row_ptr(r);
    const float inv = ll > 0.f ? 1.f / ll : 0.f;
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.o) + at * D + c) = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
    if (c == 0 && a.lse) a.lse[at] = ll > 0.f ? mm + logf(ll) : kLseEmpty;
  }
  if (csize > 1) cluster_sync();          // nobody leaves while its memory is read
}

// 16 keys x 32 columns (from c0 on) of a product's result added to the keys' gradients: neighbouring lanes trade halves of their two
// rows for vectors of four
__device__ __forceinline__ void add_rows(float* base, const float (*x)[4], int tok0, int tok1, int c0, int t4) {
  const bool odd = t4 & 1;
  const int tok = odd ? tok1 : tok0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float r0 = __shfl_xor_sync(0xffffffffu, odd ? x[j][0] : x[j][2], 1);
    const float r1 = __shfl_xor_sync(0xffffffffu, odd ? x[j][1] : x[j][3], 1);
    const float4 v = odd ? make_float4(r0, r1, x[j][2], x[j][3]) : make_float4(x[j][0], x[j][1], r0, r1);
    if (tok >= 0)
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(base + (size_t)tok * D + c0 + 8 * j + 4 * (t4 >> 1)), "f"(v.x),
                   "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
  }
}

__global__ void __launch_bounds__(kThreads, 2)
f32_tile_bwd_kernel(const AttnArgs a, const int csize) {
  extern __shared__ float4 sm4[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(sm4);
  const uint32_t sQ = smem_addr(smem), sDO = sQ + kTileBytes, sK = sDO + kTileBytes, sV = sK + kTileBytes;
  KeyInfo* ki = reinterpret_cast<KeyInfo*>(smem + kBwdBytes);
  const SelList sl = sel_list(a, ki + 1);
  __shared__ __align__(16) float s_lse[kR], s_delta[kR], s_scale[kR];
  __shared__ size_t s_row[kR];
  __shared__ __align__(16) uint32_t s_att[2][2][kR], s_bad[4][kR];                 // (K, V, Q, dO)
  const int tid = threadIdx.x, warp = (tid >> 5) & 3, half = tid >> 7, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int G = a.Hq / a.Hkv, n_rows = a.T * G, tiles = (n_rows + kR - 1) / kR;
  const int rank = (int)blockIdx.x & (csize - 1), work = (int)blockIdx.x / csize;
  const int units = a.B * a.Hkv, bh = work % units, b = bh / a.Hkv, hkv = bh % a.Hkv;
  const int row0 = (tiles - 1 - work / units) * kR;
  const int t_first = row0 / G, t_last = (min(row0 + kR, n_rows) - 1) / G;
  auto row_ptr = [&](int r) -> size_t {
    const int f = row0 + r;
    return ((size_t)b * a.Hq + hkv * G + f % G) * a.T + f / G;
  };
  const float* q = reinterpret_cast<const float*>(a.q);
  const float* d_o = reinterpret_cast<const float*>(a.d_o);
  for (int i = tid; i < 4 * kR; i += kThreads) s_bad[i / kR][i % kR] = 0u;
  __syncthreads();
  const TileKeys tk = tile_keys<kThreads>(a, bh, t_first, t_last, sl);
  const bool repeats = a.kind == 2 && *sl.repeats;
  const int n_kt = (tk.n + kK - 1) / kK;
  const size_t kvoff = (size_t)bh * a.Lk * D;
  const float* kbase = reinterpret_cast<const float*>(a.k) + kvoff;
  const float* vbase = reinterpret_cast<const float*>(a.v) + kvoff;
  float* dkb = a.dk_acc + kvoff;
  float* dvb = a.dv_acc + kvoff;
  const RowKeys rk(a, row0 + (tid & (kR - 1)), n_rows, G, t_first);
  if (rank < n_kt) fill_tile(a, tk, sl, ki, s_att, rk, 0, rank);
  // Q (scaled), dO (times the gate of a gated branch), lse and delta; four threads per row
  bool rows_bad = false;
  {
    const int r = tid >> 2, part = tid & 3;
    const bool in = row0 + r < n_rows;
    const size_t row = in ? row_ptr(r) : 0;
    const float rs = in && a.row_scale ? a.row_scale[row] : 1.f;
    float dot = 0.f;
#pragma unroll 1
    for (int c = part; c < D / 8; c += 4) {
      float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, y[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (in) {
        load8(q + row * D + 8 * c, x);
        load8(d_o + row * D + 8 * c, y);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) { x[e] *= a.scale; y[e] *= rs; }
      if (in && !a.row_dot) {
        float o[8];
        load8(reinterpret_cast<const float*>(a.o) + row * D + 8 * c, o);
#pragma unroll
        for (int e = 0; e < 8; ++e) dot = fmaf(y[e], o[e], dot);
      }
      rows_bad |= put_terms(sQ, s_bad[2], r, c, x);
      rows_bad |= put_terms(sDO, s_bad[3], r, c, y);
    }
    dot += __shfl_xor_sync(0xffffffffu, dot, 1);
    dot += __shfl_xor_sync(0xffffffffu, dot, 2);
    if (part == 0) {
      const float lse = in ? a.lse[row] : 0.f, delta = in ? (a.row_dot ? rs * a.row_dot[row] : dot) : 0.f;
      s_lse[r] = lse; s_delta[r] = delta; s_scale[r] = rs; s_row[r] = row;
    }
  }
  float dq[4][4];                         // rows 16 warp ..., columns 32 half ...
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) dq[j][e] = 0.f;
  int buf = 0;
  for (int kt = rank; kt < n_kt; kt += csize, buf ^= 1) {
    __syncthreads();                      // the last tile is done with; this one's keys are known
    bool bad = load_terms(sK, s_bad[0], kbase, ki->tok[buf]);
    bad |= load_terms(sV, s_bad[1], vbase, ki->tok[buf]);
    bad = __syncthreads_or(bad || rows_bad);
    if (kt + csize < n_kt) fill_tile(a, tk, sl, ki, s_att, rk, buf ^ 1, kt + csize);
    // S and dP, keys x rows: this lane's keys are key0 and 8 on, its rows r0 + 8 j and the next
    const int key0 = 16 * warp + g, r0 = 32 * half + 2 * t4;
    const int tok[2] = {ki->tok[buf][key0], ki->tok[buf][key0 + 8]};
    float s[4][4], ds[4][4];
    product<D / 16>(s, [&](int kk, uint32_t (*x)[4]) { ldsm_terms(sK + at_a(lane, 16 * warp, 2 * kk), x); },
                    [&](int t, int kk, int j, uint32_t* y) { ldsm4(sQ + t * kTermBytes + at_b(lane, 32 * half + 8 * j, 2 * kk), y); });
    product<D / 16>(ds, [&](int kk, uint32_t (*x)[4]) { ldsm_terms(sV + at_a(lane, 16 * warp, 2 * kk), x); },
                    [&](int t, int kk, int j, uint32_t* y) { ldsm4(sDO + t * kTermBytes + at_b(lane, 32 * half + 8 * j, 2 * kk), y); });
    const uint32_t key_bit = 1u << (key0 & 31);
    if (bad) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int r = r0 + 8 * j + (e & 1), k = key0 + 8 * (e >> 1);
          if (!(s_att[buf][warp >> 1][r] & (key_bit << (8 * (e >> 1))))) continue;
          if (s_bad[0][k] | s_bad[2][r]) s[j][e] = dot_row(q + s_row[r] * D, a.scale, kbase + (size_t)tok[e >> 1] * D);
          if (s_bad[1][k] | s_bad[3][r]) ds[j][e] = dot_row(d_o + s_row[r] * D, s_scale[r], vbase + (size_t)tok[e >> 1] * D);
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 lse = *reinterpret_cast<const float2*>(s_lse + r0 + 8 * j), delta = *reinterpret_cast<const float2*>(s_delta + r0 + 8 * j);
      const uint2 att = *reinterpret_cast<const uint2*>(&s_att[buf][warp >> 1][r0 + 8 * j]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool in = ((e & 1) ? att.y : att.x) & (key_bit << (8 * (e >> 1)));
        const float x = expf(s[j][e] - ((e & 1) ? lse.y : lse.x));          // for all: a select below, not a branch around it
        const float p = in ? x : kMasked;
        ds[j][e] = in ? p * (ds[j][e] - ((e & 1) ? delta.y : delta.x)) : 0.f;
        s[j][e] = p;
      }
    }
    if (repeats) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int n = attended(s[j][e]) ? times_listed(a, bh, (row0 + r0 + 8 * j + (e & 1)) / G, tok[e >> 1]) : 1;
          if (n > 1) { s[j][e] *= (float)n; ds[j][e] *= (float)n; }
        }
    }
    __syncthreads();                      // V has been read: P, then dS, take its place, [key][row]
    auto put = [&](const float (*x)[4]) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t t[3];
          split2(x[j][2 * i], x[j][2 * i + 1], t[0], t[1], t[2]);
          const uint32_t at = sV + (key0 + 8 * i) * 128 + (((4 * half + j) ^ g) << 4) + 4 * t4;
#pragma unroll
          for (int m = 0; m < 3; ++m) asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + m * kTermBytes), "r"(t[m]) : "memory");
        }
    };
    const uint8_t* w = smem + 3 * kTileBytes;
    // the columns of rows that are zeros in their tile (noted in s_bad[which]), for what attends them
    auto add_bad_rows = [&](float (*acc)[4], int which, const float* x) {
#pragma unroll 1
      for (int r = 0; r < kR; ++r) {
        const uint32_t chunks = s_bad[which][r] >> (4 * half), att = s_att[buf][warp >> 1][r] >> (key0 & 31);
        if (!(chunks & 15u)) continue;
        const float f0 = of_terms(w, key0, r), f1 = of_terms(w, key0 + 8, r), rs = which == 2 ? a.scale : s_scale[r];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (!((chunks >> j) & 1u)) continue;
          const float2 y = __ldg(reinterpret_cast<const float2*>(x + s_row[r] * D + 32 * half + 8 * j + 2 * t4));
          if (att & 1u) { acc[j][0] = fmaf(f0, y.x * rs, acc[j][0]); acc[j][1] = fmaf(f0, y.y * rs, acc[j][1]); }
          if (att & 256u) { acc[j][2] = fmaf(f1, y.x * rs, acc[j][2]); acc[j][3] = fmaf(f1, y.y * rs, acc[j][3]); }
        }
      }
    };
    auto keys_a = [&](int kk, uint32_t (*x)[4]) { ldsm_terms(sV + at_a(lane, 16 * warp, 2 * kk), x); };
    float acc[4][4];
    put(s);
    __syncthreads();
    product<kR / 16>(acc, keys_a, [&](int t, int kk, int j, uint32_t* y) { ldsm4t(sDO + t * kTermBytes + at_a(lane, 16 * kk, 4 * half + j), y); });
    if (bad) add_bad_rows(acc, 3, d_o);
    add_rows(dvb, acc, tok[0], tok[1], 32 * half, t4);               // dV += P^T dO
    __syncthreads();
    put(ds);
    __syncthreads();
    product<kR / 16>(acc, keys_a, [&](int t, int kk, int j, uint32_t* y) { ldsm4t(sQ + t * kTermBytes + at_a(lane, 16 * kk, 4 * half + j), y); });
    if (bad) add_bad_rows(acc, 2, q);
    add_rows(dkb, acc, tok[0], tok[1], 32 * half, t4);               // dK += dS^T Q (Q carries the scale)
    product<kK / 16>(acc, [&](int kk, uint32_t (*x)[4]) {
#pragma unroll
                       for (int t = 0; t < 3; ++t) ldsm4t(sV + t * kTermBytes + at_b(lane, 16 * kk, 2 * warp), x[t]);
                     },
                     [&](int t, int kk, int j, uint32_t* y) { ldsm4t(sK + t * kTermBytes + at_a(lane, 16 * kk, 4 * half + j), y); });
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) dq[j][e] += acc[j][e];             // dQ += dS K
    if (bad) {
      const int r = 16 * warp + g;
#pragma unroll 1
      for (int k = 0; k < kK; ++k) {
        const uint32_t chunks = s_bad[0][k] >> (4 * half);
        if (!(chunks & 15u)) continue;
        const float f0 = of_terms(w, k, r), f1 = of_terms(w, k, r + 8);
        const uint32_t a0 = s_att[buf][k >> 5][r] >> (k & 31), a1 = s_att[buf][k >> 5][r + 8] >> (k & 31);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (!((chunks >> j) & 1u)) continue;
          const float2 y = __ldg(reinterpret_cast<const float2*>(kbase + (size_t)ki->tok[buf][k] * D + 32 * half + 8 * j + 2 * t4));
          if (a0 & 1u) { dq[j][0] = fmaf(f0, y.x, dq[j][0]); dq[j][1] = fmaf(f0, y.y, dq[j][1]); }
          if (a1 & 1u) { dq[j][2] = fmaf(f1, y.x, dq[j][2]); dq[j][3] = fmaf(f1, y.y, dq[j][3]); }
        }
      }
      __syncthreads();                    // the notes have been read: clean for the next tile
      if (tid < 2 * kK) s_bad[tid / kK][tid % kK] = 0u;
    }
  }
  if (csize == 1) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = 16 * warp + g + 8 * i;
      if (row0 + r >= n_rows) continue;
      float* dst = reinterpret_cast<float*>(a.dq) + row_ptr(r) * D;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float2*>(dst + 32 * half + 8 * j + 2 * t4) = make_float2(dq[j][2 * i] * a.scale, dq[j][2 * i + 1] * a.scale);
    }
    return;
  }
  // dQ of the cluster's CTAs, over their K tiles, in rank order
  float* sD = reinterpret_cast<float*>(smem + 2 * kTileBytes);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<float2*>(sD + (16 * warp + g + 8 * i) * kLd + 32 * half + 8 * j + 2 * t4) = make_float2(dq[j][2 * i], dq[j][2 * i + 1]);
  cluster_sync();
  for (int i = tid; i < kR / csize * (D / 4); i += kThreads) {
    const int r = (i / (D / 4)) * csize + rank, c = (i % (D / 4)) * 4;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < csize; ++k) {
      const float4 v = ld_peer_f32x4(sD + r * kLd + c, k);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    if (row0 + r < n_rows)
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.dq) + row_ptr(r) * D + c) =
          make_float4(acc.x * a.scale, acc.y * a.scale, acc.z * a.scale, acc.w * a.scale);
  }
  cluster_sync();                         // nobody leaves while its memory is read
}

}  // namespace

// CTAs that share a row tile, each taking every csize-th key tile.  In row tiles per SM (1 | 2 | 4 CTAs, us): selection at 0.43 forward
// 49 | 34 | 33, backward 90 | 56 | 48; at 0.85 81 | 56 | 53 and 151 | 104 | 92; at 0.89 59 | 43 | 48 and 108 | 78 | 79; at 1.7 181 | 113 | 144 and
// 355 | 242 | 256; at 3.5 202 | 217 | 276 and 438 | 429 | 485; at 5.2 309 | 321 | 402 and 606 | 626 | 715.  Window, which has nine key
// tiles a row tile, at 0.43 44 | 29 | 27 and 81 | 51 | 45; at 0.85 48 | 39 | 46 and 92 | 79 | 77; at 1.7 66 | 71 | 90 and 142 | 142 | 151.
static int f32_cluster_size(const AttnArgs& a) {
  const long long tiles = n_tiles(a), sms = sm_count();
  const long long n_kt = ((a.kind == 0 ? (long long)a.window + kR / (a.Hq / a.Hkv) : a.Lk) + kK - 1) / kK;    // (any window)
  int csize;
  if (a.kind == 2) csize = 8 * tiles <= 7 * sms ? 4 : tiles <= 3 * sms ? 2 : 1;
  else csize = 2 * tiles <= sms ? 4 : 3 * tiles <= 4 * sms ? 2 : 1;
  while (csize > 1 && n_kt < 2 * csize) csize >>= 1;
  return csize;
}

int f32_tile_launch(const AttnArgs& a, bool bwd, cudaStream_t st) {
  const int csize = f32_cluster_size(a);
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)csize;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)n_tiles(a) * csize);   // in x, which takes any number of units
  cfg.blockDim = dim3(kThreads);
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = csize > 1 ? 1 : 0;
  const auto kernel = bwd ? f32_tile_bwd_kernel : f32_tile_fwd_kernel;
  cfg.dynamicSmemBytes = (bwd ? kBwdBytes : kFwdBytes) + extra_smem(a);
  NSA_CUDA_OK(func_smem((const void*)kernel, cfg.dynamicSmemBytes));
  KernelScope ks(branch_name(bwd ? kBwdNames : kFwdNames, a.kind), st);
  NSA_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, a, csize));
  NSA_LAUNCH_OK("f32_tile kernel");
  return NSA_OK;
}

}  // namespace nsa
