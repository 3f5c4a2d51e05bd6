// Bookkeeping shared by the kernels on tiles of 64 rows x 64 keys (simt_tile.cu, f32_tile.cu): which keys a row tile
// attends, tile by tile, and what marks a key that a row does not.
#pragma once

#include "common.cuh"

namespace nsa {
int f32_tile_launch(const AttnArgs& a, bool bwd, cudaStream_t st);   // f32_tile.cu
namespace {

constexpr int kR = 64;           // rows per tile
constexpr int kK = 64;           // keys per tile
constexpr int kMaxBlocks = 1024; // blocks a selection tile can tell apart

// What a tile's rows attend: keys [first, first + n) of the unit, or the union of listed blocks.
struct TileKeys {
  int first, n;            // window / compression: first key and their number; selection: 0, keys of the union
};

struct SelList {           // selection only, in shared memory: as many blocks as the sequence has
  unsigned long long* mask;   // queries of the tile that list a block
  int* n_list;
  int* repeats;               // not 0: some query lists a block more than once
  uint16_t* list;             // the listed blocks, ascending
};
__host__ __device__ __forceinline__ int sel_blocks(const AttnArgs& a) { return (a.T + a.block_size - 1) / a.block_size; }
__device__ __forceinline__ SelList sel_list(const AttnArgs& a, void* at) {
  SelList s;
  s.mask = (unsigned long long*)at;
  s.n_list = (int*)(s.mask + (a.kind == 2 ? sel_blocks(a) : 0));
  s.repeats = s.n_list + 1;
  s.list = (uint16_t*)(s.n_list + 2);
  return s;
}

// shared memory of one tile's key bookkeeping, double buffered: the next tile is fetched ahead
struct KeyInfo {
  int tok[2][kK];                        // token (or summary) of a key, -1: none
  unsigned long long mask[2][kK];        // selection: queries that list its block
};

template <int kThreads>
__device__ __forceinline__ TileKeys tile_keys(const AttnArgs& a, int bh, int t_first, int t_last, const SelList& sl) {
  TileKeys k;
  k.first = 0; k.n = 0;
  if (a.kind == 0) {
    k.first = max(0, t_first - a.window + 1);
    k.n = max(0, min(t_last, a.Lk - 1) - k.first + 1);
  } else if (a.kind == 1) {
    k.n = cmp_visible(t_last, a.block_size, a.window, a.Lk);   // compression: window holds the stride
  } else {
    const int n_blk = (t_last + a.block_size) / a.block_size;   // blocks that start at or before t_last
    for (int i = threadIdx.x; i < n_blk; i += kThreads) sl.mask[i] = 0ull;
    if (threadIdx.x == 0) *sl.repeats = 0;
    __syncthreads();
    const int32_t* idx = a.block_idx + ((size_t)bh * a.T + t_first) * a.S;
    const int n_e = (t_last - t_first + 1) * a.S;
    for (int e = threadIdx.x; e < n_e; e += kThreads) {
      const int ql = e / a.S;
      const int blk = __ldg(idx + e);
      if (blk >= 0 && (long long)blk * a.block_size <= t_first + ql &&
          (atomicOr(&sl.mask[blk], 1ull << ql) >> ql & 1ull))
        *sl.repeats = 1;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      int n = 0;
      for (int b0 = 0; b0 < n_blk; b0 += 32) {
        const int b = b0 + threadIdx.x;
        const bool on = b < n_blk && sl.mask[b] != 0ull;
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (on) sl.list[n + __popc(m & ((1u << threadIdx.x) - 1u))] = (uint16_t)b;
        n += __popc(m);
      }
      if (threadIdx.x == 0) *sl.n_list = n;
    }
    __syncthreads();
    k.n = *sl.n_list * a.block_size;
  }
  return k;
}

// How often query t lists the block of token tok.  A block listed twice counts twice, as it does in the
// row kernels, which go through the slots one by one.
__device__ __forceinline__ int times_listed(const AttnArgs& a, int bh, int t, int tok) {
  const int32_t* slot = a.block_idx + ((size_t)bh * a.T + t) * a.S;
  const int blk = tok / a.block_size;
  int n = 0;
#pragma unroll 1
  for (int s = 0; s < a.S; ++s) n += __ldg(slot + s) == blk;
  return n;
}

// token and, where asked for, membership of key tile i's keys (threads 0..63)
template <bool kMask>
__device__ __forceinline__ void fill_keys(const AttnArgs& a, const TileKeys& tk, const SelList& sl, KeyInfo* ki, int buf, int i) {
  if (threadIdx.x >= kK) return;
  const int k = i * kK + threadIdx.x;
  int tok = -1;
  unsigned long long m = 0ull;
  if (k < tk.n) {
    if (a.kind == 2) {
      const int b = sl.list[k / a.block_size];
      tok = b * a.block_size + k % a.block_size;
      if (kMask) m = sl.mask[b];
      if (tok >= a.T) tok = -1;
    } else {
      tok = tk.first + k;
    }
  }
  ki->tok[buf][threadIdx.x] = tok;
  if (kMask) ki->mask[buf][threadIdx.x] = m;
}

// keys [lo, hi] a row of query t may see by position
__device__ __forceinline__ void row_range(const AttnArgs& a, int t, int& lo, int& hi) {
  lo = 0;
  hi = min(t, a.Lk - 1);
  if (a.kind == 0) lo = max(0, t - a.window + 1);
  else if (a.kind == 1) hi = cmp_visible(t, a.block_size, a.window, a.Lk) - 1;
}

// What stands for a key that a row does not attend in the tile of P: the sign tells it from a probability of
// zero.  As a factor it is a zero, as long as the other factor is finite; a tile that holds a value
// that is not goes through loops that leave these keys out, so that such a value stays with the rows
// (and keys) that it belongs to.
constexpr float kMasked = -0.f;
__device__ __forceinline__ bool attended(float p) { return __float_as_uint(p) != 0x80000000u; }

inline long long n_tiles(const AttnArgs& a) {
  return ((long long)a.T * (a.Hq / a.Hkv) + kR - 1) / kR * a.B * a.Hkv;
}

inline size_t extra_smem(const AttnArgs& a) { return sizeof(KeyInfo) + 16 + (a.kind == 2 ? (size_t)sel_blocks(a) * 10 : 0); }

}  // namespace
}  // namespace nsa
