// Builds the index structures of sel_plan.cuh in three launches, count, scan and fill, or in one where the sequence
// is short.  A CTA of the first and the last takes a chunk of consecutive queries of one unit and
// marks its list entries in a bitmap [key tile][query] in shared memory, from which ranks are
// population counts; nothing but the counts and the results touches global memory.  At 16 units of
// 32768 queries x 16 slots: 0.17 ms, against 0.30 ms and eight launches with the bitmap in global
// memory (bound by the scattered 4-byte stores of the pairs); at 4 units of 1024 queries 16 us,
// bound by latency.
#include "cluster.cuh"
#include "sel_plan.cuh"

namespace nsa {
namespace {

constexpr int kKeysPerTile = 64;
constexpr int kThreads = 256;

// key tile of a list entry of query t, -1 when the entry is empty or lies after t
__device__ __forceinline__ int tile_of(int blk, int t, int block_size) {
  if (blk < 0 || (long long)blk * block_size > t) return -1;
  return (blk * block_size) / kKeysPerTile;
}

// Bitmap words are laid out [word][tile]: the entries a warp marks together name different tiles of
// one or two queries, so they fall into different banks.
__device__ __forceinline__ void mark_chunk(const int32_t* idx, uint32_t* bm, int t0, int n_q, int S,
                                           int block_size, int n_kt, int cw) {
  for (int i = threadIdx.x; i < n_kt * cw; i += blockDim.x) bm[i] = 0u;
  __syncthreads();
#pragma unroll 4
  for (int e = threadIdx.x; e < n_q * S; e += blockDim.x) {
    const int ql = e / S;
    const int j = tile_of(ld_plain(idx + e), t0 + ql, block_size);
    if (j >= 0) atomicOr(&bm[(ql >> 5) * n_kt + j], 1u << (ql & 31));
  }
  __syncthreads();
}

// counts[unit][chunk][tile] and, per CTA, the distinct (query tile, key tile) pairs
__global__ void __launch_bounds__(kThreads)
plan_count_kernel(const int32_t* block_idx, int32_t* __restrict__ counts, int32_t* __restrict__ unions,
                  SelPlanHeader* __restrict__ hdr, int T, int S, int block_size, int n_kt, int cw, int n_chunks,
                  int nq_union) {
  extern __shared__ uint32_t bm[];
  chain_wait();
  chain_go();
  const int chunk = blockIdx.x, unit = blockIdx.y;
  if (chunk == 0 && unit == 0 && threadIdx.x == 0) { hdr->union_tiles = 0ull; hdr->pairs = 0ull; hdr->repeats = 0ull; }
  const int t0 = chunk * cw * 32, n_q = min(T - t0, cw * 32);
  mark_chunk(block_idx + ((size_t)unit * T + t0) * S, bm, t0, n_q, S, block_size, n_kt, cw);
  int uni = 0;
  const int per = nq_union < 32 ? nq_union : 32;        // a query tile is a part of a word or whole words
  const int tw = nq_union > 32 ? nq_union / 32 : 1;
  const uint32_t mask = per == 32 ? 0xffffffffu : (1u << per) - 1u;
  for (int j = threadIdx.x; j < n_kt; j += kThreads) {
    int c = 0;
    uint32_t run = 0u;
    for (int w = 0; w < cw; ++w) {
      const uint32_t b = bm[w * n_kt + j];
      c += __popc(b);
      if (per < 32) {
        for (int k = 0; k < 32; k += per) uni += ((b >> k) & mask) != 0u;
      } else {
        run |= b;
        if ((w + 1) % tw == 0 || w + 1 == cw) { uni += run != 0u; run = 0u; }
      }
    }
    counts[((size_t)unit * n_chunks + chunk) * n_kt + j] = c;
  }
  __shared__ int s_uni;
  if (threadIdx.x == 0) s_uni = 0;
  __syncthreads();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) uni += __shfl_xor_sync(0xffffffffu, uni, o);
  if ((threadIdx.x & 31) == 0 && uni) atomicAdd(&s_uni, uni);
  __syncthreads();
  if (threadIdx.x == 0) unions[unit * n_chunks + chunk] = s_uni;
}

// exclusive scan of v over the CTA's NT threads; *total gets the sum
template <int NT>
__device__ __forceinline__ int block_scan(int v, int* warp_sums, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = lane < NT / 32 ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += u;
    }
    warp_sums[lane] = w;
  }
  __syncthreads();
  const int before = warp ? warp_sums[warp - 1] : 0;
  *total = warp_sums[NT / 32 - 1];
  __syncthreads();
  return before + incl - v;
}

// One CTA per unit: offsets of the key tiles, the start of every (chunk, tile) run in place of its
// count, and the work items in (tile, chunk) order.  Up to NT tiles a pass; with fewer tiles the
// chunks are dealt out over groups of threads, so the column sums are not one long chain of loads.  256 threads of
// at most 48 registers find room beside two CTAs of the window kernel on an SM; 1024 wait until they are done.
template <int NT>
__global__ void __launch_bounds__(NT, NT == 256 ? 5 : 1)
plan_scan_kernel(int32_t* __restrict__ counts, const int32_t* unions, SelPlan p, int T, int S,
                 int n_kt, int n_chunks, int nq) {
  constexpr int kBatch = NT == 256 ? 8 : 16;  // loads in flight per thread
  __shared__ int warp_sums[32];
  __shared__ int part_sum[NT];
  chain_wait();
  chain_go();
  const int unit = blockIdx.x, tid = threadIdx.x;
  int32_t* cnt = counts + (size_t)unit * n_chunks * n_kt;
  int pair_carry = unit * T * S, item_carry = 0;
  int32_t* off = p.offsets + (size_t)unit * (n_kt + 1);
  int4* items = p.items + (size_t)unit * p.max_items;
  int width = 32;                             // tiles per pass, a power of two
  while (width < NT && width < n_kt) width <<= 1;
  const int parts = NT / width, part = tid / width;
  const int per = (n_chunks + parts - 1) / parts;
  const int c0 = min(n_chunks, part * per), c1 = min(n_chunks, c0 + per);
  for (int j0 = 0; j0 < n_kt; j0 += width) {
    const int j = j0 + (tid & (width - 1));
    int n = 0;
    if (j < n_kt) {
#pragma unroll 16
      for (int c = c0; c < c1; ++c) n += cnt[(size_t)c * n_kt + j];
    }
    part_sum[tid] = n;
    __syncthreads();
    int before = 0, all = 0;                  // pairs of tile j in earlier groups of chunks / in all
    for (int q = 0; q < parts; ++q) {
      const int v = part_sum[q * width + (tid & (width - 1))];
      if (q < part) before += v;
      all += v;
    }
    const bool first_part = part == 0 && j < n_kt;
    const int n_rt = (all + nq - 1) / nq;
    // at least one item, so that a tile nobody lists still gets its zero gradients
    const int n_it = first_part ? max(1, (n_rt + kSelChunkTiles - 1) / kSelChunkTiles) : 0;
    int total, total_it;
    const int start = pair_carry + block_scan<NT>(first_part ? all : 0, warp_sums, &total);
    const int first = item_carry + block_scan<NT>(n_it, warp_sums, &total_it);
    if (first_part) {
      off[j] = start;
      for (int k = 0; k < n_it && first + k < p.max_items; ++k)
        items[first + k] = make_int4(unit, j, k * kSelChunkTiles, n_it);
      part_sum[tid] = start;
    }
    __syncthreads();
    if (j < n_kt) {
      int run = part_sum[tid & (width - 1)] + before;
      for (int c = c0; c < c1; c += kBatch) {
        int v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) v[k] = c + k < c1 ? cnt[(size_t)(c + k) * n_kt + j] : 0;
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          if (c + k < c1) cnt[(size_t)(c + k) * n_kt + j] = run;
          run += v[k];
        }
      }
    }
    __syncthreads();
    pair_carry += total;
    item_carry += total_it;
  }
  int uni = 0;
  for (int c = tid; c < n_chunks; c += NT) uni += unions[unit * n_chunks + c];
  int uni_total;
  block_scan<NT>(uni, warp_sums, &uni_total);
  if (tid == 0) {
    off[n_kt] = pair_carry;
    p.n_items[unit] = min(item_carry, p.max_items);
    atomicAdd(&p.hdr->union_tiles, (unsigned long long)uni_total);
    atomicAdd(&p.hdr->pairs, (unsigned long long)(pair_carry - unit * T * S));
  }
}

// Every entry's pair: the start of its (chunk, tile) run plus the rank of its query in the bitmap.
// kMatch: a query's S entries sit in one warp (S divides 32), so the entries of one query that
// name the same tile find one another by a warp match instead of reading the list again.
template <bool kMatch>
__device__ __forceinline__ void fill_chunk(const int32_t* idx, const uint32_t* bm, const uint16_t* before,
                                           const int32_t* st, int32_t* __restrict__ pairs, int32_t* __restrict__ pos,
                                           SelPlanHeader* __restrict__ hdr, int t0, int n_q, int S, int block_size, int n_kt) {
  const uint32_t one = (1u << (block_size >> 4)) - 1u;              // column groups of one block
  const int n_e = n_q * S;
  for (int e0 = 0; e0 < n_e; e0 += blockDim.x) {
    const int e = e0 + threadIdx.x;
    const bool in = e < n_e;
    const int ql = in ? e / S : 0, t = t0 + ql, slot = e - ql * S;
    const int blk = in ? ld_plain(idx + e) : -1;
    const int j = tile_of(blk, t, block_size);
    uint32_t groups = j < 0 ? 0u : one << ((blk * block_size - j * kKeysPerTile) >> 4);
    bool dup = false;
    if (kMatch) {
      const uint32_t peers = __match_any_sync(0xffffffffu, j < 0 ? -1 - (int)threadIdx.x : (ql << 16) | j);
      dup = (peers & ((1u << (threadIdx.x & 31)) - 1u)) != 0u;
      if (block_size < kKeysPerTile) {
        groups = __reduce_or_sync(peers, groups);
        if (j >= 0 && __popc(peers) * __popc(one) != __popc(groups)) hdr->repeats = 1ull;
      }
    } else if (j >= 0) {
      const int32_t* row = idx + ql * S;
      for (int s = 0; s < S; ++s) {
        const int b2 = ld_plain(row + s);
        if (tile_of(b2, t, block_size) != j) continue;
        dup |= s < slot;
        if (block_size < kKeysPerTile && s < slot && b2 == blk) hdr->repeats = 1ull;
        groups |= one << ((b2 * block_size - j * kKeysPerTile) >> 4);
      }
    }
    int r = -1;
    if (j >= 0 && !dup) {
      const int at = (ql >> 5) * n_kt + j;
      r = st[j] + before[at] + __popc(bm[at] & ((1u << (ql & 31)) - 1u));
      pairs[r] = (int32_t)((uint32_t)t | (groups << kPairPosBits));
    }
    if (in) pos[e] = r;
  }
}

template <bool kMatch>
__global__ void __launch_bounds__(kThreads)
plan_fill_kernel(const int32_t* block_idx, const int32_t* starts,
                 int32_t* __restrict__ pairs, int32_t* __restrict__ pair_of_slot, SelPlanHeader* __restrict__ hdr, int T, int S,
                 int block_size, int n_kt, int cw, int n_chunks) {
  extern __shared__ uint32_t bm[];
  chain_wait();
  chain_go();
  uint16_t* before = reinterpret_cast<uint16_t*>(bm + n_kt * cw);   // [word][tile]: queries in earlier words
  const int chunk = blockIdx.x, unit = blockIdx.y;
  const int t0 = chunk * cw * 32, n_q = min(T - t0, cw * 32);
  const int32_t* idx = block_idx + ((size_t)unit * T + t0) * S;
  mark_chunk(idx, bm, t0, n_q, S, block_size, n_kt, cw);
  for (int j = threadIdx.x; j < n_kt; j += kThreads) {
    int run = 0;
    for (int w = 0; w < cw; ++w) {
      before[w * n_kt + j] = (uint16_t)run;
      run += __popc(bm[w * n_kt + j]);
    }
  }
  __syncthreads();
  fill_chunk<kMatch>(idx, bm, before, starts + ((size_t)unit * n_chunks + chunk) * n_kt, pairs,
                     pair_of_slot + ((size_t)unit * T + t0) * S, hdr, t0, n_q, S, block_size, n_kt);
}

// The three steps in one launch for sequences of up to kClusterChunk * kClusterSize tokens: a cluster to a unit, whose
// CTAs take a chunk of queries each and read one another's counts through distributed shared memory, so that nothing
// but the results touches global memory.  The header is zeroed before.  At 4 units of 1024 queries x 16 slots
// 8 us against 14 for the three kernels and the gaps between them; at 4096 queries 22 against 18, at 8192 38
// against 22: eight CTAs a unit are then too few.
constexpr int kClusterSize = 8;
constexpr int kClusterChunk = 256;            // queries
constexpr int kClusterThreads = 1024;
template <bool kMatch>
__global__ void __launch_bounds__(kClusterThreads)
plan_cluster_kernel(const int32_t* block_idx, SelPlan p, int T, int S, int block_size, int n_kt, int cw, int nq,
                    int nq_union) {
  extern __shared__ uint32_t bm[];
  int32_t* cnt = reinterpret_cast<int32_t*>(bm + n_kt * cw);         // [n_kt] pairs of this chunk
  int32_t* st = cnt + n_kt;                                          // [n_kt] first pair of this chunk
  uint16_t* before = reinterpret_cast<uint16_t*>(st + n_kt);         // [word][tile]: queries in earlier words
  __shared__ int warp_sums[32];
  const int rank = (int)blockIdx.x % kClusterSize, unit = (int)blockIdx.x / kClusterSize, tid = threadIdx.x;
  const int t0 = min(T, rank * cw * 32), n_q = min(T - t0, cw * 32);
  const int32_t* idx = block_idx + ((size_t)unit * T + t0) * S;
  mark_chunk(idx, bm, t0, n_q, S, block_size, n_kt, cw);
  int uni = 0;
  const int per = nq_union < 32 ? nq_union : 32, tw = nq_union > 32 ? nq_union / 32 : 1;
  const uint32_t mask = per == 32 ? 0xffffffffu : (1u << per) - 1u;
  for (int j = tid; j < n_kt; j += kClusterThreads) {
    int c = 0;
    uint32_t run = 0u;
    for (int w = 0; w < cw; ++w) {
      const uint32_t b = bm[w * n_kt + j];
      before[w * n_kt + j] = (uint16_t)c;
      c += __popc(b);
      if (per < 32) {
        for (int k = 0; k < 32; k += per) uni += ((b >> k) & mask) != 0u;
      } else {
        run |= b;
        if ((w + 1) % tw == 0 || w + 1 == cw) { uni += run != 0u; run = 0u; }
      }
    }
    cnt[j] = c;
  }
  cluster_sync();
  int pair_carry = unit * T * S, item_carry = 0;
  int32_t* off = p.offsets + (size_t)unit * (n_kt + 1);
  int4* items = p.items + (size_t)unit * p.max_items;
  for (int j0 = 0; j0 < n_kt; j0 += kClusterThreads) {
    const int j = j0 + tid;
    int earlier = 0, all = 0;
    if (j < n_kt) {
#pragma unroll
      for (int r = 0; r < kClusterSize; ++r) {
        const int v = ld_peer_s32(cnt + j, r);
        if (r < rank) earlier += v;
        all += v;
      }
    }
    const int n_rt = (all + nq - 1) / nq;
    const int n_it = j < n_kt ? max(1, (n_rt + kSelChunkTiles - 1) / kSelChunkTiles) : 0;
    int total, total_it;
    const int start = pair_carry + block_scan<kClusterThreads>(all, warp_sums, &total);
    const int first = item_carry + block_scan<kClusterThreads>(n_it, warp_sums, &total_it);
    if (j < n_kt) {
      st[j] = start + earlier;
      if (rank == 0) {
        off[j] = start;
        for (int k = 0; k < n_it && first + k < p.max_items; ++k)
          items[first + k] = make_int4(unit, j, k * kSelChunkTiles, n_it);
      }
    }
    pair_carry += total;
    item_carry += total_it;
  }
  int uni_total;
  block_scan<kClusterThreads>(uni, warp_sums, &uni_total);
  if (tid == 0) {
    if (rank == 0) {
      off[n_kt] = pair_carry;
      p.n_items[unit] = min(item_carry, p.max_items);
      atomicAdd(&p.hdr->pairs, (unsigned long long)(pair_carry - unit * T * S));
    }
    atomicAdd(&p.hdr->union_tiles, (unsigned long long)uni_total);
  }
  __syncthreads();
  fill_chunk<kMatch>(idx, bm, before, st, p.pairs, p.pair_of_slot + ((size_t)unit * T + t0) * S, p.hdr, t0, n_q, S, block_size, n_kt);
  cluster_sync();                            // nobody leaves while its counts are read
}

}  // namespace

SelPlanLayout sel_plan_layout(int units, int T, int S, int nq) {
  SelPlanLayout l;
  l.n_ktiles = (T + kKeysPerTile - 1) / kKeysPerTile;
  // sum over tiles of max(1, ceil(ceil(n_q / nq) / chunk)) <= tiles * (1 + 1/chunk) + pairs / (chunk * nq)
  l.max_items = (int)((size_t)l.n_ktiles + l.n_ktiles / kSelChunkTiles + (size_t)T * S / ((size_t)kSelChunkTiles * nq) + 2);
  // queries per chunk: a long chunk keeps the scan short, a short one keeps the SMs busy and the
  // bitmap inside 64 KB
  int cw = 16;
  while (cw > 1 && ((size_t)l.n_ktiles * cw * 4 > 64 * 1024 || (cw > 2 && (long long)units * ((T + 32 * cw - 1) / (32 * cw)) < 148))) cw >>= 1;
  l.chunk_words = cw;
  l.n_chunks = (T + 32 * cw - 1) / (32 * cw);
  const size_t cap = (size_t)units * T * S;
  size_t off = 0;
  auto take = [&](size_t bytes) { const size_t at = off; off += align_up(bytes, 256); return at; };
  l.hdr = take(sizeof(SelPlanHeader));
  l.n_items = take((size_t)units * 4);
  l.items = take((size_t)units * l.max_items * sizeof(int4));
  l.offsets = take((size_t)units * (l.n_ktiles + 1) * 4);
  l.pairs = take(cap * 4);
  l.pos = take(cap * 4);
  l.scratch = take(((size_t)units * l.n_chunks * l.n_ktiles + (size_t)units * l.n_chunks) * 4);
  l.total = off;
  return l;
}

SelPlan sel_plan_at(const void* base, const SelPlanLayout& l) {
  char* b = (char*)base;
  SelPlan p;
  p.hdr = (SelPlanHeader*)(b + l.hdr);
  p.n_items = (int32_t*)(b + l.n_items);
  p.items = (int4*)(b + l.items);
  p.offsets = (int32_t*)(b + l.offsets);
  p.pairs = (int32_t*)(b + l.pairs);
  p.pair_of_slot = (int32_t*)(b + l.pos);
  p.max_items = l.max_items;
  return p;
}

int sel_plan_build(const int32_t* block_idx, void* base, const SelPlanLayout& l, int units, int T, int S,
                   int block_size, int nq, int nq_union, cudaStream_t st) {
  if (units == 0 || T == 0) return NSA_OK;
  const SelPlan p = sel_plan_at(base, l);
  int32_t* counts = (int32_t*)((char*)base + l.scratch);
  int32_t* unions = counts + (size_t)units * l.n_chunks * l.n_ktiles;
  const size_t smem = (size_t)l.n_ktiles * l.chunk_words * 4;
  const dim3 grid(l.n_chunks, units);
  const bool match = S <= 32 && 32 % S == 0 && l.n_ktiles < (1 << 16);
  if (T <= kClusterChunk * kClusterSize && units <= 64) {       // (more units: the three kernels fill the GPU)
    // chunks of whole query tiles of the union count (at most 64 queries), so that none is counted twice
    const int cw = ((T + kClusterSize - 1) / kClusterSize + 63) / 64 * 2;
    const size_t smem1 = (size_t)l.n_ktiles * (cw * 6 + 8);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kClusterSize;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)units * kClusterSize);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = smem1;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    NSA_CUDA_OK(cudaMemsetAsync(p.hdr, 0, sizeof(SelPlanHeader), st));
    KernelScope ks("plan_cluster_kernel", st);
    auto go = [&](auto kernel) -> int {
      NSA_CUDA_OK(func_smem((const void*)kernel, smem1));
      NSA_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, block_idx, p, T, S, block_size, l.n_ktiles, cw, nq, nq_union));
      return NSA_OK;
    };
    return match ? go(plan_cluster_kernel<true>) : go(plan_cluster_kernel<false>);
  }
  NSA_CUDA_OK(func_smem((const void*)plan_count_kernel, smem));
  NSA_CUDA_OK(match ? func_smem((const void*)plan_fill_kernel<true>, smem + smem / 2)
                    : func_smem((const void*)plan_fill_kernel<false>, smem + smem / 2));
  { KernelScope ks("plan_count_kernel", st);
    NSA_CUDA_OK(launch_chained(plan_count_kernel, grid, kThreads, smem, st, block_idx, counts, unions, p.hdr, T, S, block_size,
                               l.n_ktiles, l.chunk_words, l.n_chunks, nq_union)); }
  { KernelScope ks("plan_scan_kernel", st);
    const bool small = l.n_ktiles <= 256;
    NSA_CUDA_OK(launch_chained(small ? plan_scan_kernel<256> : plan_scan_kernel<1024>, units, small ? 256 : 1024, 0, st, counts, unions,
                               p, T, S, l.n_ktiles, l.n_chunks, nq)); }
  { KernelScope ks("plan_fill_kernel", st);
    NSA_CUDA_OK(launch_chained(match ? plan_fill_kernel<true> : plan_fill_kernel<false>, grid, kThreads, smem + smem / 2, st, block_idx,
                               counts, p.pairs, p.pair_of_slot, p.hdr, T, S, block_size, l.n_ktiles, l.chunk_words, l.n_chunks)); }
  NSA_LAUNCH_OK("selection plan kernels");
  return NSA_OK;
}

}  // namespace nsa
