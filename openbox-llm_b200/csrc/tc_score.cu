// Block scoring + top-n on the tensor cores (replaces the dense scoring pass of
// nsa_model.py:343-355).
//
// Same row tile as the forward kernel: 128 rows = nq queries x Gp heads of one (batch, kv head).
// For every 64-summary tile: S = Q Kc^T by tcgen05.mma; the thread that owns a row turns it
// into compression-branch probabilities p = exp2(s*scale*log2e - lse*log2e) with the LSE the
// compression forward stored; the probabilities go to shared memory and are summed over the Gp
// heads of each query (ascending head order, fp32).  The 128 threads are dealt out 128 / nq per
// query; each keeps in registers the best 16 of the candidates it scanned, ordered by
// (importance descending, block index ascending), and a tournament over the lists' heads writes
// the query's top-n at the end.  Slots with no causally valid block are -1.
#include "tc_common.cuh"
#include "tc_host.cuh"

namespace nsa {
namespace tc {

struct ScoreArgs {
  const float* lse;
  int32_t* block_idx;
  float* imp_out;
  int* status;
  int B, Hq, Hkv, T, n_blk, G, Gp, nq, block_size, n_sel, n_qtiles, n_init, n_local;
  // general geometry (lanes kernel): n_blk summaries of block_size tokens every `stride`; selection
  // blocks of sel_block = r * stride tokens; overlap: block_size == 2 * stride; imp_out has imp_cols columns
  int stride, sel_block, r, overlap, imp_cols;
  float scale_log2;
};


__host__ __device__ inline size_t score_smem_bytes(int D, int nq) {
  return (size_t)(kRows * 128 + 2 * kKeys * 128) * (D / 64) + (size_t)kRows * kKeys * 4 +
         (size_t)nq * kKeys * 4 + 256 + 4 * 32 * 8 + 1024;
}

template <int D>
__global__ void __launch_bounds__(128, 2)
tc_score_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const ScoreArgs p) {
  constexpr int kSlabs = D / 64;
  constexpr int kQBytes = kRows * 128 * kSlabs, kKBytes = kKeys * 128 * kSlabs;
  constexpr uint32_t kTmemCols = 64;
  constexpr uint32_t kIdescQK = idesc_bf16(128, kKeys, 0, 0);

  extern __shared__ uint8_t smem_raw[];
  chain_wait();
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // pointer arithmetic keeps the shared address space
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + kQBytes;                        // 2 stages
  float* sP = (float*)(sK + 2 * kKBytes);            // [128][64] probabilities
  float* sImp = sP + kRows * kKeys;                  // [nq][64] group sums
  uint64_t* bars = (uint64_t*)(sImp + p.nq * kKeys);
  uint64_t* bar_q = bars + 0;
  uint64_t* bar_k = bars + 1;   // [2]
  uint64_t* bar_s = bars + 3;
  uint64_t* bar_drain = bars + 4;   // an aborted CTA waits here for its last MMAs
  uint32_t* s_tmem = (uint32_t*)(bars + 5);
  volatile int* s_abort = (volatile int*)(s_tmem + 1);

  const int tid = threadIdx.x, warp = tid >> 5;
  const int qtile = p.n_qtiles - 1 - (int)blockIdx.x;
  const int bh = blockIdx.y;
  const int b = bh / p.Hkv, hkv = bh % p.Hkv;
  const int t0 = qtile * p.nq;
  const int t_last = min(p.T - 1, t0 + p.nq - 1);
  const int g = tid / p.nq, ql = tid % p.nq;
  const int t = t0 + ql;
  const bool row_ok = (g < p.G) && (t < p.T);

  if (tid == 0) {
    *s_abort = (*(volatile int*)p.status != 0) ? 1 : 0;
    mbar_init(bar_q, 1);
    mbar_init(bar_k + 0, 1); mbar_init(bar_k + 1, 1);
    mbar_init(bar_s, 1);
    mbar_init(bar_drain, 1);
    fence_barrier_init();
    prefetch_tensormap(&tm_q); prefetch_tensormap(&tm_k);
  }
  __syncthreads();
  if (*s_abort) return;

  const int hi_last = min(p.n_blk, (t_last + 1) / p.block_size) - 1;
  int n_tiles = hi_last < 0 ? 0 : hi_last / kKeys + 1;
  // forced blocks (the first n_init, the n_local most recent including the block holding t)
  // are candidates even when incomplete: the tiles reach the block holding the last query
  const bool forcing = p.n_init > 0 || p.n_local > 0;
  if (forcing) n_tiles = max(n_tiles, (t_last / p.block_size) / kKeys + 1);

  // Running top-16 lists: the 128 threads are dealt out Lq = 128 / nq per query; each keeps, in
  // registers, the best 16 of the candidates it has scanned (64 / Lq per tile), ordered by
  // (importance descending, block index ascending).  The Lq lists of a query are merged at the
  // end by a 16-round tournament over their heads.
  constexpr int kList = 16;
  const int Lq = kRows / p.nq;
  const int my_q = tid / Lq, my_sub = tid % Lq;
  const int per_lane = kKeys / Lq;
  const int my_t = t0 + my_q;
  float lv[kList];
  int li[kList];
#pragma unroll
  for (int k = 0; k < kList; ++k) { lv[k] = -1.f; li[k] = -1; }

  uint32_t tmem = 0;
  bool aborted = false;
  int k_loaded = 0, k_seen = 0;   // thread 0: K tiles whose load was issued / whose arrival was seen
  bool q_seen = false;
  if (n_tiles > 0) {
    if (warp == 0) {
      tmem_alloc(s_tmem, kTmemCols);
      tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem = *s_tmem;
    chain_go();
    const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
    const float lse2 = row_ok ? ld_plain(p.lse + (size_t)(b * p.Hq + hkv * p.G + g) * p.T + t) * kLog2e : 0.f;

    auto load_k = [&](int i) {
      uint64_t* bar = bar_k + (i & 1);
      mbar_expect_tx(bar, kKBytes);
#pragma unroll
      for (int s = 0; s < kSlabs; ++s)
        tma_load_3d(sK + (i & 1) * kKBytes + s * (kKeys * 128), &tm_k, bar, s * 64, i * kKeys, bh);
      k_loaded = i + 1;
    };
    auto issue_s = [&](int i) {
      const uint32_t qa = desc_lo_kmajor(smem_u32(sQ)), ka = desc_lo_kmajor(smem_u32(sK + (i & 1) * kKBytes));
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t slab = kk >> 2, in = (kk & 3) * 32;
        mma_ss(tmem, desc_at(qa, slab * (kRows * 128) + in), desc_at(ka, slab * (kKeys * 128) + in),
               kIdescQK, kk > 0);
      }
      tc_commit(bar_s);
    };
    if (tid == 0) {
      mbar_expect_tx(bar_q, kQBytes);
#pragma unroll
      for (int s = 0; s < kSlabs; ++s)
        tma_load_3d(sQ + s * (kRows * 128), &tm_q, bar_q, s * 64, t0, b * p.Hq + hkv * p.G);
      load_k(0);
      if (n_tiles > 1) load_k(1);
      q_seen = mbar_wait(bar_q, 0, p.status, s_abort, 1);
      if (mbar_wait(bar_k, 0, p.status, s_abort, 2)) k_seen = 1;
      tc_fence_after();
      if (!*s_abort) issue_s(0);
    }

    for (int i = 0; i < n_tiles; ++i) {
      const int key0 = i * kKeys;
      const bool s_ok = mbar_wait(bar_s, i & 1, p.status, s_abort, 4);
      tc_fence_after();
      if (tid == 0 && i + 2 < n_tiles && s_ok) load_k(i + 2);
      __syncwarp();
      uint32_t r[64];
      tmem_ld32(lane_base, r);
      tmem_ld32(lane_base + 32, r + 32);
      tmem_wait_ld();
      tc_fence_before();
      const int hi = row_ok ? min(kKeys - 1, min(p.n_blk, (t + 1) / p.block_size) - 1 - key0) : -1;
      float4* dst = reinterpret_cast<float4*>(sP + tid * kKeys);
#pragma unroll
      for (int c4 = 0; c4 < 16; ++c4) {
        float4 v;
        v.x = (c4 * 4 + 0 <= hi) ? ex2(__uint_as_float(r[c4 * 4 + 0]) * p.scale_log2 - lse2) : 0.f;
        v.y = (c4 * 4 + 1 <= hi) ? ex2(__uint_as_float(r[c4 * 4 + 1]) * p.scale_log2 - lse2) : 0.f;
        v.z = (c4 * 4 + 2 <= hi) ? ex2(__uint_as_float(r[c4 * 4 + 2]) * p.scale_log2 - lse2) : 0.f;
        v.w = (c4 * 4 + 3 <= hi) ? ex2(__uint_as_float(r[c4 * 4 + 3]) * p.scale_log2 - lse2) : 0.f;
        // 16-byte chunk index XOR row: a warp's stores spread over the banks
        dst[c4 ^ (tid & 15)] = v;
      }
      // all of S is read, all of P is in shared memory; one decision for the whole CTA: after a
      // given-up wait nothing more is issued or written
      if (__syncthreads_or(*s_abort)) { aborted = true; break; }
      if (tid == 0 && i + 1 < n_tiles) {
        tc_fence_after();
        if (mbar_wait(bar_k + ((i + 1) & 1), ((i + 1) >> 1) & 1, p.status, s_abort, 2)) {
          k_seen = i + 2;
          issue_s(i + 1);
        }
      }
      // group sums: importance[ql][c] = sum over heads, ascending; four columns per thread
      for (int e = tid; e < p.nq * (kKeys / 4); e += 128) {
        const int qq = e / (kKeys / 4), c4 = e % (kKeys / 4);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int gg = 0; gg < p.G; ++gg) {
          const int row = gg * p.nq + qq;
          const float4 v = *reinterpret_cast<const float4*>(sP + row * kKeys + ((c4 ^ (row & 15)) << 2));
          acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        *reinterpret_cast<float4*>(sImp + qq * kKeys + c4 * 4) = acc;
        if (p.imp_out && t0 + qq < p.T) {
          const int hq = min(p.n_blk, (t0 + qq + 1) / p.block_size) - 1 - key0;   // last valid column
          float* out = p.imp_out + ((size_t)bh * p.T + t0 + qq) * p.n_blk + key0 + c4 * 4;
          const float vals[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (key0 + c4 * 4 + e < p.n_blk) out[e] = (c4 * 4 + e <= hq) ? vals[e] : 0.f;
        }
      }
      __syncthreads();
      // top-16 update: this thread scans its share of the query's 64 candidates
      {
        const int hq = my_t < p.T ? min(kKeys - 1, min(p.n_blk, (my_t + 1) / p.block_size) - 1 - key0) : -1;
        const int my_cur = my_t / p.block_size;
        const int hf = (forcing && my_t < p.T) ? min(kKeys - 1, my_cur - key0) : -1;
        for (int k = 0; k < per_lane; ++k) {
          const int c = my_sub * per_lane + k;
          if (c > max(hq, hf)) break;
          const int cj = key0 + c;
          float cv = c <= hq ? sImp[my_q * kKeys + c] : -1.f;
          if (forcing) {                     // cj <= my_cur here
            if (cj < p.n_init) cv = kForcedInit - (float)cj;
            else if (cj > my_cur - p.n_local) cv = kForcedLocal - (float)(my_cur - cj);
          }
          if (cv > lv[kList - 1]) {          // beats the list's last entry (empty slots hold -1)
#pragma unroll
            for (int r = kList - 1; r >= 1; --r) {   // strict '>' keeps earlier (lower) indices ahead
              const bool up = cv > lv[r - 1];
              const bool here = cv > lv[r];
              li[r] = up ? li[r - 1] : (here ? cj : li[r]);
              lv[r] = up ? lv[r - 1] : (here ? cv : lv[r]);
            }
            if (cv > lv[0]) { lv[0] = cv; li[0] = cj; }
          }
        }
      }
      __syncthreads();                         // sP / sImp are rewritten by the next tile
    }
    if (!aborted) aborted = __syncthreads_or(*s_abort) != 0;
    if (aborted) {
      // Give-up path: no list is written.  Thread 0 waits (bounded) for the loads still on their
      // way into this CTA's shared memory and for the MMAs already issued, then the tensor memory
      // goes back.
      if (tid == 0) {
        if (!q_seen) mbar_wait_drain(bar_q, 0);
        for (int j = k_seen; j < k_loaded; ++j) mbar_wait_drain(bar_k + (j & 1), (j >> 1) & 1);
        tc_commit(bar_drain);
        mbar_wait_drain(bar_drain, 0);
      }
      tc_fence_before();
      __syncthreads();
      if (warp == 0) tmem_dealloc(tmem, kTmemCols);
      return;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, kTmemCols);
  }

  // ---- merge the Lq lists of each query: n_sel rounds, each takes the best head ------------------
  for (int r = 0; r < p.n_sel; ++r) {
    float bv = lv[0];
    int bj = li[0];
    for (int o = 1; o < Lq; o <<= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oj = __shfl_xor_sync(0xffffffffu, bj, o);
      if (ov > bv || (ov == bv && oj >= 0 && (bj < 0 || oj < bj))) { bv = ov; bj = oj; }
    }
    if (bj >= 0 && li[0] == bj) {            // this list gave the winner: pop its head
#pragma unroll
      for (int k = 0; k < kList - 1; ++k) { lv[k] = lv[k + 1]; li[k] = li[k + 1]; }
      lv[kList - 1] = -1.f;
      li[kList - 1] = -1;
    }
    if (my_sub == 0 && my_t < p.T) p.block_idx[((size_t)bh * p.T + my_t) * p.n_sel + r] = bj;
  }
  // importance columns no tile covered are zero
  if (p.imp_out && my_t < p.T) {
    float* out = p.imp_out + ((size_t)bh * p.T + my_t) * p.n_blk;
    for (int c = n_tiles * kKeys + my_sub; c < p.n_blk; c += Lq) out[c] = 0.f;
  }
}


// Sorts N candidates by value, largest first, and index, smallest first (Batcher's odd-even merge sort: 63 exchanges
// for 16).  K and P are its merge distance and run length; template arguments, so that every index is a constant.
template <int N, int P = 1, int K = 1>
__device__ __forceinline__ void sort_candidates(float (&v)[N], int (&j)[N]) {
#pragma unroll
  for (int a = 0; a < N - K; ++a) {
    const int b = a + K, s = a - K % P;
    if (s >= 0 && s % (2 * K) < K && a / (2 * P) == b / (2 * P)) {
      const bool swap = v[b] > v[a] || (v[b] == v[a] && j[b] < j[a]);
      const float tv = swap ? v[b] : v[a];
      const int tj = swap ? j[b] : j[a];
      v[b] = swap ? v[a] : v[b]; j[b] = swap ? j[a] : j[b];
      v[a] = tv; j[a] = tj;
    }
  }
  if constexpr (K > 1) sort_candidates<N, P, K / 2>(v, j);
  else if constexpr (2 * P < N) sort_candidates<N, 2 * P, 2 * P>(v, j);
}

// ------------------------------------------------------------------------------------------
// The same for GQA groups of 4, 8 or 16 (padded) heads, with the score tile turned round: summaries in the lanes of tensor
// memory, rows (query-major: query * GP + head, one TMA box from the (D, heads, T) view of q) in its columns.  A thread has
// one summary and adds the heads of a query up in registers, in the order (h, h + GP/2), ..., (h, h + 1); the sums go through
// shared memory to the GP lanes of the query, lane g taking the tile's summaries [g * n / GP, (g + 1) * n / GP) into
// its top-16 list.  A tile has 128 summaries, or, where 64 or 32 are left, two or four copies of those, so that all warps have
// columns to do: warp w does n columns of its copy.
// What bounds it: exponentials (1024 cycles of a full tile's 3.9 k at 64 heads) and the lists' bookkeeping, three CTAs of four warps an SM (four
// at D = 64), and in short calls fetching instructions: insertions are loops, not unrolled.  Rows in the lanes, heads added by a
// recursive-halving exchange of shuffles, took 240 instructions of a warp per 64 summaries; 64 heads of 128 x 65536 tokens 2.37 ->
// 1.97 ms, 8 x 32768 tokens of 16 heads 2.0 -> 1.64, 8 x 4096 tokens of 12 heads of 64 109 -> 81 us.  The first tile's candidates go into
// the empty lists by a sorting network (8 x 4096 tokens: 110 -> 101 us when it came).
// Groups of 4 at D = 128 hold 18 KB of sums beside 64 KB of Q and K: two CTAs an SM, which took longer than the shuffles from some 150 CTAs on.
// There the sums lie over K, for a third CTA, and the next K is fetched after the lists, under the other CTAs' work (the shuffles | two
// CTAs | this, us): 8192 tokens of 16 heads on 4 41 | 51 | 39, 16384 101 | 113 | 88, 65536 987 | 761 | 586; overlapping summaries every 16
// tokens, 4096 29 | 38 | 28, 16384 184 | 254 | 173 (195 of it with divisions and five sums a block instead of shifts and four).
// Forced blocks on the summaries' grid go into the lists by themselves, before the others (the shuffles | every candidate looked at one
// by one for their sake | this, block 0 and two local ones, 32768 tokens): 12 heads of 64 on 4 317 | 367 | 181, 16 on 2 224 | 234 | 152, 12 of 128
// on 4 332 | 544 | 223, 16 on 1 203 | 209 | 172; at 1024 tokens 14.6 to 15.9 | 14.6 | 12.8 to 14.6.
// ------------------------------------------------------------------------------------------
constexpr int kImpLd = 144;              // floats of a query's row of sums: 128, and 4 more after every 32 (16-byte reads without conflicts)

template <int D, int GP> struct ScoreLanes {
  static constexpr int kSlabs = D / 64;
  static constexpr int kQBytes = kRows * 128 * kSlabs, kKBytes = 128 * 128 * kSlabs;
  // Groups of 4 at D = 128: 18 KB of sums beside Q and K would leave two CTAs an SM; they take the place of K, and the next K waits.
  static constexpr bool kOverK = D == 128 && GP == 4;
  static constexpr int kImpBytes = kOverK ? 0 : kRows / GP * kImpLd * 4;
  static constexpr size_t kSmem = kQBytes + kKBytes + kImpBytes + 128 * 4 /*lse*/ + 64 /*barriers*/ + 1024;
  static constexpr int kCtas = (int)(227 * 1024 / (kSmem + 1024)) > 4 ? 4 : (int)(227 * 1024 / (kSmem + 1024));
};

// kForm: kApart, summaries and blocks on grids of their own; kSame, the same grid; kPlain, that without forced blocks and
// importances, whose code the others would fetch and step over (the op on 512 tokens, 16 heads on 4, replayed from a graph 36.3 us with it, 35.1
// without; 131072 tokens, 24 heads on 4, the scorer 2401 and 2323).
enum ScoreForm { kApart, kSame, kPlain };
template <int D, int GP, ScoreForm kForm>
__global__ void __launch_bounds__(128, ScoreLanes<D, GP>::kCtas)
tc_score_lanes_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const ScoreArgs p) {
  using L = ScoreLanes<D, GP>;
  constexpr int kSlabs = L::kSlabs, kQBytes = L::kQBytes, kKBytes = L::kKBytes;
  constexpr bool kOverK = L::kOverK, kAligned = kForm != kApart;
  constexpr uint32_t kTmemCols = 128;
  constexpr uint32_t kIdescKQ = idesc_bf16(128, 128, 0, 0);
  constexpr int NQ = kRows / GP;       // queries per tile
  constexpr int PER = 128 / GP;        // summaries of a full tile that a lane takes
  constexpr int kList = 16;

  extern __shared__ uint8_t smem_raw[];
  chain_wait();
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + kQBytes;
  float* s_imp = (float*)(kOverK ? sK : sK + kKBytes);              // [NQ][kImpLd]
  float* s_lse = (float*)(sK + kKBytes + L::kImpBytes);            // [128], negative, log2 units
  uint64_t* bars = (uint64_t*)(s_lse + 128);
  uint64_t* bar_q = bars + 0;
  uint64_t* bar_k = bars + 1;
  uint64_t* bar_s = bars + 2;
  uint64_t* bar_drain = bars + 3;   // an aborted CTA waits here for its last MMAs
  uint32_t* s_tmem = (uint32_t*)(bars + 4);
  volatile int* s_abort = (volatile int*)(s_tmem + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int qtile = p.n_qtiles - 1 - (int)blockIdx.x;
  const int bh = blockIdx.y;
  const int b = bh / p.Hkv, hkv = bh % p.Hkv;
  const int t0 = qtile * NQ;
  const int t_last = min(p.T - 1, t0 + NQ - 1);
  const int g = tid % GP, ql = tid / GP;
  const int t = t0 + ql;
  const bool row_ok = (g < p.G) && (t < p.T);

  if (tid == 0) {
    *s_abort = (*(volatile int*)p.status != 0) ? 1 : 0;
    mbar_init(bar_q, 1);
    mbar_init(bar_k, 1);
    mbar_init(bar_s, 1);
    mbar_init(bar_drain, 1);
    fence_barrier_init();
    prefetch_tensormap(&tm_q); prefetch_tensormap(&tm_k);
  }
  __syncthreads();
  if (*s_abort) return;

  int n_sum = cmp_visible(t_last, p.block_size, p.stride, p.n_blk);      // summaries to go through
  // (a block is a candidate from the summary before it on where they overlap: its own may be in the next tile)
  if (!kAligned && n_sum > 0) n_sum += p.overlap;
  const bool forcing = kForm != kPlain && (p.n_init > 0 || p.n_local > 0);
  // forced blocks are candidates whatever their importance: as far as the block that holds the last query
  if (forcing) n_sum = max(n_sum, p.r * (t_last / p.sel_block + 1));
  const int n_tiles = (n_sum + 127) / 128;
  // summaries in tile i: 128, or 64 or 32 (several copies) where that is what is left; whole blocks for each lane
  auto size_of = [&](int i) -> int {
    const int left = n_sum - 128 * i;
    return left > 64 ? 128 : left > 32 || (!kAligned && p.r * GP > 32) ? 64 : 32;
  };

  float lv[kList];
  int li[kList];
#pragma unroll
  for (int k = 0; k < kList; ++k) { lv[k] = -1.f; li[k] = -1; }

  if (n_tiles > 0) {
    int k_loaded = 0, k_seen = 0;   // thread 0: K tiles whose load was issued / whose arrival was seen
    auto load_k = [&](int i) {
      const int groups = size_of(i) / 32;
      mbar_expect_tx(bar_k, kKBytes);
#pragma unroll
      for (int sl = 0; sl < kSlabs; ++sl)
#pragma unroll
        for (int r = 0; r < 4; ++r)
          tma_load_3d(sK + sl * (128 * 128) + r * (32 * 128), &tm_k, bar_k, sl * 64, i * 128 + 32 * (r % groups), bh);
      k_loaded = i + 1;
    };
    if (tid == 0) {                 // on their way while the rest is set up
      mbar_expect_tx(bar_q, kQBytes);
#pragma unroll
      for (int sl = 0; sl < kSlabs; ++sl)     // box: 64 columns x GP heads x NQ tokens
        tma_load_3d(sQ + sl * (kRows * 128), &tm_q, bar_q, sl * 64, b * p.Hq + hkv * p.G, t0);
      load_k(0);
    }
    __syncwarp();
    if (warp == 0) {
      tmem_alloc(s_tmem, kTmemCols);
      tmem_relinquish();
    }
    s_lse[tid] = row_ok ? ld_plain(p.lse + (size_t)(b * p.Hq + hkv * p.G + g) * p.T + t) * -kLog2e : 0.f;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;
    chain_go();
    const uint64_t sc2 = pack_f32x2(p.scale_log2, p.scale_log2);
    bool aborted = false, q_seen = false;
    const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
    const int n_vis = t < p.T ? cmp_visible(t, p.block_size, p.stride, p.n_blk) : 0;   // summaries query t sees
    const int my_cur = t / p.sel_block;              // selection block that holds t
    float carry = 0.f;                               // last summary of the previous tile (overlap)

    auto insert = [&](float cv, int cj) {
      if (cv > lv[kList - 1]) {                // beats the list's last entry (empty slots hold -1)
#pragma unroll
        for (int r = kList - 1; r >= 1; --r) {   // strict '>' keeps earlier (lower) indices ahead
          const bool up = cv > lv[r - 1];
          const bool here = cv > lv[r];
          li[r] = up ? li[r - 1] : (here ? cj : li[r]);
          lv[r] = up ? lv[r - 1] : (here ? cv : lv[r]);
        }
        if (cv > lv[0]) { lv[0] = cv; li[0] = cj; }
      }
    };
    auto issue_s = [&]() {
      const uint32_t qa = desc_lo_kmajor(smem_u32(sQ)), ka = desc_lo_kmajor(smem_u32(sK));
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t at = (kk >> 2) * (128 * 128) + (kk & 3) * 32;
        mma_ss(tmem, desc_at(ka, at), desc_at(qa, at), kIdescKQ, kk > 0);
      }
      tc_commit(bar_s);
    };
    if (tid == 0) {
      q_seen = mbar_wait(bar_q, 0, p.status, s_abort, 1);
      if (mbar_wait(bar_k, 0, p.status, s_abort, 2)) k_seen = 1;
      tc_fence_after();
      if (!*s_abort) issue_s();
    }

    for (int i = 0; i < n_tiles; ++i) {
      const int key0 = i * 128, size = size_of(i);
      const int per = size / GP;                     // of the tile's summaries, a lane's
      const bool s_ok = mbar_wait(bar_s, i & 1, p.status, s_abort, 4);
      tc_fence_after();
      __syncwarp();
      if (!kOverK && tid == 0 && s_ok && i + 1 < n_tiles) load_k(i + 1);          // the MMAs have read this tile's
      {
        const int at = 32 * (warp % (size / 32)) + lane;               // this thread's summary in the tile
        const int c0 = warp / (size / 32) * size;                      // and its columns
        float* imp = s_imp + at + 4 * (at >> 5);
#pragma unroll 1
        for (int c = c0; c < c0 + size; c += 32) {
          uint32_t r[32];
          tmem_ld32(lane_base + c, r);
          uint64_t e[16];                            // two columns each
          tmem_wait_ld();
#pragma unroll
          for (int k = 0; k < 16; k += 2) {
            const ulonglong2 l = *reinterpret_cast<const ulonglong2*>(s_lse + c + 2 * k);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              float e0, e1;
              unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[2 * (k + x)]), __uint_as_float(r[2 * (k + x) + 1])), sc2, x ? l.y : l.x), e0, e1);
              e0 = ex2(e0);
              e1 = ex2(e1);
              // (padding: rows of the next group, or none)
              const int h = 2 * (k + x) % GP;
              if (h > GP / 2 && h >= p.G) e0 = 0.f;
              if (h + 1 > GP / 2 && h + 1 >= p.G) e1 = 0.f;
              e[k + x] = pack_f32x2(e0, e1);
            }
          }
#pragma unroll
          for (int q = 0; q < 32 / GP; ++q) {
#pragma unroll
            for (int o = GP / 4; o >= 1; o >>= 1)
#pragma unroll
              for (int h = 0; h < o; ++h) e[q * GP / 2 + h] = add_f32x2(e[q * GP / 2 + h], e[q * GP / 2 + h + o]);
            float e0, e1;
            unpack_f32x2(e[q * GP / 2], e0, e1);
            imp[(c / GP + q) * kImpLd] = e0 + e1;
          }
        }
        tc_fence_before();
      }
      // the sums are there, and S has been read: the next MMA may overwrite it; one decision for the whole CTA:
      // after a given-up wait nothing more is issued or written
      if (__syncthreads_or(*s_abort)) { aborted = true; break; }
      auto next_s = [&]() {
        tc_fence_after();
        if (mbar_wait(bar_k, (i + 1) & 1, p.status, s_abort, 2)) {
          k_seen = i + 2;
          issue_s();
        }
      };
      if (!kOverK && tid == 0 && i + 1 < n_tiles) next_s();
      __syncwarp();
      // the query's sum at place k of the tile; what it does not see is zero
      auto sum_at = [&](int k) -> float { return key0 + k < n_vis ? s_imp[ql * kImpLd + k + 4 * (k >> 5)] : 0.f; };
      float* out = (!kAligned && p.imp_out && t < p.T) ? p.imp_out + ((size_t)bh * p.T + t) * p.imp_cols : nullptr;
      // A candidate below entry 16 / GP (counted from 1) of every one of the query's GP lists has
      // at least 16 entries ahead of it, so it cannot reach the merged top 16 and need not enter a
      // list; the bound only rises while the tile is scanned.
      auto bound = [&]() -> float {
        float tau = lv[kList / GP - 1];
#pragma unroll
        for (int o = 1; o < GP; o <<= 1) tau = fminf(tau, __shfl_xor_sync(0xffffffffu, tau, o));
        return tau;
      };
      // Forced blocks, with values of more than any sum: the first n_init, and those from loc0 to the query's.
      const int last_cur = forcing && t < p.T ? my_cur : -1, loc0 = max(p.n_init, my_cur - p.n_local + 1);
      if (kAligned) {
        // summaries and blocks coincide: lane g's are c0 + k, and the first n_cand of them candidates
        const int c0 = key0 + g * per, n_cand = min(per, n_vis - c0);
        float v[PER];
        if (per >= 4) {
          const int at = g * per;
          const float* imp = s_imp + ql * kImpLd + at + 4 * (at >> 5);
#pragma unroll
          for (int k = 0; k < PER; k += 4) {
            if (k >= per) break;
            const float4 x = *reinterpret_cast<const float4*>(imp + k);
            v[k] = x.x; v[k + 1] = x.y; v[k + 2] = x.z; v[k + 3] = x.w;
          }
        } else {
          v[0] = sum_at(g * per); v[1] = sum_at(g * per + 1);
        }
        const int c1 = c0 + per - 1, hi1 = min(min(c1, p.n_init - 1), last_cur), lo2 = max(c0, loc0), hi2 = min(c1, last_cur);
        uint32_t by_force = 0u;                      // not candidates by their sums
        if (kForm == kSame && c0 <= hi1) by_force |= (2u << (hi1 - c0)) - 1u;
        if (kForm == kSame && lo2 <= hi2) by_force |= ((2u << (hi2 - lo2)) - 1u) << (lo2 - c0);
        constexpr int kSort = 64 / GP;               // candidates of the first tile that are sorted into the empty lists
        if (i == 0) {
          float sv[kSort];
          int sj[kSort];
#pragma unroll
          for (int k = 0; k < kSort; ++k) {
            sv[k] = k < n_cand && !((by_force >> k) & 1u) && v[k] >= 0.f ? v[k] : -1.f;    // (not what is NaN, which enters no list)
            sj[k] = c0 + k;
          }
          sort_candidates<kSort>(sv, sj);
#pragma unroll
          for (int k = 0; k < kSort; ++k) {
            lv[k] = sv[k];
            li[k] = sv[k] > -1.f ? sj[k] : -1;
          }
        }
        // (Importances, where asked for: a warp's lanes write 32 columns of each of its queries.  A lane its own summaries: 16 heads of 64 on 4,
        // 32768 tokens 326 us with the call's other work, now 229; 16 of 128 on 4, 8192 tokens 45 -> 40.)
        if (kForm != kPlain && p.imp_out) {
          for (int k = lane; k < size; k += 32) {
            const float* imp = s_imp + warp * (32 / GP) * kImpLd + k + 4 * (k >> 5);
            float* row = p.imp_out + ((size_t)bh * p.T + t0 + warp * (32 / GP)) * p.imp_cols + key0 + k;
#pragma unroll
            for (int q = 0; q < 32 / GP; ++q) {
              const int sees = __shfl_sync(0xffffffffu, n_vis, q * GP);
              if (t0 + warp * (32 / GP) + q < p.T && key0 + k < p.imp_cols) row[(size_t)q * p.imp_cols] = key0 + k < sees ? imp[q * kImpLd] : 0.f;
            }
          }
        }
        if (by_force) {
#pragma unroll 1
          for (uint32_t f = by_force; f; f &= f - 1u) {
            const int cj = c0 + __ffs(f) - 1;
            insert(cj < p.n_init ? kForcedInit - (float)cj : kForcedLocal - (float)(my_cur - cj), cj);
          }
        }
        if (i == 0 && per <= kSort) break;           // (the one tile there is)
        // those that are left, a bit each: a lane's next one a round, for as many rounds as the lane with most of them needs
        const float tau = bound();
        uint32_t left = 0u;
#pragma unroll
        for (int k = 0; k < PER; ++k)
          if (k < n_cand && !(i == 0 && k < kSort) && v[k] > lv[kList - 1] && v[k] >= tau) left |= 1u << k;
        left &= ~by_force;
        while (__any_sync(0xffffffffu, left != 0u)) {
          if (left) {
            const int k = __ffs(left) - 1;
            left &= left - 1u;
            insert(sum_at(g * per + k), c0 + k);
          }
          __syncwarp();
        }
      } else {
        // A selection block is r consecutive summaries (plus, when the summaries overlap, the one before them); it is a
        // candidate once its first summary is visible.
        const int r_ = p.r, ov_ = p.overlap, log_r = 31 - __clz(p.r);       // (r: a power of two)
        const float tau = bound();
        float last = !ov_ ? 0.f : g == 0 ? carry : sum_at(g * per - 1);     // the summary ahead, where blocks share one
#pragma unroll 1
        for (int k = g * per; k < (g + 1) * per; k += r_) {
          float acc = ov_ ? last : 0.f;
#pragma unroll 1
          for (int e = 0; e < r_; ++e) acc += last = sum_at(k + e);
          const int cj = (key0 + k) >> log_r;                        // block index
          const bool visible = max(0, r_ * cj - ov_) < n_vis;        // first overlapping summary
          if (out && cj < p.imp_cols) out[cj] = visible ? acc : 0.f;
          float cv = visible ? acc : -1.f;
          if (cj <= last_cur) {
            if (cj < p.n_init) cv = kForcedInit - (float)cj;
            else if (cj >= loc0) cv = kForcedLocal - (float)(my_cur - cj);
          }
          if (cv >= tau) insert(cv, cj);
        }
        carry = sum_at(size - 1);
      }
      if (i + 1 < n_tiles) {
        if (kOverK) fence_proxy_async();
        __syncthreads();                             // the next tile's sums (or itself) may be written
        if (kOverK && tid == 0) {
          load_k(i + 1);
          next_s();
        }
        if (kOverK) __syncwarp();
      }
    }
    if (!aborted) aborted = __syncthreads_or(*s_abort) != 0;
    if (aborted) {
      // Give-up path: no list is written.  Thread 0 waits (bounded) for the loads still on their
      // way into this CTA's shared memory and for the MMAs already issued, then the tensor memory
      // goes back.
      if (tid == 0) {
        if (!q_seen) mbar_wait_drain(bar_q, 0);
        for (int j = k_seen; j < k_loaded; ++j) mbar_wait_drain(bar_k, j & 1);
        tc_commit(bar_drain);
        mbar_wait_drain(bar_drain, 0);
      }
      tc_fence_before();
      __syncthreads();
      if (warp == 0) tmem_dealloc(tmem, kTmemCols);
      return;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, kTmemCols);
  }

  // ---- merge the GP lists of each query: n_sel rounds, each takes the best head ------------------
  for (int r = 0; r < p.n_sel; ++r) {
    float bv = lv[0];
    int bj = li[0];
#pragma unroll
    for (int o = 1; o < GP; o <<= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oj = __shfl_xor_sync(0xffffffffu, bj, o);
      if (ov > bv || (ov == bv && oj >= 0 && (bj < 0 || oj < bj))) { bv = ov; bj = oj; }
    }
    if (bj >= 0 && li[0] == bj) {            // this list gave the winner: pop its head
#pragma unroll
      for (int k = 0; k < kList - 1; ++k) { lv[k] = lv[k + 1]; li[k] = li[k + 1]; }
      lv[kList - 1] = -1.f;
      li[kList - 1] = -1;
    }
    if (g == 0 && t < p.T) p.block_idx[((size_t)bh * p.T + t) * p.n_sel + r] = bj;
  }
  // importance columns no tile covered are zero
  if (kForm != kPlain && p.imp_out && t < p.T) {
    float* out = p.imp_out + ((size_t)bh * p.T + t) * p.imp_cols;
    const int seen = n_tiles > 0 ? (n_tiles - 1) * 128 + size_of(n_tiles - 1) : 0;
    for (int c = seen / (kAligned ? 1 : p.r) + g; c < p.imp_cols; c += GP) out[c] = 0.f;
  }
}

template <int D, int GP>
static int launch_score_lanes(const void* q, const void* k_cmp, const NsaDims& d, int n_blk, ScoreArgs p,
                              cudaStream_t st) {
  p.nq = kRows / GP;
  p.n_qtiles = (d.T + p.nq - 1) / p.nq;
  CUtensorMap tm_q, tm_k;
  int rc = make_map_query_rows(&tm_q, q, d.D, d.T, d.B * d.Hq, GP, p.nq);
  if (rc == NSA_OK) rc = make_map(&tm_k, k_cmp, d.D, n_blk, d.B * d.Hkv, 32, 1);
  if (rc != NSA_OK) return rc;
  const size_t smem = ScoreLanes<D, GP>::kSmem;
  KernelScope ks("tc_score_topn", st);
  const bool same = p.r == 1 && p.overlap == 0, plain = same && !p.imp_out && p.n_init <= 0 && p.n_local <= 0;
  const auto kernel = plain ? tc_score_lanes_kernel<D, GP, kPlain> : same ? tc_score_lanes_kernel<D, GP, kSame> : tc_score_lanes_kernel<D, GP, kApart>;
  NSA_CUDA_OK(func_smem((const void*)kernel, smem));
  NSA_CUDA_OK(launch_chained(kernel, dim3(p.n_qtiles, d.B * d.Hkv), 128, smem, st, tm_q, tm_k, p));
  return NSA_OK;
}

}  // namespace tc

bool tc_topn_ok(const NsaDims& d, int n_blk, int n_sel, int cmp_len, int stride, int sel_block) {
  if (d.dtype != NSA_DTYPE_BF16 || (d.D != 64 && d.D != 128)) return false;
  if (n_sel < 1 || n_sel > 16 || n_blk < 1) return false;
  const int G = d.Hq / d.Hkv;
  if (G > 32) return false;   // at least 4 queries per tile, so the lanes of one query sit in one warp
  if (cmp_len == stride && stride == sel_block) return true;
  // summaries and selection blocks on different grids: the lane-exchange kernel only
  const int gp = tc::group_pad(G);
  if (gp != 4 && gp != 8 && gp != 16) return false;
  if (stride <= 0 || sel_block % stride || cmp_len % stride) return false;
  const int r = sel_block / stride, o = cmp_len / stride;
  return (r & (r - 1)) == 0 && r <= tc::kKeys / gp && (o == 1 || o == 2);
}

int tc_topn(const void* q, const void* k_cmp, const float* lse, int32_t* block_idx, float* imp_out,
            const NsaDims& d, int n_blk, int block_size, int n_sel, int n_init, int n_local, int stride,
            int sel_block, int imp_cols, cudaStream_t st) {
  using namespace tc;
  ScoreArgs p;
  p.lse = lse; p.block_idx = block_idx; p.imp_out = imp_out;
  p.status = device_status_ptr();
  if (!p.status) { set_error("device status word unavailable"); return NSA_ERR_CUDA; }
  p.B = d.B; p.Hq = d.Hq; p.Hkv = d.Hkv; p.T = d.T; p.n_blk = n_blk;
  p.G = d.Hq / d.Hkv; p.Gp = group_pad(p.G); p.nq = kRows / p.Gp;
  p.block_size = block_size; p.n_sel = n_sel; p.n_init = n_init; p.n_local = n_local;
  p.stride = stride; p.sel_block = sel_block; p.r = sel_block / stride;
  p.overlap = block_size / stride - 1; p.imp_cols = imp_cols;
  p.n_qtiles = (d.T + p.nq - 1) / p.nq;
  p.scale_log2 = kLog2e / sqrtf((float)d.D);
  if (p.Gp == 4 || p.Gp == 8 || p.Gp == 16) {
    int rc = NSA_ERR_UNSUPPORTED;
    if (d.D == 128) rc = p.Gp == 4 ? launch_score_lanes<128, 4>(q, k_cmp, d, n_blk, p, st)
                       : p.Gp == 8 ? launch_score_lanes<128, 8>(q, k_cmp, d, n_blk, p, st)
                                   : launch_score_lanes<128, 16>(q, k_cmp, d, n_blk, p, st);
    else rc = p.Gp == 4 ? launch_score_lanes<64, 4>(q, k_cmp, d, n_blk, p, st)
            : p.Gp == 8 ? launch_score_lanes<64, 8>(q, k_cmp, d, n_blk, p, st)
                        : launch_score_lanes<64, 16>(q, k_cmp, d, n_blk, p, st);
    if (rc != NSA_OK) return rc;
    NSA_LAUNCH_OK("tc_score_lanes_kernel");
    return NSA_OK;
  }
  CUtensorMap tm_q, tm_k;
  int rc = make_map(&tm_q, q, d.D, d.T, d.B * d.Hq, p.nq, p.Gp);
  if (rc == NSA_OK) rc = make_map(&tm_k, k_cmp, d.D, n_blk, d.B * d.Hkv, kKeys, 1);
  if (rc != NSA_OK) return rc;
  const size_t smem = score_smem_bytes(d.D, p.nq);
  dim3 grid(p.n_qtiles, d.B * d.Hkv);
  if (d.D == 128) {
    NSA_CUDA_OK(func_smem((const void*)tc_score_kernel<128>, smem));
    KernelScope ks("tc_score_topn", st);
    NSA_CUDA_OK(launch_chained(tc_score_kernel<128>, grid, 128, smem, st, tm_q, tm_k, p));
  } else {
    NSA_CUDA_OK(func_smem((const void*)tc_score_kernel<64>, smem));
    KernelScope ks("tc_score_topn", st);
    NSA_CUDA_OK(launch_chained(tc_score_kernel<64>, grid, 128, smem, st, tm_q, tm_k, p));
  }
  NSA_LAUNCH_OK("tc_score_kernel");
  return NSA_OK;
}

}  // namespace nsa
