// tcgen05 / TMEM attention kernels for sm_100a.
//
// One CTA owns a tile of 128 rows = nq consecutive query tokens x the G query heads of one
// (batch, kv head) group (row r -> token r / G, head r % G), so the heads of a GQA group share
// every K/V tile; nq = 128 / G, so a group of 3 fills 126 rows.  The CTA walks a list of 64-key tiles:
//   window      the tiles covering [t_first - W + 1, t_last]
//   compression the tiles covering summaries [0, (t_last + 1) / Bsz - 1]
//   selection   the 64-key tiles holding blocks (of 16, 32 or 64 tokens) listed for the tile's nq
//               queries, found in shared memory, with a membership bit per (query, block)
// Per tile: a TMA warp brings K and V (128B-swizzled boxes) into a ring; an MMA warp issues
// S = Q K^T (tcgen05.mma, accumulator in one of two TMEM buffers); each of the 128 softmax threads
// owns one row of S (tcgen05.ld, lane = row), masks it, runs the online softmax in the log2 domain
// without any cross-thread traffic and writes P as packed bf16 over S in TMEM (tcgen05.st); the MMA
// warp then issues O += P V with P as the TMEM A operand and V as an MN-major shared-memory B
// operand.  The running maximum is only raised when it grows by more than 8 (log2 units), so the O
// accumulator in TMEM is rescaled rarely.
#include <algorithm>

#include "sel_row.cuh"
#include "tc_common.cuh"
#include "tc_host.cuh"

namespace nsa {
namespace tc {

struct FwdArgs {
  const int32_t* block_idx;
  __nv_bfloat16* o;
  float* lse;
  int* status;
  int B, Hq, Hkv, T, Lk, S, G, nq;
  int kind, window, block_size;
  const SelPlanHeader* plan;         // selection: statistics for the variant choice (null: this kernel serves the call)
  int force;
  int nq_union;              // queries per query tile in the plan's statistics (G padded to a power of two)
  int debug_starve;          // test only: the V load of the second key tile is never sent
  int n_qtiles, nb_sel;      // nb_sel = ceil(T / 64) key tiles a selection list may name
  int nw;                    // 32-bit membership words per block = ceil(nq / 32)
  int n_sub;                 // selection: list blocks per 64-key tile (64 / block_size)
  float scale_log2;
  const __nv_bfloat16* q;    // three-term selection: the rows that are done again one by one
  const __nv_bfloat16* k;
  const __nv_bfloat16* v;
  float neg_zero;            // -0: what a product is added to where it has to be rounded by itself (a packed mul
                             //     and the add after it are merged into one fma, whatever their rounding says)
};

// D = 128: Q 32 KB + two stages of K and V = 96 KB, two CTAs per SM.  D = 64: four stages in 80 KB.
template <int D> struct FwdSmem {
  static constexpr int kSlabs = D / 64;
  static constexpr int kStages = D == 64 ? 4 : 2;
  static constexpr int kQBytes = kRows * 128 * kSlabs;
  static constexpr int kKVBytes = kKeys * 128 * kSlabs;
  static constexpr int kFixed = kQBytes + 2 * kStages * kKVBytes;
  static constexpr int kBars = 9 + 4 * kStages + (D == 128 ? 4 : 0);
};

__host__ __device__ inline size_t fwd_smem_bytes(int D, int nb_sel, int nw, int n_sub, int kind) {
  size_t extra = 256 /*barriers etc*/ + 132 * 4 /*scan*/;
  if (kind == 2) extra += (size_t)nb_sel * n_sub * nw * 4 + (size_t)nb_sel * 2 + 16;
  return (D == 64 ? FwdSmem<64>::kFixed : FwdSmem<128>::kFixed) + extra + 1024 /*alignment slack*/;
}

constexpr int kFwdThreads = 192;
constexpr int kFwdSoftmax = 128;

// One kernel for the three branches (kKind: 0 window, 1 compression, 2 selection).  192 threads in roles: warps 0-3 (thread = row
// = TMEM lane) own the softmax, warp 4 sends the TMA loads, warp 5 issues the MMAs; two CTAs per SM,
// each walking many row tiles (tile w, w + gridDim.x, ...), long rows first.
//
// What bounds it: one row tile is a chain S -> exponentials -> P V per key tile, and with a single S
// buffer the hand-overs of that chain (two barrier hops, two MMA latencies) took twice the
// arithmetic: 1.34 k cycles per key tile and SM with two chains running, where the exponentials
// need 512 (16 MUFU results per clock), the MMAs as much, and shared memory 768 (operands and
// incoming tiles, D = 128).  Two S buffers take the MMA latency out of the chain: S of the next key
// tile is computed while the softmax works on this one.  They fill the tensor memory that Q
// occupied before (O 128 + 2 x 64 columns per CTA), so S takes both operands from shared memory.
// The producer runs ahead into the next row tile, whose first S is computed while the threads write
// this tile's output.  Every barrier's phase follows a running count (of row tiles, or of key tiles
// over all row tiles) that each role keeps itself.
//
// Selection builds the list of a row tile's key tiles first, all threads together, and so works row
// tile by row tile.
//
// Score * scale is rounded before the maximum is subtracted, and a tile's probabilities are summed in
// column order: the three branches give the same bits on the same keys.  (A shift common to all keys
// leaves a softmax as it is, so the gradients of the summaries sum to zero over the keys and the
// gradient of the key pooling's position parameters is what rounding leaves of that sum, 3e-4 of the
// other gradients.  Any other rounding here, or order of the sum in backward, is as exact and replaces
// these values by others of their size.)
//
// kThreeTerm (selection on 16- and 32-token blocks, whose results are fp32 arithmetic rounded once): P goes to the
// tensor cores as three bf16 terms, each what the ones before it leave of P: all 24 bits of an fp32 value, at the price
// of two more products.  The first two take the 64 columns that S leaves behind; the third has 32 columns of its own at
// D = 64, those that O does not use, and at D = 128, where tensor memory is full, follows into the columns of the first
// as soon as that one's product is done.  2 x 1024 tokens, 16 heads of 128, 8 blocks of 16 a list: 42 us (50 with columns
// for all terms, which leave room for one CTA an SM; 32 with two terms, whose 16 bits show in sums that cancel; 27
// with one).  A block listed twice counts twice; a row whose result is not finite (V of a key it does not attend may be
// infinite: zero times that is NaN) is done again by itself.
template <int D, int kKind, bool kThreeTerm>
__global__ void __launch_bounds__(kFwdThreads, 2)
tc_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
              const __grid_constant__ CUtensorMap tm_v, const FwdArgs p) {
  using L = FwdSmem<D>;
  constexpr int kSlabs = L::kSlabs, kStages = L::kStages;
  constexpr bool kSel = kKind == 2, kCmp = kKind == 1;
  constexpr uint32_t kTmemCols = 256;
  constexpr bool kLate = kThreeTerm && D == 128;    // the third term of P waits for the first to be used
  // O in columns 0-127, two buffers of S (P, bf16, is written over the first 32 columns of its S by the
  // thread that read the row; three-term: over all 64, and the third term of buffer b at kColP3 + b * kP3Step)
  constexpr uint32_t kColO = 0, kColS = 128, kColP3 = kLate ? kColS : 64, kP3Step = kLate ? kKeys : 32;
  constexpr uint32_t kIdescQK = idesc_bf16(128, kKeys, 0, 0);
  constexpr uint32_t kIdescPV = idesc_bf16(128, D, 0, 1);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // pointer arithmetic keeps the shared address space
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + L::kQBytes;
  uint8_t* sV = sK + kStages * L::kKVBytes;
  uint64_t* bars = (uint64_t*)(sV + kStages * L::kKVBytes);
  uint64_t* bar_q = bars + 0;        // Q tile landed (TMA bytes); phase = row tile count
  uint64_t* q_free = bars + 1;       // the last S MMA of a row tile has read Q
  uint64_t* bar_s = bars + 2;        // [2] S of a key tile is in tensor memory; phase = (key tile count) >> 1
  uint64_t* bar_p = bars + 4;        // [2] the 128 rows of P are written (and S is read)
  uint64_t* bar_o = bars + 6;        // [2] PV of a key tile is done; phase = (key tile count) >> 1 (two in turn: the
                                     //     PVs of two tiles may be under way when a thread waits for the later)
  uint64_t* bar_drain = bars + 8;    // an aborted CTA waits here for its last MMAs
  uint64_t* bar_k = bars + 9;                  // [kStages] K stage landed; phase = (key tile count) / kStages
  uint64_t* bar_v = bar_k + kStages;           // [kStages] V stage landed
  uint64_t* k_free = bar_v + kStages;          // [kStages] the S MMA that read the stage is done
  uint64_t* v_free = k_free + kStages;         // [kStages] the PV MMA that read the stage is done
  uint64_t* bar_p1 = v_free + kStages;         // kLate: [2] the product of P's first term is done
  uint64_t* bar_p3 = bar_p1 + 2;               // kLate: [2] the 128 rows of the third term are written
  uint32_t* s_tmem = (uint32_t*)(bars + L::kBars);
  volatile int* s_abort = (volatile int*)(s_tmem + 1);
  int* s_ntiles = (int*)(s_tmem + 2);
  int* s_repeats = (int*)(s_tmem + 3);              // three-term: a query of the row tile lists a block more than once
  int* s_scan = (int*)(s_tmem + 4);                 // [129]
  uint32_t* s_member = (uint32_t*)(s_scan + 132);   // [nb_sel][n_sub][nw]   (selection only)
  const int tile_words = p.n_sub * p.nw;
  uint16_t* s_tiles = (uint16_t*)(s_member + (kSel ? p.nb_sel * tile_words : 0));

  if (kSel && p.plan != nullptr) chain_wait();    // the header is read first
  if (kSel && p.plan != nullptr && prefer_pairs(p.plan, p.nq_union, p.force))
    return;   // the block-outer variant serves this call: leave before anything is set up
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    *s_abort = (*(volatile int*)p.status != 0) ? 1 : 0;
    mbar_init(bar_q, 1);
    mbar_init(q_free, 1);
    for (int k = 0; k < 2; ++k) { mbar_init(bar_s + k, 1); mbar_init(bar_p + k, kFwdSoftmax); mbar_init(bar_o + k, 1); }
    mbar_init(bar_drain, 1);
    for (int k = 0; k < 4 * kStages; ++k) mbar_init(bar_k + k, 1);
    if (kLate)
      for (int k = 0; k < 2; ++k) { mbar_init(bar_p1 + k, 1); mbar_init(bar_p3 + k, kFwdSoftmax); }
    fence_barrier_init();
    prefetch_tensormap(&tm_q); prefetch_tensormap(&tm_k); prefetch_tensormap(&tm_v);
  }
  __syncthreads();
  if (*s_abort) { chain_wait(); return; }      // the kernels behind take its end for that of all before
  if (warp == 0) {
    tmem_alloc(s_tmem, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  if (kSel || kCmp) chain_wait();
  if (kCmp) chain_go();            // the scorer is next

  // row tile w of the launch: long rows first, the units of one token range next to each other
  const int units = p.B * p.Hkv;
  const int n_work = p.n_qtiles * units;
  struct Tile { int bh, t0, t_last, first_key, n_tiles; };
  auto tile_of = [&](int w) -> Tile {
    Tile x;
    x.bh = w % units;
    const int qtile = p.n_qtiles - 1 - w / units;
    x.t0 = qtile * p.nq;
    x.t_last = min(p.T - 1, x.t0 + p.nq - 1);
    x.first_key = 0;
    if (kSel) {
      x.n_tiles = *s_ntiles;
    } else if (!kCmp) {
      x.first_key = max(0, x.t0 - p.window + 1) & ~(kKeys - 1);
      x.n_tiles = (min(x.t_last, p.Lk - 1) - x.first_key) / kKeys + 1;
    } else {
      const int hi_last = cmp_visible(x.t_last, p.block_size, p.window, p.Lk) - 1;   // window: the stride
      x.n_tiles = hi_last < 0 ? 0 : hi_last / kKeys + 1;
    }
    return x;
  };
  auto key0_of = [&](const Tile& x, int i) -> int { return kSel ? (int)s_tiles[i] * kKeys : x.first_key + i * kKeys; };
  // the key tiles that hold a block listed by one of the row tile's queries, with a membership bit per
  // (query, list block)
  auto build_list = [&](int w) {
    const int bh = w % units, t0 = (p.n_qtiles - 1 - w / units) * p.nq, t_last = min(p.T - 1, t0 + p.nq - 1);
    const int n_vis = t_last / kKeys + 1;              // key tiles that start at or before the last query
    for (int i = tid; i < n_vis * tile_words; i += kFwdThreads) s_member[i] = 0u;
    if (kThreeTerm && tid == 0) *s_repeats = 0;
    __syncthreads();
    const int32_t* idx = p.block_idx + ((size_t)bh * p.T + t0) * p.S;
    const int n_entries = (t_last - t0 + 1) * p.S;
    for (int e = tid; e < n_entries; e += kFwdThreads) {
      const int q_local = e / p.S;
      const int blk = ld_plain(idx + e);
      // list block blk = part blk % n_sub of key tile blk / n_sub
      if (blk >= 0 && (long long)blk * p.block_size <= t0 + q_local) {
        const uint32_t was = atomicOr(&s_member[blk * p.nw + (q_local >> 5)], 1u << (q_local & 31));
        if (kThreeTerm && (was >> (q_local & 31) & 1u)) *s_repeats = 1;
      }
    }
    __syncthreads();
    const int per = (n_vis + 127) / 128;               // the first 128 threads scan `per` tiles each
    const int j0 = tid < 128 ? min(n_vis, tid * per) : n_vis, j1 = min(n_vis, j0 + per);
    int cnt = 0;
    for (int j = j0; j < j1; ++j) {
      uint32_t any = 0;
      for (int k = 0; k < tile_words; ++k) any |= s_member[j * tile_words + k];
      cnt += any != 0;
    }
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s_scan[warp] = incl;
    __syncthreads();
    int pos = incl - cnt;
    for (int k = 0; k < warp && k < 4; ++k) pos += s_scan[k];
    for (int j = j0; j < j1; ++j) {
      uint32_t any = 0;
      for (int k = 0; k < tile_words; ++k) any |= s_member[j * tile_words + k];
      if (any) s_tiles[pos++] = (uint16_t)j;
    }
    if (tid == 0) *s_ntiles = s_scan[0] + s_scan[1] + s_scan[2] + s_scan[3];
    __syncthreads();
  };

  int sent_k = 0, sent_v = 0, sent_q = 0;     // producer: loads sent so far (key tiles, row tiles)
  int c = 0, it = 0;                          // running counts of key tiles and of live row tiles
  bool ok = true;
  // softmax threads: row of a tile = thread index
  const int row = tid & (kFwdSoftmax - 1);
  const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const int ql = row / p.G, g = row % p.G;

  for (int w0 = blockIdx.x; w0 < n_work; w0 += kSel ? gridDim.x : n_work) {
    if (kSel) build_list(w0);
    const int w_end = kSel ? w0 + 1 : n_work;
    if (warp == 4) {
      // ---- producer -------------------------------------------------------------------------
      if (lane == 0) {
        for (int w = w0; ok && w < w_end; w += gridDim.x) {
          const Tile x = tile_of(w);
          if (x.n_tiles == 0) continue;
          const int b = x.bh / p.Hkv, hkv = x.bh % p.Hkv;
          if (it > 0) ok = mbar_wait(q_free, (it - 1) & 1, p.status, s_abort, 0x8000);
          if (!ok) break;
          mbar_expect_tx(bar_q, (uint32_t)(p.nq * p.G * 128 * kSlabs));
#pragma unroll
          for (int s = 0; s < kSlabs; ++s)
            tma_load_3d(sQ + s * (kRows * 128), &tm_q, bar_q, s * 64, b * p.Hq + hkv * p.G, x.t0);
          sent_q = ++it;
          for (int i = 0; i < x.n_tiles; ++i, ++c) {
            const int st = c % kStages, use = c / kStages, key0 = key0_of(x, i);
            // a stage is free once the MMAs of the tile kStages back, which read it, are done
            if (use > 0) ok = mbar_wait(k_free + st, (use - 1) & 1, p.status, s_abort, 0x4000);
            if (!ok) break;
            mbar_expect_tx(bar_k + st, L::kKVBytes);
#pragma unroll
            for (int s = 0; s < kSlabs; ++s)
              tma_load_3d(sK + st * L::kKVBytes + s * (kKeys * 128), &tm_k, bar_k + st, s * 64, key0, x.bh);
            sent_k = c + 1;
            if (use > 0) ok = mbar_wait(v_free + st, (use - 1) & 1, p.status, s_abort, 0x4000);
            if (!ok) break;
            if (!(p.debug_starve && c == 1)) {           // test only: this tile's wait has to run out
              mbar_expect_tx(bar_v + st, L::kKVBytes);
#pragma unroll
              for (int s = 0; s < kSlabs; ++s)
                tma_load_3d(sV + st * L::kKVBytes + s * (kKeys * 128), &tm_v, bar_v + st, s * 64, key0, x.bh);
              sent_v = c + 1;
            }
          }
        }
      }
    } else if (warp == 5) {
      // ---- MMA issuer ------------------------------------------------------------------------
      {
        const uint32_t lead = elect_one(), tmem_u = uniform(tmem);
        // Every wait is the whole warp's: the lanes come out of it together and with one answer.  A lane that fell two phases
        // behind the issuing one would wait for a parity that has come round, up to the limit.
        auto ready = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
          return __all_sync(0xffffffffu, mbar_wait(bar, parity, p.status, s_abort, code));
        };
        auto both = [&](uint64_t* a, uint32_t pa, int ca, uint64_t* b, uint32_t pb, int cb) -> bool {    // one vote
          return __all_sync(0xffffffffu, mbar_wait(a, pa, p.status, s_abort, ca) && mbar_wait(b, pb, p.status, s_abort, cb));
        };
        auto issue_s = [&](int cc, bool last) {   // S = Q K^T of running key tile cc
          const int st = cc % kStages;
          const uint32_t qa = desc_lo_kmajor(smem_u32(sQ)), ka = desc_lo_kmajor(smem_u32(sK + st * L::kKVBytes));
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t slab = kk >> 2, in = (kk & 3) * 32;
            mma_ss_by(lead, tmem_u + kColS + (cc & 1) * kKeys, desc_at(qa, slab * (kRows * 128) + in),
                   desc_at(ka, slab * (kKeys * 128) + in), kIdescQK, kk > 0);
          }
          tc_commit_by(lead, bar_s + (cc & 1));
          tc_commit_by(lead, k_free + st);
          if (last) tc_commit_by(lead, q_free);
        };
        for (int w = w0; ok && w < w_end; w += gridDim.x) {
          const Tile x = tile_of(w);
          if (x.n_tiles == 0) continue;
          ok = both(bar_q, it & 1, 1, bar_k + c % kStages, (c / kStages) & 1, 2);
          // An S MMA overwrites the P of two key tiles back: that tile's PV has to be complete (MMAs of
          // different shapes and operand sources are not ordered by their issue).  Here every earlier
          // one is waited for; the threads that write the last row tile's output wait for it as well.
          if (ok && c > 0) ok = ready(bar_o + ((c - 1) & 1), ((c - 1) >> 1) & 1, 0x2000);
          if (!ok) break;
          tc_fence_after();
          issue_s(c, x.n_tiles == 1);
          for (int i = 0; i < x.n_tiles; ++i, ++c) {
            if (i + 1 < x.n_tiles) {
              uint64_t* k_next = bar_k + (c + 1) % kStages;
              ok = i > 0 ? both(k_next, ((c + 1) / kStages) & 1, 2, bar_o + ((c - 1) & 1), ((c - 1) >> 1) & 1, 0x2000)
                         : ready(k_next, ((c + 1) / kStages) & 1, 2);
              if (!ok) break;
              tc_fence_after();
              issue_s(c + 1, i + 2 == x.n_tiles);
            }
            const int st = c % kStages;
            ok = both(bar_p + (c & 1), (c >> 1) & 1, 0x2000, bar_v + st, (c / kStages) & 1, 16);
            if (!ok) break;
            tc_fence_after();
            const uint32_t va = desc_lo_mnmajor(smem_u32(sV + st * L::kKVBytes), kKeys * 128);   // O (+)= P V
#pragma unroll
            for (int kk = 0; kk < kKeys / 16; ++kk)
              mma_ts_by(lead, tmem_u + kColO, tmem_u + kColS + (c & 1) * kKeys + kk * 8, desc_at(va, kk * 2048), kIdescPV, (i > 0) || (kk > 0));
            if (kThreeTerm) {
              if (kLate) tc_commit_by(lead, bar_p1 + (c & 1));
#pragma unroll
              for (int kk = 0; kk < kKeys / 16; ++kk)
                mma_ts_by(lead, tmem_u + kColO, tmem_u + kColS + (c & 1) * kKeys + 32 + kk * 8, desc_at(va, kk * 2048), kIdescPV, 1);
              if (kLate) {
                ok = ready(bar_p3 + (c & 1), (c >> 1) & 1, 0x2000);
                if (!ok) break;
                tc_fence_after();
              }
#pragma unroll
              for (int kk = 0; kk < kKeys / 16; ++kk)
                mma_ts_by(lead, tmem_u + kColO, tmem_u + kColP3 + (c & 1) * kP3Step + kk * 8, desc_at(va, kk * 2048), kIdescPV, 1);
            }
            tc_commit_by(lead, bar_o + (c & 1));
            tc_commit_by(lead, v_free + st);
          }
          ++it;
        }
      }
    } else {
      // ---- softmax: thread = row ---------------------------------------------------------------
      for (int w = w0; w < w_end; w += gridDim.x) {
        const Tile x = tile_of(w);
        const int t = x.t0 + ql;
        const bool row_ok = ql < p.nq && t < p.T;
        const int b = x.bh / p.Hkv, head = (x.bh % p.Hkv) * p.G + g;
        __nv_bfloat16* orow = p.o + ((size_t)(b * p.Hq + head) * p.T + t) * D;
        float* lrow = p.lse + (size_t)(b * p.Hq + head) * p.T + t;
        if (x.n_tiles == 0) {                       // rows without a key: zeros, no barrier is touched
          if (row_ok) {
            uint4* dst = reinterpret_cast<uint4*>(orow);
#pragma unroll
            for (int v4 = 0; v4 < D / 8; ++v4) dst[v4] = make_uint4(0, 0, 0, 0);
            *lrow = kLseEmpty;
          }
          continue;
        }
        float m_used = -INFINITY, l_sum = 0.f;      // log2 units
        bool listed = false;                        // three-term: the row attends a key
        const bool repeats = kThreeTerm && *s_repeats;
        for (int i = 0; i < x.n_tiles; ++i, ++c) {
          const int key0 = key0_of(x, i);
          // valid columns of this row in this tile: one range [lo, hi] and, for selection, 16-column groups
          int lo = 0, hi = -1;
          uint32_t groups = 0xfu;
          if (row_ok) {
            if (kSel) {
              hi = min(kKeys - 1, t - key0);
              const uint32_t* mem = s_member + (key0 / kKeys) * tile_words + (ql >> 5);
              if (p.n_sub == 1) {
                if (!((mem[0] >> (ql & 31)) & 1u)) hi = -1;
              } else {
                groups = 0u;
                for (int k = 0; k < p.n_sub; ++k)
                  if ((mem[k * p.nw] >> (ql & 31)) & 1u) groups |= ((1u << (p.block_size >> 4)) - 1u) << (k * (p.block_size >> 4));
              }
            } else if (!kCmp) {
              lo = max(0, t - p.window + 1 - key0);
              hi = min(kKeys - 1, t - key0);
            } else {
              hi = min(kKeys - 1, cmp_visible(t, p.block_size, p.window, p.Lk) - 1 - key0);
            }
            if (lo > hi) { lo = 0; hi = -1; }
          }
          ok = mbar_wait(bar_s + (c & 1), (c >> 1) & 1, p.status, s_abort, 4) && ok;
          if (!__all_sync(0xffffffffu, ok)) break;              // the whole warp leaves together
          tc_fence_after();
          const uint32_t s_base = lane_base + kColS + (c & 1) * kKeys;
          uint32_t r[64];
          tmem_ld32(s_base, r);
          tmem_ld32(s_base + 32, r + 32);
          tmem_wait_ld();
          // the running maximum is only raised when it grows by more than 8 powers of two
          float alpha = 1.f;
          bool rescale = false;
          uint32_t pk[32];
          // Masking is by select: what a row does not attend may be infinite or NaN.  A row that attends the
          // whole tile or none of it needs no work per element (none: its P is set to zero below); only
          // rows whose range ends inside the tile, or that attend some 16-column groups of it, do.
          const bool none = hi < 0;
          if (kThreeTerm) listed |= !none && groups != 0u;
          if (!(lo <= 0 && (hi >= kKeys - 1 || none) && (!kSel || groups == 0xfu))) {
            if (kSel) {
#pragma unroll
              for (int cc = 0; cc < 64; ++cc)
                if (cc < lo || cc > hi || !((groups >> (cc >> 4)) & 1u)) r[cc] = __float_as_uint(-INFINITY);
            } else {
              // a bit per column instead of two compares: 8 x 4096 tokens, 12 heads of 64, window 512: 126 -> 118 us (selection
              // masks few tiles and its extra registers cost as much: 400 -> 403)
              const uint64_t attended = none ? 0ull : (hi >= 63 ? ~0ull : (2ull << hi) - 1ull) >> lo << lo;
#pragma unroll
              for (int cc = 0; cc < 64; ++cc)
                if (!((uint32_t)(attended >> (cc & 32)) >> (cc & 31) & 1u)) r[cc] = __float_as_uint(-INFINITY);
            }
          }
          float tmax[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int cc = 0; cc < 64; ++cc) tmax[cc & 3] = fmaxf(tmax[cc & 3], __uint_as_float(r[cc]));
          // (the scale is positive: the largest scaled score is the scaled largest score)
          const float tm = none ? -INFINITY : fmaxf(fmaxf(tmax[0], tmax[1]), fmaxf(tmax[2], tmax[3])) * p.scale_log2;
          if (tm > m_used + 8.f) {                 // also the first finite maximum (m_used = -inf)
            if (m_used != -INFINITY) {
              alpha = ex2(m_used - tm);
              rescale = true;
              l_sum *= alpha;
            }
            m_used = tm;
          }
          const float msub = (m_used == -INFINITY) ? 0.f : m_used;
          const uint64_t nz2 = pack_f32x2(p.neg_zero, p.neg_zero);
          const uint64_t sc2 = pack_f32x2(p.scale_log2, p.scale_log2), mn2 = pack_f32x2(-msub, -msub);
          float psum = 0.f;
          float times[4] = {1.f, 1.f, 1.f, 1.f};     // how often the row's list names the block of a 16-column group
          if (kThreeTerm && repeats && !none) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              times[k] = (float)times_listed(p.block_idx + ((size_t)x.bh * p.T + t) * p.S, p.S, (key0 + 16 * k) / p.block_size);
          }
#pragma unroll
          for (int cc = 0; cc < 32; ++cc) {
            float p0, p1;
            unpack_f32x2(add_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[2 * cc]), __uint_as_float(r[2 * cc + 1])), sc2, nz2),
                                   mn2), p0, p1);
            p0 = ex2(p0);
            p1 = ex2(p1);
            if (kThreeTerm && repeats) {
              const float n = times[cc >> 3];
              p0 *= n;
              p1 *= n;
            }
            psum += p0 + p1;
            pk[cc] = pack_bf16(p0, p1);
            if (kThreeTerm) {                      // what the first term leaves, exactly
              r[2 * cc] = __float_as_uint(p0 - __uint_as_float(pk[cc] << 16));
              r[2 * cc + 1] = __float_as_uint(p1 - __uint_as_float(pk[cc] & 0xffff0000u));
            }
          }
          if (none) {
            psum = 0.f;
#pragma unroll
            for (int cc = 0; cc < 32; ++cc) pk[cc] = 0u;
            if (kThreeTerm)
#pragma unroll
              for (int cc = 0; cc < 64; ++cc) r[cc] = 0u;
          }
          l_sum += psum;
          if constexpr (kThreeTerm) {              // (before the rescaling below needs the registers)
            tmem_st32(s_base, pk);
#pragma unroll
            for (int cc = 0; cc < 32; ++cc) {
              pk[cc] = pack_bf16(__uint_as_float(r[2 * cc]), __uint_as_float(r[2 * cc + 1]));
              r[2 * cc] = __float_as_uint(__uint_as_float(r[2 * cc]) - __uint_as_float(pk[cc] << 16));
              r[2 * cc + 1] = __float_as_uint(__uint_as_float(r[2 * cc + 1]) - __uint_as_float(pk[cc] & 0xffff0000u));
            }
            tmem_st32(s_base + 32, pk);
#pragma unroll
            for (int cc = 0; cc < 32; ++cc) pk[cc] = pack_bf16(__uint_as_float(r[2 * cc]), __uint_as_float(r[2 * cc + 1]));
            if (!kLate) tmem_st32(lane_base + kColP3 + (c & 1) * kP3Step, pk);
          }
          // O may be touched once PV of the tile before is done; only a warp that has to rescale waits
          if (i > 0 && __any_sync(0xffffffffu, rescale)) {
            ok = mbar_wait(bar_o + ((c - 1) & 1), ((c - 1) >> 1) & 1, p.status, s_abort, 8);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after();
#pragma unroll
            for (int cc = 0; cc < D / 32; ++cc) {
              uint32_t o32[32];
              tmem_ld32(lane_base + kColO + cc * 32, o32);
              tmem_wait_ld();
#pragma unroll
              for (int e = 0; e < 32; ++e) o32[e] = __float_as_uint(__uint_as_float(o32[e]) * alpha);
              tmem_st32(lane_base + kColO + cc * 32, o32);
            }
          }
          if (!kThreeTerm) tmem_st32(s_base, pk);  // over the S columns this thread has just read
          tmem_wait_st();
          tc_fence_before();
          mbar_arrive(bar_p + (c & 1));
          if constexpr (kLate) {
            ok = mbar_wait(bar_p1 + (c & 1), (c >> 1) & 1, p.status, s_abort, 8);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after();
            tmem_st32(lane_base + kColP3 + (c & 1) * kP3Step, pk);
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(bar_p3 + (c & 1));
          }
        }
        if (!__all_sync(0xffffffffu, ok)) break;
        // ---- this row tile's output: the last PV, then O / l -------------------------------------
        ok = mbar_wait(bar_o + ((c - 1) & 1), ((c - 1) >> 1) & 1, p.status, s_abort, 8);
        if (!__all_sync(0xffffffffu, ok)) break;
        tc_fence_after();
        const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
        float nan_sum = 0.f;                         // x * 0: 0 or NaN
#pragma unroll
        for (int cc = 0; cc < D / 32; ++cc) {
          uint32_t o32[32];
          tmem_ld32(lane_base + kColO + cc * 32, o32);
          tmem_wait_ld();
          if (kThreeTerm)
#pragma unroll
            for (int e = 0; e < 32; ++e) nan_sum = fmaf(__uint_as_float(o32[e]), 0.f, nan_sum);
          if (row_ok) {
            uint4* dst = reinterpret_cast<uint4*>(orow + cc * 32);
#pragma unroll
            for (int v4 = 0; v4 < 4; ++v4) {
              uint4 u;
              u.x = pack_bf16(__uint_as_float(o32[v4 * 8 + 0]) * inv, __uint_as_float(o32[v4 * 8 + 1]) * inv);
              u.y = pack_bf16(__uint_as_float(o32[v4 * 8 + 2]) * inv, __uint_as_float(o32[v4 * 8 + 3]) * inv);
              u.z = pack_bf16(__uint_as_float(o32[v4 * 8 + 4]) * inv, __uint_as_float(o32[v4 * 8 + 5]) * inv);
              u.w = pack_bf16(__uint_as_float(o32[v4 * 8 + 6]) * inv, __uint_as_float(o32[v4 * 8 + 7]) * inv);
              if (l_sum > 0.f) dst[v4] = u; else dst[v4] = make_uint4(0, 0, 0, 0);
            }
          }
        }
        if (row_ok) *lrow = l_sum > 0.f ? (m_used + log2f(l_sum)) * kLn2 : kLseEmpty;
        if (kThreeTerm && row_ok && listed && !(nan_sum == 0.f && l_sum > 0.f && l_sum < INFINITY))
          sel_row_forward<D>(p.q + ((size_t)(b * p.Hq + head) * p.T + t) * D, p.k + (size_t)x.bh * p.Lk * D,
                             p.v + (size_t)x.bh * p.Lk * D, p.block_idx + ((size_t)x.bh * p.T + t) * p.S, p.S, p.block_size,
                             t, p.scale_log2, orow, lrow);
        tc_fence_before();     // the O columns are read: the next row tile's first PV (behind this thread's next P) may overwrite them
      }
    }
    // the row tile's list may be overwritten once every role is through with it
    if (kSel && __syncthreads_or(*s_abort)) break;
  }
  if (warp == 5) {
    // the tensor pipe is idle before tensor memory is given back, whatever happened
    tc_commit_by(elect_one(), bar_drain);
    if (!mbar_wait(bar_drain, 0, p.status, s_abort, 0x1000)) mbar_wait_drain(bar_drain, 0);
  }

  // ---- teardown -------------------------------------------------------------------------------
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*s_abort) {
    // Give-up path: nothing more is written.  The producer waits (bounded) for the loads still on
    // their way into this CTA's shared memory; the MMA thread has waited for the tensor pipe above.
    if (warp == 4 && lane == 0) {
      if (sent_q > 0) mbar_wait_drain(bar_q, (sent_q - 1) & 1);
      for (int k = max(0, sent_k - kStages); k < sent_k; ++k) mbar_wait_drain(bar_k + k % kStages, (k / kStages) & 1);
      for (int k = max(0, sent_v - kStages); k < sent_v; ++k)
        if (!(p.debug_starve && k == 1)) mbar_wait_drain(bar_v + k % kStages, (k / kStages) & 1);
    }
    __syncthreads();
  }
  if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

static const char* const kFwdNames[3] = {"tc_fwd_win", "tc_fwd_cmp", "tc_fwd_slc"};

}  // namespace tc

bool tc_shape_ok(const NsaDims& d, int block_size) {
  if (d.dtype != NSA_DTYPE_BF16) return false;
  if (d.D != 64 && d.D != 128) return false;
  if (block_size != 16 && block_size != 32 && block_size != tc::kKeys) return false;   // whole 16-column groups of a key tile
  const int G = d.Hq / d.Hkv;
  if (G < 2 || G > 128) return false;   // the backward tiles hold at most 64 queries
  if (d.T < 1) return false;
  const int nq = tc::kRows / G;
  const int nb = (d.T + tc::kKeys - 1) / tc::kKeys;
  if (nb > 65535) return false;
  if (tc::fwd_smem_bytes(d.D, nb, (nq + 31) / 32, tc::kKeys / block_size, 2) > 224 * 1024) return false;
  return true;
}

int get_option_debug_starve_load();   // api.cu

static int launch_fwd(const AttnArgs& a, const SelPlanHeader* plan, int force, cudaStream_t st) {
  using namespace tc;
  FwdArgs p;
  p.plan = plan; p.force = force; p.nq_union = kRows / group_pad(a.Hq / a.Hkv);
  p.debug_starve = get_option_debug_starve_load();
  p.block_idx = a.block_idx;
  p.o = (__nv_bfloat16*)a.o;
  p.lse = a.lse;
  p.status = device_status_ptr();
  if (!p.status) { set_error("device status word unavailable"); return NSA_ERR_CUDA; }
  p.B = a.B; p.Hq = a.Hq; p.Hkv = a.Hkv; p.T = a.T; p.Lk = a.Lk; p.S = a.S;
  p.G = a.Hq / a.Hkv;
  p.nq = kRows / p.G;
  p.kind = a.kind; p.window = a.window; p.block_size = a.block_size;
  p.n_qtiles = (a.T + p.nq - 1) / p.nq;
  p.nb_sel = (a.T + kKeys - 1) / kKeys;
  p.nw = (p.nq + 31) / 32;
  p.n_sub = a.kind == 2 ? kKeys / a.block_size : 1;
  p.scale_log2 = a.scale * kLog2e;
  p.neg_zero = -0.f;
  p.q = (const __nv_bfloat16*)a.q; p.k = (const __nv_bfloat16*)a.k; p.v = (const __nv_bfloat16*)a.v;
  CUtensorMap tm_q, tm_k, tm_v;
  int rc = make_map_query_rows(&tm_q, a.q, a.D, a.T, a.B * a.Hq, p.G, p.nq);
  if (rc == NSA_OK) rc = make_map(&tm_k, a.k, a.D, a.Lk, a.B * a.Hkv, kKeys, 1);
  if (rc == NSA_OK) rc = make_map(&tm_v, a.v, a.D, a.Lk, a.B * a.Hkv, kKeys, 1);
  if (rc != NSA_OK) return rc;
  const size_t smem = fwd_smem_bytes(a.D, p.nb_sel, p.nw, p.n_sub, a.kind);
  // persistent CTAs, two per SM, each walking its share of the row tiles
  const long long n_work = (long long)p.n_qtiles * a.B * a.Hkv;
  if (n_work == 0) return NSA_OK;
  NSA_CHECK_ARG(n_work < (1LL << 31), "too many row tiles");
  const unsigned grid = (unsigned)std::min<long long>(n_work, 2LL * sm_count());
  KernelScope ks(branch_name(kFwdNames, a.kind), st);
  auto go = [&](auto kernel) -> int {
    NSA_CUDA_OK(func_smem((const void*)kernel, smem));
    if (a.kind == 2 || a.chained)          // behind scorer, plan or pooling
      NSA_CUDA_OK(launch_chained(kernel, grid, kFwdThreads, smem, st, tm_q, tm_k, tm_v, p));
    else kernel<<<grid, kFwdThreads, smem, st>>>(tm_q, tm_k, tm_v, p);
    return NSA_OK;
  };
  if (a.three_term)
    rc = a.D == 128 ? go(tc_fwd_kernel<128, 2, true>) : go(tc_fwd_kernel<64, 2, true>);
  else if (a.D == 128)
    rc = a.kind == 2 ? go(tc_fwd_kernel<128, 2, false>) : a.kind == 1 ? go(tc_fwd_kernel<128, 1, false>) : go(tc_fwd_kernel<128, 0, false>);
  else
    rc = a.kind == 2 ? go(tc_fwd_kernel<64, 2, false>) : a.kind == 1 ? go(tc_fwd_kernel<64, 1, false>) : go(tc_fwd_kernel<64, 0, false>);
  if (rc != NSA_OK) return rc;
  NSA_LAUNCH_OK("tc_fwd_kernel");
  return NSA_OK;
}

int tc_attn_fwd(const AttnArgs& a, cudaStream_t st) { return launch_fwd(a, nullptr, 0, st); }

int tc_fwd_union_launch(const AttnArgs& a, const SelPlanHeader* plan, int force, cudaStream_t st) {
  return launch_fwd(a, plan, force, st);
}

}  // namespace nsa
