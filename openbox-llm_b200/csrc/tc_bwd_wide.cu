// tcgen05 backward of the window branch on tiles of 128 keys.
//
// A tcgen05.mma of 128 x 64 x 16 takes as long as one of 128 x 128 x 16 (70 cycles against 65; an operand tile of 128 rows
// is fetched for either), so the tiles of 64 keys that selection blocks ask for leave half of the tensor pipe unused.  The
// window's keys are ranges and can have 128 a tile.  With keys on the TMEM lanes P stays out of shared memory:
//   S^T  = K Q^T            (A: K  K-major,  B: Q  K-major)       keys x rows
//   dP^T = V dO^T           (A: V  K-major,  B: dO K-major)
//   dV  += P^T dO           (A: P^T in TMEM, B: dO MN-major)
//   dK  += dS^T Q           (A: dS K-major from shared memory, B: Q MN-major)
//   dQ   = dS K             (A: dS MN-major, B: K MN-major), only the 16-key steps that the row tile attends
// p = exp2(s * scale * log2e - lse * log2e + log2(gate)) and dS = p * (dP - delta) * scale of a (key, row) are computed
// by the thread of the key's lane; lse and delta of the rows are subtracted by one more step of each product.  One CTA
// has a key tile of one (batch, kv head); dK and dV stay in TMEM until the end and leave as rows; dQ of every row tile
// leaves as a bf16 partial tile, one per 128 keys (dq_reduce3_kernel adds them up): 5 a query for a window of 512
// where tiles of 64 keys leave 9.
// Roles: eight compute warps (two per TMEM lane quadrant, half of the rows each), four dQ warps, one warp each for Q,
// dO, the row statistics and the MMAs.  Each hand-over is an mbarrier with a bounded wait.
//
// What is not finite: a V stays with the rows that attend its key, a row of dO (or its delta) or Q reaches dK and dV of the key
// tiles that its query attends, a K dQ of the rows that share one of its steps of 16 keys: 0 x inf in a product is NaN.
//
// What bounds it: at D = 128 the chain S -> p -> dP -> dS of one row tile, whose S and dP fill what TMEM dV and dK leave
// (4.8 k cycles a row tile, the MMAs alone 2.7 k); at D = 64 the MMAs (4.2 k against 2.2 k by themselves, 33 of them: the warp that
// issues them shares its scheduler with compute warps, and their operands share shared memory with dS and the tiles
// going in and out).  8 x 32768 tokens, 16 heads of 128, window 512: 3.6 ms, 5.2 with tiles of 64 keys; 8 x 4096, 12 heads
// of 64: 267 us, 428.
#include <type_traits>

#include "tc_bwd_wide.cuh"
#include "tc_host.cuh"

namespace nsa {
namespace tc {

constexpr int kWideThreads = 512;

template <int D> struct Wide {
  static constexpr int kSlabs = D / 64;
  static constexpr int kStages = D == 64 ? 3 : 2;                 // Q / dO tiles in shared memory
  static constexpr int kKVBytes = kWideKeys * 128 * kSlabs;
  static constexpr int kRowBytes = kRows * 128 * kSlabs;          // Q or dO
  static constexpr int kSlabBytes = 128 * 128;                    // 64 columns of any tile here
  static constexpr int kDsTiles = D == 64 ? 2 : 1;                // dS tiles
  static constexpr int kDsBytes = 2 * kSlabBytes;                 // 128 keys x 128 rows
  // dQ on its way out: at D = 128 over dS, which its MMA has read; at D = 64 a tile of its own
  static constexpr bool kOwnStage = D == 64;
  static constexpr int kStageOut = kOwnStage ? kRowBytes : 0;
  // dQ columns of their own, or over dP
  static constexpr bool kOwnDq = D == 64;
  static constexpr uint32_t kColS = 0, kColDP = 128, kColDV = 256, kColDK = kColDV + D, kColDQ = kOwnDq ? kColDK + D : kColDP;
  // P^T of rows 0-63 and 64-127: columns of their own, or over the first of each half of S^T
  static constexpr bool kOwnP = D == 64;
  static constexpr uint32_t kColP = kOwnP ? kColDQ + D : kColS, kStepP = kOwnP ? 32 : 64;
  static constexpr int kStats = D == 64 ? 4 : 1;                  // row statistics: ring of lse(0), delta(0), lse(1), ...
  static constexpr int kStatBytes = kRows * 16;                   // a row: three bf16 terms of the value, zeros
  static constexpr int kBarS = 2 + 4 * kStages, kBars = kBarS + 7 + kDsTiles + 2 * kStats;
  static constexpr int kOffDs = 2 * kKVBytes + kStages * 2 * kRowBytes, kOffBars = kOffDs + kDsTiles * kDsBytes + kStageOut + kStats * kStatBytes + 256;
  static constexpr size_t kSmem = 2 * kKVBytes + (size_t)kStages * 2 * kRowBytes + kDsTiles * kDsBytes + kStageOut + kStats * kStatBytes +
                                  256 /*ones*/ + 256 /*barriers*/ + 512 /*alignment slack*/;
};

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// two products in one instruction
__device__ __forceinline__ void mul_f32x2(uint32_t a0, uint32_t a1, float b0, float b1, float& x0, float& x1) {
  uint64_t a, b, x;
  asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "r"(a0), "r"(a1));
  asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(b0), "f"(b1));
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(x) : "l"(a), "l"(b));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x0), "=f"(x1) : "l"(x));
}
__device__ __forceinline__ void st_shared_16b(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// barrier of `threads` threads that gives every one of them the same answer on whether any brought a non-zero `pred`
__device__ __forceinline__ bool group_or(int id, int threads, int pred) {
  uint32_t out;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %3, 0;\n\t"
      "bar.red.or.pred p, %1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(out)
      : "r"(id), "r"(threads), "r"(pred)
      : "memory");
  return out != 0;
}

// The compute warps' work of a CTA by select: what a key is not attended by may be infinite or NaN.  `smem` and `bars` as in the
// kernel below.  Not inlined, so that the registers and the schedule of the usual loop stay what they are: as a second form of its
// body, 8 x 4096 tokens of 12 heads of 64 took 295 us instead of 270, with checks in it 327.
template <int D>
__device__ __noinline__ void masked_row_tiles(const WideArgs& p, uint8_t* smem, uint32_t tmem) {
  using L = Wide<D>;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBars);
  uint64_t *s_full = bars + L::kBarS, *dp_full = s_full + 1, *p_full = dp_full + 1, *ds_full = p_full + 1, *ds_free = ds_full + 3;
  uint64_t* dv_done = ds_free + L::kDsTiles;
  volatile int* s_abort = reinterpret_cast<volatile int*>(reinterpret_cast<uint32_t*>(bars + L::kBars) + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3, half = warp >> 2;
  const int key0 = blockIdx.x * kWideKeys, kr = quad * 32 + lane, key = key0 + kr;
  const int n_q = min(p.T - 1, key0 + kWideKeys - 1 + p.window - 1) - key0 + 1, n_tiles = (n_q + p.nq - 1) / p.nq;
  const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16) + half * 64;
  const uint32_t p_base = tmem + ((uint32_t)(quad * 32) << 16) + L::kColP + half * L::kStepP;
#pragma unroll 1
  for (int k = 0; k < n_tiles; ++k) {
    const int qi0 = k * p.nq, to_key = key - key0 - qi0;             // queries from the tile's first to the key
    const uint32_t ds_row = smem_u32(smem + L::kOffDs) + k % L::kDsTiles * L::kDsBytes + half * L::kSlabBytes + kr * 128;
    const int lo = min(max(to_key, 0), p.nq) * p.G, hi = key >= p.T ? 0 : min(min(p.nq, n_q - qi0), to_key + p.window) * p.G;
    const int lo_h = min(max(lo - half * 64, 0), 64), hi_h = min(max(hi - half * 64, 0), 64);
    const uint64_t upto = hi_h == 64 ? ~0ull : (1ull << hi_h) - 1ull;
    const uint64_t attended = lo_h == 64 ? 0ull : upto >> lo_h << lo_h;
    bool ok = mbar_wait(s_full, k & 1, p.status, s_abort, 64);
    if (ok && L::kOwnP && k > 0) ok = mbar_wait(dv_done, (k - 1) & 1, p.status, s_abort, 64);
    if (!__all_sync(0xffffffffu, ok)) return;                // the whole warp leaves together
    tc_fence_after();
    uint32_t pr[64];
    tmem_ld32(lane_base + L::kColS, pr);
    tmem_ld32(lane_base + L::kColS + 32, pr + 32);
    tmem_wait_ld();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t in = (uint32_t)(attended >> (h * 32));
      uint32_t pk[16];
#pragma unroll
      for (int c2 = 0; c2 < 16; ++c2) {
#pragma unroll
        for (int c = h * 32 + c2 * 2; c < h * 32 + c2 * 2 + 2; ++c)
          pr[c] = in >> (c & 31) & 1u ? __float_as_uint(ex2(__uint_as_float(pr[c]) * p.scale_log2)) : 0u;
        pk[c2] = pack_bf16(__uint_as_float(pr[h * 32 + c2 * 2]), __uint_as_float(pr[h * 32 + c2 * 2 + 1]));
      }
      tmem_st16(p_base + h * 16, pk);
    }
    tmem_wait_st();
    tc_fence_before();
    mbar_arrive(p_full);
    ok = mbar_wait(dp_full, k & 1, p.status, s_abort, 64);
    if (ok && k >= L::kDsTiles) ok = mbar_wait(ds_free + k % L::kDsTiles, (k / L::kDsTiles - 1) & 1, p.status, s_abort, 64);
    if (!__all_sync(0xffffffffu, ok)) return;
    tc_fence_after();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t in = (uint32_t)(attended >> (h * 32));
      uint32_t dp[32];
      tmem_ld32(lane_base + L::kColDP + h * 32, dp);
      tmem_wait_ld();
#pragma unroll
      for (int c = 0; c < 32; ++c)
        dp[c] = in >> c & 1u ? __float_as_uint(__uint_as_float(pr[h * 32 + c]) * (__uint_as_float(dp[c]) * p.scale)) : 0u;
#pragma unroll
      for (int v4 = 0; v4 < 4; ++v4) {
        uint32_t b[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) b[e] = pack_bf16(__uint_as_float(dp[v4 * 8 + e * 2]), __uint_as_float(dp[v4 * 8 + e * 2 + 1]));
        st_shared_16b(ds_row + ((uint32_t)((h * 4 + v4) ^ (kr & 7)) << 4), b[0], b[1], b[2], b[3]);
      }
    }
    fence_proxy_async();
    tc_fence_before();
    mbar_arrive(ds_full);
  }
}

template <int D>
__global__ void __launch_bounds__(kWideThreads, 1)
tc_bwd_wide_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                   const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                   const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ WideArgs p) {
  using L = Wide<D>;
  constexpr int kSlabs = L::kSlabs, kStages = L::kStages, kSlabBytes = L::kSlabBytes;
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kIdescS = idesc_bf16(128, 128, 0, 0), kIdescT = idesc_bf16(128, D, 0, 1), kIdescDQ = idesc_bf16(128, D, 1, 1);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sK = smem;
  uint8_t* sV = sK + L::kKVBytes;
  uint8_t* sRow = sV + L::kKVBytes;               // [kStages] dO, Q
  uint8_t* sDs = sRow + kStages * 2 * L::kRowBytes;   // [kDsTiles] two slabs of 64 rows, a key per 128 bytes
  uint8_t* sOut = L::kOwnStage ? sDs + L::kDsTiles * L::kDsBytes : sDs;
  uint8_t* sStat = sDs + L::kDsTiles * L::kDsBytes + L::kStageOut;  // [kStats]
  uint8_t* sOnes = sStat + L::kStats * L::kStatBytes; // eight rows of 1, 1, 1, 0, 0, 0, 0, 0; eight of zeros
  uint64_t* bars = reinterpret_cast<uint64_t*>(sOnes + 256);
  uint64_t* bar_kv = bars + 0;
  uint64_t* bar_drain = bars + 1;
  uint64_t* do_full = bars + 2;                   // [kStages] dO has landed
  uint64_t* q_full = do_full + kStages;           // [kStages] Q has landed
  uint64_t* do_free = q_full + kStages;           // [kStages] the dV and dP MMAs are done
  uint64_t* q_free = do_free + kStages;           // [kStages] the dK MMAs are done
  uint64_t* s_full = bars + L::kBarS;             // S^T is in TMEM
  uint64_t* dp_full = s_full + 1;                 // dP^T is in TMEM
  uint64_t* p_full = dp_full + 1;                 // P^T is in TMEM (256 arrivals)
  uint64_t* ds_full = p_full + 1;                 // dS is in shared memory, dP has been read (256 arrivals)
  uint64_t* acc_full = ds_full + 1;               // the tile's MMAs are done: dQ is in TMEM, dS has been read
  uint64_t* dq_read = acc_full + 1;               // dQ has left TMEM (128 arrivals)
  uint64_t* ds_free = dq_read + 1;                // [kDsTiles] the MMAs have read dS and, at D = 128, dQ has left its tile
  uint64_t* dv_done = ds_free + L::kDsTiles;               // the dV MMAs have read P^T: S^T may be written again
  uint64_t* stat_full = dv_done + 1;              // [kStats] the statistics are written (32 arrivals)
  uint64_t* stat_free = stat_full + L::kStats;    // [kStats] the MMAs have read them
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + L::kBars);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
  static_assert(L::kBars * 8 + 8 <= 256, "barrier region");

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int j = blockIdx.x, bh = blockIdx.y;
  const int b = bh / p.Hkv, hkv = bh % p.Hkv;
  const int key0 = j * kWideKeys;
  const int head0 = b * p.Hq + hkv * p.G;

  // the queries that attend this key tile: n_q from t_lo, nq of them a row tile
  const int window = p.window, t_lo = key0;
  const int n_q = min(p.T - 1, key0 + kWideKeys - 1 + window - 1) - t_lo + 1;
  const int n_tiles = (n_q + p.nq - 1) / p.nq;

  if (tid == 0) {
    int bad = (*(volatile int*)p.status != 0) ? 1 : 0;
    if ((size_t)((uint8_t*)(bars + 32) - smem_raw) > L::kSmem) {
      atomicOr(p.status, 256);   // the shared-memory window is less aligned than assumed
      bad = 1;
    }
    *s_abort = bad;
    mbar_init(bar_kv, 1);
    mbar_init(bar_drain, 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(do_full + s, 1); mbar_init(q_full + s, 1); mbar_init(do_free + s, 1); mbar_init(q_free + s, 1);
    }
    mbar_init(s_full, 1); mbar_init(dp_full, 1); mbar_init(p_full, 256); mbar_init(ds_full, 256);
    mbar_init(acc_full, 1); mbar_init(dq_read, 128); mbar_init(dv_done, 1);
    for (int s = 0; s < L::kDsTiles; ++s) mbar_init(ds_free + s, 1);
    for (int s = 0; s < L::kStats; ++s) { mbar_init(stat_full + s, 32); mbar_init(stat_free + s, 1); }
    fence_barrier_init();
  } else if (tid == 32) {
    prefetch_tensormap(&tm_k); prefetch_tensormap(&tm_v);
    prefetch_tensormap(&tm_q); prefetch_tensormap(&tm_do); prefetch_tensormap(&tm_dq);
  }
  __syncthreads();
  if (*s_abort) return;
  const uint32_t tile_bytes = (uint32_t)(p.nq * p.G * 128 * kSlabs);     // of Q or dO
  // everything up to the loads of the first tiles overlaps with them
  if (warp == 12 && lane == 0) {
    mbar_expect_tx(bar_kv, 2 * L::kKVBytes);
#pragma unroll
    for (int s = 0; s < kSlabs; ++s) tma_load_3d(sK + s * kSlabBytes, &tm_k, bar_kv, s * 64, key0, bh);
  } else if (warp == 15 && lane == 0) {
#pragma unroll
    for (int s = 0; s < kSlabs; ++s) tma_load_3d(sV + s * kSlabBytes, &tm_v, bar_kv, s * 64, key0, bh);
  }
  uint32_t tmem = 0;
  if (warp < 12 || warp == 14) {
    // rows past nq * G of a Q / dO tile are never loaded, and dV / dK sum over all 128: keep them zero
    if (warp < 12) {
      const int r0 = p.nq * p.G, n = (kRows - r0) * 8;
      for (int i = tid; i < 2 * kSlabs * kStages * n; i += 12 * 32)
        *reinterpret_cast<uint4*>(sRow + (i / n) * kSlabBytes + r0 * 128 + (i % n) * 16) = make_uint4(0, 0, 0, 0);
      if (tid < 16) *reinterpret_cast<uint4*>(sOnes + tid * 16) = tid < 8 ? make_uint4(0x3f803f80u, 0x3f80u, 0, 0) : make_uint4(0, 0, 0, 0);
      fence_proxy_async();
    }
    if (warp == 0) {
      tmem_alloc(s_tmem, kTmemCols);
      tmem_relinquish();
    }
    tc_fence_before();
    asm volatile("bar.sync 2, 416;" ::: "memory");         // warps 0-11 and 14
    tc_fence_after();
    tmem = *s_tmem;
  }

  if (warp == 12 || warp == 15) {
    // ---- producers: the Q or dO rows of every tile, consecutive tokens: one box per slab -------------
    const bool is_q = warp == 12;
    uint64_t *full = is_q ? q_full : do_full, *free = is_q ? q_free : do_free;
    int issued = 0;
    if (lane == 0) {
      for (int k = 0; k < n_tiles; ++k) {
        const int st = k % kStages, u = k / kStages;
        if (u > 0 && !mbar_wait(free + st, (u - 1) & 1, p.status, s_abort, 128)) break;
        mbar_expect_tx(full + st, tile_bytes);
        uint8_t* dst = sRow + (2 * st + (is_q ? 1 : 0)) * L::kRowBytes;
#pragma unroll
        for (int s = 0; s < kSlabs; ++s)
          tma_load_3d(dst + s * kSlabBytes, is_q ? &tm_q : &tm_do, full + st, s * 64, head0, t_lo + k * p.nq);
        issued = k + 1;
      }
      // the loads land (bounded wait) before the teardown barrier, whether the CTA has given up or gives up later
      mbar_wait_drain(bar_kv, 0);
      for (int k = max(0, issued - kStages); k < issued; ++k) mbar_wait_drain(full + k % kStages, (k / kStages) & 1);
    }
  } else if (warp == 13) {
    // ---- row statistics of every tile: lse for S, delta for dP, as the terms that one more step of 16 adds to the
    // product: S - lse / (scale log2e) and dP - delta come out of the MMAs (24 bits of the value in three bf16 terms).
    // A lane has a key, so the compute warps would have to get 256 numbers dealt out per tile: loads from shared
    // memory wait behind the operands of the MMAs, which take all of its bandwidth, and shuffles are no faster ---------
    int use = 0;
    auto terms = [](float x) -> uint2 {
      const uint32_t h = pack_bf16(x, 0.f) & 0xffffu;
      const float r1 = x - __uint_as_float(h << 16);
      const bool finite = r1 == r1;                  // what an infinite value leaves is NaN
      const uint32_t m = pack_bf16(finite ? r1 : 0.f, 0.f) & 0xffffu;
      return make_uint2(h | (m << 16), pack_bf16(finite ? r1 - __uint_as_float(m << 16) : 0.f, 0.f));
    };
    auto write = [&](const uint2* x) -> bool {
      const int slot = use % L::kStats, u = use / L::kStats;
      const bool ok = u == 0 || mbar_wait(stat_free + slot, (u - 1) & 1, p.status, s_abort, 128);
      if (!__all_sync(0xffffffffu, ok)) return false;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        st_shared_16b(smem_u32(sStat + slot * L::kStatBytes) + (i * 32 + lane) * 16, x[i].x, x[i].y, 0u, 0u);
      fence_proxy_async();
      mbar_arrive(stat_full + slot);
      ++use;
      return true;
    };
    int ql[4];
    size_t at0[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = i * 32 + lane;
      ql[i] = r / p.G;
      at0[i] = (size_t)(head0 + r % p.G) * p.T + t_lo + ql[i];
      if (ql[i] >= p.nq) ql[i] = 1 << 30;
    }
    float lse[4], delta[4], gate[4];
    auto fetch = [&](int k) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int q0 = k * p.nq;
        const bool ok = ql[i] < n_q - q0;
        const size_t at = at0[i] + q0;
        lse[i] = ok ? ldg_f32_now(p.lse + at) : 0.f;
        delta[i] = ok ? ldg_f32_now(p.delta + at) : 0.f;
        gate[i] = ok && p.row_scale ? ldg_f32_now(p.row_scale + at) : 1.f;
      }
    };
    fetch(0);
    for (int k = 0; k < n_tiles; ++k) {
      uint2 ls[4], dd[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // gate * p = 2^(s * scale * log2e - lse * log2e + log2(gate)): the branch's dO is gate * dO
        float x = (__log2f(gate[i]) - lse[i] * kLog2e) / p.scale_log2;
        if (x < -1e30f) x = -1e30f;                // a gate of 0: p is 0
        ls[i] = terms(x);
        dd[i] = terms(-delta[i]);
      }
      if (!write(ls) || !write(dd)) break;
      if (k + 1 < n_tiles) fetch(k + 1);         // (behind the fences, which wait for loads under way)
    }
  } else if (warp == 14) {
    // ---- MMA issuer --------------------------------------------------------------------------
    {
      const uint32_t lead = elect_one(), tmem_u = uniform(tmem);
      const uint32_t ka = desc_lo_kmajor(smem_u32(sK)), va = desc_lo_kmajor(smem_u32(sV));
      const uint32_t kb = desc_lo_mnmajor(smem_u32(sK), kSlabBytes);
      auto ds_tile = [&](int k) -> uint32_t { return smem_u32(sDs + k % L::kDsTiles * L::kDsBytes); };
      auto row_tile = [&](int k, int which) -> uint32_t { return smem_u32(sRow + (2 * (k % kStages) + which) * L::kRowBytes); };
      auto ready = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
        return __all_sync(0xffffffffu, mbar_wait(bar, parity, p.status, s_abort, code));
      };
      // no swizzle: groups of 8 rows x 16 bytes, the statistics' one behind the other, the ones' the same for all rows; the
      // second half of a step of 16 is zeros there and reads the first half again here (so that an infinite delta comes out NaN)
      auto plain = [](const void* t, uint32_t lbo_bytes, uint32_t sbo_bytes) -> uint64_t {
        return (uint64_t)((smem_u32(t) >> 4) & 0x3fffu) | (uint64_t)(lbo_bytes >> 4) << 16 | (uint64_t)(sbo_bytes >> 4) << 32 | 1ull << 46;
      };
      const uint64_t ones = plain(sOnes, 128, 0);
      auto stat_tile = [&](int use) -> uint64_t { return plain(sStat + use % L::kStats * L::kStatBytes, 0, 128); };
      auto stat_ready = [&](int use) -> bool { return ready(stat_full + use % L::kStats, (use / L::kStats) & 1, 512); };
      auto issue_s = [&](int k) -> bool {
        // (MMAs of different shapes and operand sources are not ordered by their issue)
        if (!ready(q_full + k % kStages, (k / kStages) & 1, 512) || (!L::kOwnP && k > 0 && !ready(dv_done, (k - 1) & 1, 64)) ||
            !stat_ready(2 * k)) return false;
        tc_fence_after();
        const uint32_t qa = desc_lo_kmajor(row_tile(k, 1));
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t at = (kk >> 2) * kSlabBytes + (kk & 3) * 32;
          mma_ss_by(lead, tmem_u + L::kColS, desc_at(ka, at), desc_at(qa, at), kIdescS, kk > 0);
        }
        mma_ss_by(lead, tmem_u + L::kColS, ones, stat_tile(2 * k), kIdescS, 1);
        tc_commit_by(lead, s_full);
        tc_commit_by(lead, stat_free + 2 * k % L::kStats);
        return true;
      };
      auto issue_dp = [&](int k) -> bool {
        if (!ready(do_full + k % kStages, (k / kStages) & 1, 512) || !stat_ready(2 * k + 1)) return false;
        tc_fence_after();
        const uint32_t da = desc_lo_kmajor(row_tile(k, 0));
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t at = (kk >> 2) * kSlabBytes + (kk & 3) * 32;
          mma_ss_by(lead, tmem_u + L::kColDP, desc_at(va, at), desc_at(da, at), kIdescS, kk > 0);
        }
        mma_ss_by(lead, tmem_u + L::kColDP, ones, stat_tile(2 * k + 1), kIdescS, 1);
        tc_commit_by(lead, dp_full);
        tc_commit_by(lead, stat_free + (2 * k + 1) % L::kStats);
        return true;
      };
      auto issue_dv = [&](int k) -> bool {
        if (!ready(p_full, k & 1, 64) || !ready(do_full + k % kStages, (k / kStages) & 1, 512)) return false;
        tc_fence_after();
        const uint32_t db = desc_lo_mnmajor(row_tile(k, 0), kSlabBytes);
#pragma unroll
        for (int kk = 0; kk < kRows / 16; ++kk)
          mma_ts_by(lead, tmem_u + L::kColDV, tmem_u + L::kColP + (kk >> 2) * L::kStepP + (kk & 3) * 8, desc_at(db, kk * 2048), kIdescT, k > 0 || kk > 0);
        tc_commit_by(lead, dv_done);
        return true;
      };
      auto issue_dk = [&](int k) {
        const uint32_t qb = desc_lo_mnmajor(row_tile(k, 1), kSlabBytes), dsk = desc_lo_kmajor(ds_tile(k));
#pragma unroll
        for (int kk = 0; kk < kRows / 16; ++kk)
          mma_ss_by(lead, tmem_u + L::kColDK, desc_at(dsk, (kk >> 2) * kSlabBytes + (kk & 3) * 32), desc_at(qb, kk * 2048), kIdescT, k > 0 || kk > 0);
        tc_commit_by(lead, q_free + k % kStages);
      };
      auto issue_dq = [&](int k) {
        // the 16-key steps that hold a key which a row of the tile attends
        const int t0 = t_lo + k * p.nq, t1 = min(t0 + p.nq, t_lo + n_q) - 1;
        const int k0 = max(0, t0 - window + 1 - key0) >> 4, k1 = min(kWideKeys - 1, t1 - key0) >> 4;
        const uint32_t dsm = desc_lo_mnmajor(ds_tile(k), kSlabBytes);
        for (int kk = k0; kk <= k1; ++kk)
          mma_ss_by(lead, tmem_u + L::kColDQ, desc_at(dsm, kk * 2048), desc_at(kb, kk * 2048), kIdescDQ, kk > k0);
        tc_commit_by(lead, acc_full);
        if (L::kOwnStage) tc_commit_by(lead, ds_free + k % L::kDsTiles);
      };
      bool ok = ready(bar_kv, 0, 32) && issue_s(0);
      if (L::kOwnDq) {
        // S, dP of tile k + 1 are there when the compute warps are done with tile k
        ok = ok && issue_dp(0);
        for (int k = 0; ok && k < n_tiles; ++k) {
          if (!(ok = ready(p_full, k & 1, 64))) break;           // (S has been read as well)
          if (k + 1 < n_tiles && !(ok = issue_s(k + 1))) break;
          if (!(ok = issue_dv(k))) break;
          tc_commit_by(lead, do_free + k % kStages);
          if (!(ok = ready(ds_full, k & 1, 64))) break;
          tc_fence_after();
          if (k + 1 < n_tiles && !(ok = issue_dp(k + 1))) break;
          issue_dk(k);
          if (k > 0 && !(ok = ready(dq_read, (k - 1) & 1, 1024))) break;
          tc_fence_after();
          issue_dq(k);
        }
      } else {
        // dP of a tile takes the columns of the last tile's dQ: where those are still being read, dV goes first
        for (int k = 0; ok && k < n_tiles; ++k) {
          if (!(ok = ready(p_full, k & 1, 64))) break;
          const bool dp_first = k == 0 || __all_sync(0xffffffffu, mbar_test_wait(dq_read, (k - 1) & 1));
          if (!dp_first && (!(ok = issue_dv(k)) || !(ok = ready(dq_read, (k - 1) & 1, 1024)))) break;
          if (!(ok = issue_dp(k))) break;
          if (dp_first && !(ok = issue_dv(k))) break;
          tc_commit_by(lead, do_free + k % kStages);
          if (k + 1 < n_tiles && !(ok = issue_s(k + 1))) break;
          if (!(ok = ready(ds_full, k & 1, 64))) break;
          tc_fence_after();
          issue_dk(k);
          issue_dq(k);
        }
      }
      // the tensor pipe is idle before TMEM is read for dK / dV and given back, whatever happened
      tc_commit_by(lead, bar_drain);
      if (!mbar_wait(bar_drain, 0, p.status, s_abort, 4096)) mbar_wait_drain(bar_drain, 0);
    }
  } else if (warp < 8) {
    // ---- compute warps: lane = key, this warp's half of the rows -------------------------------------
    const int quad = warp & 3, half = warp >> 2;
    const int kr = quad * 32 + lane, key = key0 + kr;
    const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16) + half * 64;
    const uint32_t p_base = tmem + ((uint32_t)(quad * 32) << 16) + L::kColP + half * L::kStepP;
    const uint32_t ds_row0 = smem_u32(sDs) + half * kSlabBytes + kr * 128;
    // Where K and V are finite, P = 0 masks dS = P * (dP - delta) as well, and rows past nq * G, zeros in Q and dO, may count
    // as attended (as others they would have these warps mask every element of every tile).  A K or V that is infinite
    // or NaN spoils dS of rows that do not attend it, and rows that are not there.
    const bool odd = group_or(3, 384, 0);
    if (odd) masked_row_tiles<D>(p, smem, tmem);
    for (int k = odd ? n_tiles : 0; k < n_tiles; ++k) {
      const int qi0 = k * p.nq, t0 = t_lo + qi0;
      const uint32_t ds_row = ds_row0 + k % L::kDsTiles * L::kDsBytes;
      // rows [lo, hi) attend the key
      const int q_end = min(p.nq, n_q - qi0);
      const int q_first = key - t0, q_last = min(q_end, key - t0 + window);
      const int lo = min(max(q_first, 0), p.nq) * p.G, hi = key >= p.T ? 0 : q_last >= p.nq ? kRows : q_last * p.G;
      // of this warp's half: bit c for row half * 64 + c
      const int lo_h = min(max(lo - half * 64, 0), 64), hi_h = min(max(hi - half * 64, 0), 64);
      const uint64_t upto = hi_h == 64 ? ~0ull : (1ull << hi_h) - 1ull;
      const uint64_t attended = lo_h == 64 ? 0ull : upto >> lo_h << lo_h;
      bool ok = mbar_wait(s_full, k & 1, p.status, s_abort, 64);
      if (!__all_sync(0xffffffffu, ok)) break;                 // the whole warp leaves together
      tc_fence_after();
      uint32_t pr[64];                               // S, then p
      tmem_ld32(lane_base + L::kColS, pr);
      tmem_ld32(lane_base + L::kColS + 32, pr + 32);
      tmem_wait_ld();
      auto probabilities = [&](auto masked) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t pk[16];
#pragma unroll
          for (int c2 = 0; c2 < 16; ++c2) {
            float x[2], v[2];
            mul_f32x2(pr[h * 32 + c2 * 2], pr[h * 32 + c2 * 2 + 1], p.scale_log2, p.scale_log2, x[0], x[1]);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int c = h * 32 + c2 * 2 + e;
              v[e] = ex2(x[e]);
              if (decltype(masked)::value && !((uint32_t)(attended >> (h * 32)) >> (c2 * 2 + e) & 1u)) v[e] = 0.f;
              pr[c] = __float_as_uint(v[e]);
            }
            pk[c2] = pack_bf16(v[0], v[1]);
          }
          // (its columns may be written once dV of the last tile is there)
          if (L::kOwnP && h == 0 && k > 0) ok = mbar_wait(dv_done, (k - 1) & 1, p.status, s_abort, 64);
          __syncwarp();
          tmem_st16(p_base + h * 16, pk);
        }
      };
      if (__all_sync(0xffffffffu, attended == ~0ull)) probabilities(std::false_type());
      else probabilities(std::true_type());
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(p_full);
      ok = ok && mbar_wait(dp_full, k & 1, p.status, s_abort, 64);
      if (ok && k >= L::kDsTiles) ok = mbar_wait(ds_free + k % L::kDsTiles, (k / L::kDsTiles - 1) & 1, p.status, s_abort, 64);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t dp[32];
        tmem_ld32(lane_base + L::kColDP + h * 32, dp);
        tmem_wait_ld();
        uint32_t pk[16];
#pragma unroll
        for (int c2 = 0; c2 < 16; ++c2) {
          float x[2], v[2];
          mul_f32x2(dp[c2 * 2], dp[c2 * 2 + 1], p.scale, p.scale, x[0], x[1]);
          mul_f32x2(pr[h * 32 + c2 * 2], pr[h * 32 + c2 * 2 + 1], x[0], x[1], v[0], v[1]);
          pk[c2] = pack_bf16(v[0], v[1]);
        }
#pragma unroll
        for (int v4 = 0; v4 < 4; ++v4)
          st_shared_16b(ds_row + ((uint32_t)((h * 4 + v4) ^ (kr & 7)) << 4), pk[v4 * 4], pk[v4 * 4 + 1], pk[v4 * 4 + 2], pk[v4 * 4 + 3]);
      }
      fence_proxy_async();
      tc_fence_before();
      mbar_arrive(ds_full);
    }
  } else {
    // ---- dQ of every tile: TMEM -> bf16 -> staging tile -> partial buffer ------------------------------
    const int quad = warp & 3, lt = tid - 8 * 32;
    const int row = quad * 32 + lane;
    const int slot = j % p.n_slots;
    const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16) + L::kColDQ;
    // the dQ warps have nothing to do yet: they look at the tile's K and V for the compute warps, behind the first S (by the
    // compute warps themselves: 8192 tokens of 16 / 2 heads of 128 123 us instead of 120; 119 without)
    bool odd = false;
    if (mbar_wait(bar_kv, 0, p.status, s_abort, 32)) {
      __nv_bfloat162 z(0.f, 0.f);                    // x * 0: 0 or NaN
#pragma unroll 8
      for (int i = lt; i < 2 * L::kKVBytes / 16; i += 128) {        // (V lies behind K)
        const uint4 u = reinterpret_cast<const uint4*>(sK)[i];
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) z = __hfma2(reinterpret_cast<const __nv_bfloat162&>(w[e]), __nv_bfloat162(0.f, 0.f), z);
      }
      odd = (reinterpret_cast<const uint32_t&>(z) & 0x7fff7fffu) != 0u;
    }
    group_or(3, 384, odd);
    for (int k = 0; k < n_tiles; ++k) {
      uint8_t* stage = sOut;
      const bool ok = mbar_wait(acc_full, k & 1, p.status, s_abort, 128);
      // the store of the last tile has read the staging tile (one thread knows, the barrier tells the others)
      if (L::kOwnStage) {
        if (lt == 0) bulk_wait_read();
        if (group_or(1, 128, !ok)) break;
      }
      __syncwarp();
      tc_fence_after();
#pragma unroll
      for (int cc = 0; cc < D / 32; ++cc) {
        uint32_t r32[32];
        tmem_ld32(lane_base + cc * 32, r32);
        tmem_wait_ld();
        if (cc == D / 32 - 1) {            // dQ is in registers: its columns may be written again
          tc_fence_before();
          mbar_arrive(dq_read);
        }
#pragma unroll
        for (int v4 = 0; v4 < 4; ++v4) {
          const uint32_t ch = (uint32_t)(cc * 4 + v4);
          st_shared_16b(smem_u32(stage) + (ch >> 3) * kSlabBytes + row * 128 + (((ch & 7) ^ (row & 7)) << 4),
                        pack_bf16(__uint_as_float(r32[v4 * 8 + 0]), __uint_as_float(r32[v4 * 8 + 1])),
                        pack_bf16(__uint_as_float(r32[v4 * 8 + 2]), __uint_as_float(r32[v4 * 8 + 3])),
                        pack_bf16(__uint_as_float(r32[v4 * 8 + 4]), __uint_as_float(r32[v4 * 8 + 5])),
                        pack_bf16(__uint_as_float(r32[v4 * 8 + 6]), __uint_as_float(r32[v4 * 8 + 7])));
        }
      }
      fence_proxy_async();
      if (group_or(1, 128, !ok)) break;                   // the whole group leaves together
      if ((k + 1) * p.nq <= n_q) {
        // its rows are consecutive queries: one TMA store per slab
        if (lt == 0) {
#pragma unroll
          for (int sl = 0; sl < kSlabs; ++sl)
            tma_store_5d_hint(&tm_dq, stage + sl * kSlabBytes, sl * 64, 0, slot, t_lo + k * p.nq, bh, l2_policy_evict_first());
          bulk_commit();
          if (!L::kOwnStage) {
            bulk_wait_read();
            mbar_arrive(ds_free);
          }
        }
      } else {   // the ragged last tile: whole rows out by hand, 16 bytes a lane
        constexpr int kChunks = D / 8;
        const int c = lt % kChunks;
        for (int r = lt / kChunks; r < kRows; r += 128 / kChunks) {
          const int ql = r / p.G, qi = k * p.nq + ql;
          if (ql >= p.nq || qi >= n_q) continue;
          const uint4 v = *reinterpret_cast<const uint4*>(stage + (c >> 3) * kSlabBytes + r * 128 + (((c & 7) ^ (r & 7)) << 4));
          const size_t prow = (((size_t)bh * p.T + t_lo + qi) * p.n_slots + slot) * p.G + r % p.G;
          *reinterpret_cast<uint4*>(p.dq_part + prow * D + c * 8) = v;
        }
      }
    }
    if (lt == 0) bulk_wait_read();
  }

  // ---- dK, dV: lane = key; warps 0-3 have dV, 4-7 dK.  Through shared memory (16-byte chunks XOR key), so that they
  // leave in whole rows --------------------------------------------------------------------------------
  __syncthreads();           // the MMA thread has seen the tensor pipe drain (bar_drain)
  tc_fence_after();
  const bool gone = *s_abort != 0;
  if (warp < 8 && !gone) {
    const int quad = warp & 3, kr = quad * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16) + (warp >> 2 ? L::kColDK : L::kColDV);
    const uint32_t row = smem_u32(sRow) + ((warp >> 2) * kWideKeys + kr) * (D * 2);
#pragma unroll
    for (int cc = 0; cc < D / 32; ++cc) {
      uint32_t r[32];
      tmem_ld32(lane_base + cc * 32, r);
      tmem_wait_ld();
#pragma unroll
      for (int v4 = 0; v4 < 4; ++v4)
        st_shared_16b(row + (((cc * 4 + v4) ^ (kr & 7)) << 4), pack_bf16(__uint_as_float(r[v4 * 8 + 0]), __uint_as_float(r[v4 * 8 + 1])),
                      pack_bf16(__uint_as_float(r[v4 * 8 + 2]), __uint_as_float(r[v4 * 8 + 3])),
                      pack_bf16(__uint_as_float(r[v4 * 8 + 4]), __uint_as_float(r[v4 * 8 + 5])),
                      pack_bf16(__uint_as_float(r[v4 * 8 + 6]), __uint_as_float(r[v4 * 8 + 7])));
    }
  }
  __syncthreads();
  if (!gone) {
    constexpr int kVec = D / 8;
    for (int i = tid; i < 2 * kWideKeys * kVec; i += kWideThreads) {
      const int c = i % kVec, kr = (i / kVec) % kWideKeys, which = i / (kVec * kWideKeys);
      if (key0 + kr >= p.T) continue;
      const uint4 v = *reinterpret_cast<const uint4*>(sRow + (which * kWideKeys + kr) * (D * 2) + ((c ^ (kr & 7)) << 4));
      __nv_bfloat16* dst = (which ? p.dk : p.dv) + ((size_t)bh * p.T + key0 + kr) * D + c * 8;
      if (((uintptr_t)dst & 15) == 0) {
        *reinterpret_cast<uint4*>(dst) = v;
      } else {                                       // a caller's tensor may start anywhere
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) dst[e] = __ushort_as_bfloat16((unsigned short)(w[e >> 1] >> (16 * (e & 1))));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

template <int D>
static int launch(const WideArgs& p, const CUtensorMap* tm, dim3 grid, cudaStream_t st) {
  NSA_CUDA_OK(func_smem((const void*)tc_bwd_wide_kernel<D>, Wide<D>::kSmem));
  tc_bwd_wide_kernel<D><<<grid, kWideThreads, Wide<D>::kSmem, st>>>(tm[0], tm[1], tm[2], tm[3], tm[4], p);
  NSA_LAUNCH_OK("tc_bwd_wide_kernel");
  return NSA_OK;
}

int bwd_wide_launch(const AttnArgs& a, const WideArgs& p, const char* name, cudaStream_t st) {
  CUtensorMap tm[5];
  const int units = a.B * a.Hkv;
  int rc = make_map(&tm[0], a.k, a.D, a.T, units, kWideKeys, 1);
  if (rc == NSA_OK) rc = make_map(&tm[1], a.v, a.D, a.T, units, kWideKeys, 1);
  if (rc == NSA_OK) rc = make_map_query_rows(&tm[2], a.q, a.D, a.T, a.B * a.Hq, p.G, p.nq);
  if (rc == NSA_OK) rc = make_map_query_rows(&tm[3], a.d_o, a.D, a.T, a.B * a.Hq, p.G, p.nq);
  if (rc == NSA_OK) rc = make_map_partial(&tm[4], p.dq_part, a.D, p.G, p.n_slots, a.T, units, p.nq);
  if (rc != NSA_OK) return rc;
  KernelScope ks(name, st);
  const dim3 grid((a.T + kWideKeys - 1) / kWideKeys, units);
  return a.D == 128 ? launch<128>(p, tm, grid, st) : launch<64>(p, tm, grid, st);
}

}  // namespace tc
}  // namespace nsa
