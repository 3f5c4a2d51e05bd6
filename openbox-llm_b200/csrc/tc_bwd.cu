// tcgen05 / TMEM backward of the three attention branches, key-tile outer.
//
// One CTA owns a tile of 64 keys of one (batch, kv head): K and V of the tile are loaded
// once (TMA), dK^T and dV^T of the tile stay in TMEM for the whole CTA and are written once,
// with no atomics.  The CTA walks the (query, head) rows that attend the tile, 128 rows at a
// time (nq queries x the G heads of the group):
//   window      queries [64 j, 64 j + 63 + W - 1]  (up to a wave of tiles; more go on tiles of 128 keys, use_wide)
//   compression queries t >= (64 j + 1) * Bsz - 1
//   selection   the queries that list block j, from the block -> query CSR
// Q and dO rows arrive by TMA into 128B-swizzled tiles: one box per row tile for the window and
// compression branches (consecutive queries), one box per query and 64-column slab for
// selection.  Selection CTAs take (block, chunk of row tiles) items from a device-built work list.
// Per row tile, five MMAs:
//   S    = Q K^T          (A: Q  K-major,   B: K  K-major)
//   dP   = dO V^T         (A: dO K-major,   B: V  K-major)
//   dV^T += dO^T P        (A: dO MN-major,  B: P  MN-major)      P, dS: bf16 tiles the threads
//   dK^T += Q^T dS        (A: Q  MN-major,  B: dS MN-major)      write to shared memory
//   dQ   = dS K           (A: dS K-major,   B: K  MN-major)
// with p = exp2(s*scale*log2e - lse*log2e) and dS = scale * p * (dP - delta) computed by the
// thread that owns the row (TMEM lane = row).  dQ of a row is the sum over the key tiles it
// attends.  Two ways out of the CTA:
//   slots        every (row tile, key tile) result leaves as a bf16 partial tile (TMA store) and a
//                second kernel adds the partials of each query in fp32, in a fixed order
//                (selection always; window / compression when the caller wants dq itself);
//   accumulator  window / compression inside the whole op: the fp32 tile is added to one fp32
//                accumulator [units][T][G][D] by TMA reduce-add.  Consecutive key tiles hit the same
//                consecutive query rows at nearby times, so the adds meet in L2 and no partial
//                buffer exists; the order of the adds, hence the last bits of dq, is not fixed.
#include <algorithm>
#include <type_traits>

#include "cluster.cuh"
#include "sel_row.cuh"
#include "tc_bwd_wide.cuh"
#include "tc_common.cuh"
#include "tc_host.cuh"

namespace nsa {
namespace tc {

struct BwdArgs {
  const __nv_bfloat16* q;
  const __nv_bfloat16* k;
  const __nv_bfloat16* v;
  const __nv_bfloat16* d_o;
  const int32_t* block_idx;    // three-term selection
  const float* lse;
  const float* delta;          // sum_d dO * O per row (unscaled)
  const float* row_scale;      // gate value per row of a gated branch, or null
  SelPlan plan;                // selection
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  void* dq_part;               // bf16, fp32 for three-term selection
  float* dk_acc;               // fp32 accumulators, used when the row tiles of a key tile are split
  float* dv_acc;
  int* status;
  int split_chunk;             // row tiles per CTA when split
  size_t acc_stride;           // compression, few chunks: floats between their accumulators (0: one for all, by atomics)
  int csize;                   // CTAs per cluster
  int B, Hq, Hkv, T, Lk, G, nq;
  int kind, window, block_size, S;
  int n_ktiles, n_slots;
  int merged;                  // selection: one TMA box per (query, tensor) brings both 64-column slabs
  int dq_acc_mode;             // 1: dQ tiles are added to the fp32 accumulator (window / compression)
  float scale, scale_log2;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}

constexpr int kRowTileBytes = kRows * 128 * 2;   // Q or dO row tile: always two 64-element slabs
constexpr int kPBytes = kRows * 128;             // P or dS: 128 rows x 64 keys bf16
constexpr int kGroupThreads = 256;               // one compute group: 2 warps per TMEM lane quadrant
constexpr int kGroupBytes = 2 * kRowTileBytes + 2 * kPBytes;   // Q, dO, P, dS of one group
constexpr int kMaxNq = 64;                       // queries per row tile (group size >= 2)

__host__ __device__ inline size_t bwd_smem_bytes(int D) {
  return (size_t)2 * kKeys * 128 * (D / 64)      // K, V
         + 2 * (size_t)kGroupBytes               // two groups
         + 256                                   // barriers
         + 2 * 2 * kMaxNq * 4                    // query positions, double buffered, per group
         + 2 * 128 * 4                           // partial-row index of each tile row, per group
         + 768;                                  // alignment slack (checked at run time)
}

__device__ __forceinline__ void group_sync(int group) {
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(kGroupThreads) : "memory");
}
__device__ __forceinline__ void named_sync_b(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// Named barrier that also tells every thread whether any of them brought a non-zero `pred`: the
// way a group of warps decides together to leave after a given-up wait.
__device__ __forceinline__ bool named_or_b(int id, int threads, int pred) {
  uint32_t out;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %3, 0;\n\t"
      "bar.red.or.pred p, %1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(out)
      : "r"(id), "r"(threads), "r"(pred)
      : "memory");
  return out != 0;
}

// Two compute groups of 256 threads share the key tile and the dK^T / dV^T accumulators and
// take alternate row tiles, so that one group's MMAs and memory waits overlap the other
// group's arithmetic.  Inside a group, the two warps of a TMEM lane quadrant split the 64 key
// columns of a row between them.  Row r of a tile is head r % G of the tile's query r / G: the
// G rows of a query arrive by one TMA box each for Q and dO (128B swizzle), whatever the query
// list looks like, and leave as bf16 dQ partials through a 128B-swizzled staging tile: a full
// tile by one asynchronous TMA store per slab, the ragged last tile as whole rows by hand.
template <int D>
__global__ void __launch_bounds__(512, 1)
tc_bwd_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
              const __grid_constant__ CUtensorMap tm_q_run, const __grid_constant__ CUtensorMap tm_do_run,
              const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ CUtensorMap tm_dqacc,
              const BwdArgs p) {
  constexpr int kSlabs = D / 64;
  constexpr int kKVBytes = kKeys * 128 * kSlabs;
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kColDV = 256, kColDK = 320;   // group g: S at 128 g, dP at 128 g + 64, dQ over both
  constexpr uint32_t kIdescS = idesc_bf16(128, kKeys, 0, 0);     // rows x keys
  constexpr uint32_t kIdescT = idesc_bf16(128, kKeys, 1, 1);     // d x keys, both MN-major
  constexpr uint32_t kIdescDQ = idesc_bf16(128, D, 0, 1);        // rows x d

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // pointer arithmetic keeps the shared address space
  uint8_t* sK = smem;
  uint8_t* sV = sK + kKVBytes;
  uint8_t* sGroup = sV + kKVBytes;
  uint64_t* bars = (uint64_t*)(sGroup + 2 * kGroupBytes);
  uint64_t* bar_kv = bars + 0;
  uint32_t* s_tmem = (uint32_t*)(bars + 8);
  volatile int* s_abort = (volatile int*)(s_tmem + 1);
  int* s_rowt_all = (int*)(bars + 10);               // [2 groups][2 buffers][kMaxNq]
  uint32_t* s_prow_all = (uint32_t*)(s_rowt_all + 2 * 2 * kMaxNq);   // [2][128]

  const int tid = threadIdx.x;
  const int grp = tid / kGroupThreads, lt = tid % kGroupThreads;
  const int wg = lt >> 5, lane = lt & 31;
  const int quad = wg & 3, half = wg >> 2;           // TMEM lane quadrant, key-column half
  const int row = quad * 32 + lane;                  // row of the tile this thread works on
  uint8_t* sQ = sGroup + grp * kGroupBytes;
  uint8_t* sDO = sQ + kRowTileBytes;
  uint8_t* sP = sDO + kRowTileBytes;
  uint8_t* sDS = sP + kPBytes;
  uint64_t* bar_sp = bars + 1 + 3 * grp;
  uint64_t* bar_acc = bars + 2 + 3 * grp;
  uint64_t* bar_g = bars + 3 + 3 * grp;
  uint64_t* bar_drain = bars + 7 + 2 * grp;
  int* s_rowt = s_rowt_all + grp * 2 * kMaxNq;
  uint32_t* s_prow = s_prow_all + grp * 128;

  const int j = blockIdx.x;                          // key tile
  const int bh = blockIdx.y;
  const int b = bh / p.Hkv, hkv = bh % p.Hkv;
  const int key0 = j * kKeys;
  const int ql = row / p.G, g = row % p.G;
  const int head = hkv * p.G + g;
  const bool row_slot_ok = ql < p.nq;

  // ---- the queries that attend this key tile ---------------------------------------------
  int t_lo = 0, n_q = 0;
  if (p.kind == 0) {
    t_lo = key0;
    n_q = min(p.T - 1, key0 + kKeys - 1 + p.window - 1) - t_lo + 1;
  } else {
    t_lo = key0 * p.window + p.block_size - 1;       // first query that sees summary key0 (window: the stride)
    n_q = p.T - t_lo;
  }
  n_q = max(n_q, 0);
  const int n_rt_all = (n_q + p.nq - 1) / p.nq;
  // gridDim.z > 1: the row tiles are split in chunks and dK / dV go through fp32 atomics
  const int chunk = (int)gridDim.z > 1 ? p.split_chunk : n_rt_all;
  const int rt_begin = (int)blockIdx.z * chunk;
  const int rt_end = min(n_rt_all, rt_begin + chunk);
  const bool split = gridDim.z > 1;

  if (rt_end <= rt_begin) {
    if (!split && n_rt_all == 0) {   // nobody attends these keys: their gradients are zero
      for (int i = tid; i < kKeys * D / 8; i += blockDim.x) {
        const int key = key0 + i / (D / 8);
        if (key < p.Lk) {
          const size_t off = ((size_t)bh * p.Lk + key) * D + (i % (D / 8)) * 8;
          *reinterpret_cast<uint4*>(p.dk + off) = make_uint4(0, 0, 0, 0);
          *reinterpret_cast<uint4*>(p.dv + off) = make_uint4(0, 0, 0, 0);
        }
      }
    }
    return;
  }

  if (tid == 0) {
    int bad = (*(volatile int*)p.status != 0) ? 1 : 0;
    if ((size_t)((uint8_t*)(s_prow_all + 2 * 128) - smem_raw) > bwd_smem_bytes(D)) {
      atomicOr(p.status, 256);   // the shared-memory window is less aligned than assumed
      bad = 1;
    }
    *s_abort = bad;
    // S / dP ready (bars 1 and 4) = the MMAs have completed and the previous tile's dQ store
    // has left the staging tile, which is the P / dS tile: two arrivals
    for (int k = 0; k <= 6; ++k) mbar_init(bars + k, (k == 1 || k == 4) ? 2 : 1);
    mbar_init(bars + 7, 1); mbar_init(bars + 9, 1);   // per group: an aborted CTA waits here for its last MMAs
    fence_barrier_init();
    prefetch_tensormap(&tm_k); prefetch_tensormap(&tm_v);
    prefetch_tensormap(&tm_q_run); prefetch_tensormap(&tm_do_run);
    prefetch_tensormap(p.dq_acc_mode ? &tm_dqacc : &tm_dq);
  }
  __syncthreads();
  if (*s_abort) return;
  // Rows past nq * G of a tile (and, for D = 64, the second slab) are never loaded: keep them 0.
  for (int i = tid; i < 2 * 2 * kRowTileBytes / 16; i += blockDim.x) {
    const int buf = i / (kRowTileBytes / 16), o16 = i % (kRowTileBytes / 16);
    uint8_t* base = sGroup + (buf >> 1) * kGroupBytes + (buf & 1) * kRowTileBytes;
    *reinterpret_cast<uint4*>(base + o16 * 16) = make_uint4(0, 0, 0, 0);
  }
  fence_proxy_async();

  if (tid < 32) {
    tmem_alloc(s_tmem, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
  const uint32_t colS = grp * 128, colDP = grp * 128 + 64, colDQ = grp * 128;
  // Q / dO tiles: slab-major (8-row groups 1024 bytes apart, slabs kRows * 128 apart)
  constexpr uint32_t q_slab = kRows * 128, q_sbo = 1024u;

  if (tid == 0) {
    mbar_expect_tx(bar_kv, 2 * kKVBytes);
#pragma unroll
    for (int s = 0; s < kSlabs; ++s) {
      tma_load_3d(sK + s * (kKeys * 128), &tm_k, bar_kv, s * 64, key0, bh);
      tma_load_3d(sV + s * (kKeys * 128), &tm_v, bar_kv, s * 64, key0, bh);
    }
  }
  // dK^T / dV^T start at zero so that every MMA into them accumulates
  if (grp == 0 && half == 0) {
    uint32_t z[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) z[c] = 0u;
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) tmem_st32(lane_base + kColDV + cc * 32, z);
    tmem_wait_st();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (tid == 0 || tid == kGroupThreads) mbar_wait(bar_kv, 0, p.status, s_abort, 32);

  // query position of this thread's row in row tile i (-1: no row)
  auto row_query = [&](int i) -> int {
    const int qi = i * p.nq + ql;
    if (!row_slot_ok || qi >= n_q) return -1;
    return t_lo + qi;
  };
  auto row_index = [&](int t) -> size_t { return (size_t)(b * p.Hq + head) * p.T + t; };
  const uint32_t gather_bytes = (uint32_t)(p.nq * p.G * 128 * kSlabs * 2);
  // part: 0 = Q and dO, 1 = Q now (the byte count of both is
  // announced), 2 = dO, issued later because its tile served as staging meanwhile
  auto gather = [&](const int* rowt, int part = 0) {
    // the tile's queries are consecutive tokens, one box per slab
    if (lt == 0) {
      if (part != 2) mbar_expect_tx(bar_g, gather_bytes);
      const int tq = rowt[0] >= 0 ? rowt[0] : p.T;
#pragma unroll
      for (int s = 0; s < kSlabs; ++s) {
        if (part != 2) tma_load_3d(sQ + s * (kRows * 128), &tm_q_run, bar_g, s * 64, b * p.Hq + hkv * p.G, tq);
        if (part != 1) tma_load_3d(sDO + s * (kRows * 128), &tm_do_run, bar_g, s * 64, b * p.Hq + hkv * p.G, tq);
      }
    }
  };

  // Row metadata runs ahead of the work: the query position two tiles ahead (t_nxt) and, one
  // iteration later, its lse / delta, so that no dependent global load is waited for in line.
  int i = rt_begin + grp;
  int t_cur = i < rt_end ? row_query(i) : -1;
  int t_nxt = i + 2 < rt_end ? row_query(i + 2) : -1;
  float lse_cur = 0.f, delta_cur = 0.f, gate_cur = 1.f;
  if (t_cur >= 0) {
    lse_cur = __ldg(p.lse + row_index(t_cur));
    delta_cur = __ldg(p.delta + row_index(t_cur));
    if (p.row_scale) gate_cur = __ldg(p.row_scale + row_index(t_cur));
  }
  int buf = 0;
  bool g_pending = false;     // a gather of this group is on its way and its arrival has not been seen
  if (i < rt_end) {
    if (g == 0 && half == 0 && row_slot_ok) s_rowt[ql] = t_cur;
    group_sync(grp);
    gather(s_rowt);
    g_pending = true;
  }
  uint32_t phase = 0;
  for (; i < rt_end; i += 2, phase ^= 1, buf ^= 1) {
    const int t_nn = (i + 4 < rt_end) ? row_query(i + 4) : -1;
    float lse_nxt = 0.f, delta_nxt = 0.f, gate_nxt = 1.f;
    if (t_nxt >= 0) {
      lse_nxt = ldg_f32_now(p.lse + row_index(t_nxt));
      delta_nxt = ldg_f32_now(p.delta + row_index(t_nxt));
      if (p.row_scale) gate_nxt = ldg_f32_now(p.row_scale + row_index(t_nxt));
    }
    // query positions of this group's next tile, for the gather issued further down
    if (g == 0 && half == 0 && row_slot_ok) s_rowt[(buf ^ 1) * kMaxNq + ql] = t_nxt;
    if (mbar_wait(bar_g, phase, p.status, s_abort, 512)) g_pending = false;
    // also: the staging tile of the previous iteration has been read.  One decision for the whole
    // group: after a given-up wait it issues and writes nothing more
    if (named_or_b(grp + 1, kGroupThreads, *s_abort)) break;
    if (lt == 0) {
      tc_fence_after();
      const uint32_t qa = desc_lo_kmajor(smem_u32(sQ)), da = desc_lo_kmajor(smem_u32(sDO));
      const uint32_t ka = desc_lo_kmajor(smem_u32(sK)), va = desc_lo_kmajor(smem_u32(sV));
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t slab = kk >> 2, in = (kk & 3) * 32;
        mma_ss(tmem + colS, desc_at_sbo(qa, slab * q_slab + in, q_sbo),
               desc_at(ka, slab * (kKeys * 128) + in), kIdescS, kk > 0);
      }
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t slab = kk >> 2, in = (kk & 3) * 32;
        mma_ss(tmem + colDP, desc_at_sbo(da, slab * q_slab + in, q_sbo),
               desc_at(va, slab * (kKeys * 128) + in), kIdescS, kk > 0);
      }
      tc_commit(bar_sp);
      bulk_wait_read();
      mbar_arrive(bar_sp);
    }
    // valid key columns of this row: one range [lo, hi]
    int lo = 0, hi = -1;
    if (t_cur >= 0) {
      if (p.kind == 0) {
        lo = max(0, t_cur - p.window + 1 - key0);
        hi = min(kKeys - 1, t_cur - key0);
      } else {
        hi = min(kKeys - 1, cmp_visible(t_cur, p.block_size, p.window, p.Lk) - 1 - key0);
      }
    }
    const float lse2_cur = lse_cur * kLog2e;
    mbar_wait(bar_sp, phase, p.status, s_abort, 64);
    tc_fence_after();
    __syncwarp();
    {
      uint32_t rs[32], rp[32];
      tmem_ld32(lane_base + colS + half * 32, rs);
      tmem_ld32(lane_base + colDP + half * 32, rp);
      tmem_wait_ld();
      uint32_t pp[16], pd[16];
#pragma unroll
      for (int c2 = 0; c2 < 16; ++c2) {
        float pv[2], dv[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = half * 32 + c2 * 2 + e;
          const bool ok = (c >= lo) && (c <= hi);
          // gate_cur * p: the branch's dO is gate * dO, so dV takes (gate p)^T dO and
          // dS = scale * gate * p * (dO.v - dO.o)
          const float pr = ok ? gate_cur * ex2(__uint_as_float(rs[c2 * 2 + e]) * p.scale_log2 - lse2_cur) : 0.f;
          pv[e] = pr;
          dv[e] = pr * (__uint_as_float(rp[c2 * 2 + e]) - delta_cur) * p.scale;
        }
        pp[c2] = pack_bf16(pv[0], pv[1]);
        pd[c2] = pack_bf16(dv[0], dv[1]);
      }
      const uint32_t p_row = smem_u32(sP) + row * 128, ds_row = smem_u32(sDS) + row * 128;
#pragma unroll
      for (int k4 = 0; k4 < 4; ++k4) {
        const uint32_t chunk16 = (uint32_t)((half * 4 + k4) ^ (row & 7)) << 4;
        st_shared_v4(p_row + chunk16, pp[k4 * 4], pp[k4 * 4 + 1], pp[k4 * 4 + 2], pp[k4 * 4 + 3]);
        st_shared_v4(ds_row + chunk16, pd[k4 * 4], pd[k4 * 4 + 1], pd[k4 * 4 + 2], pd[k4 * 4 + 3]);
      }
    }
    fence_proxy_async();
    tc_fence_before();
    group_sync(grp);
    if (lt == 0) {
      tc_fence_after();
      const uint32_t qa = desc_lo_mnmajor(smem_u32(sQ), q_slab);
      const uint32_t da = desc_lo_mnmajor(smem_u32(sDO), q_slab);
      const uint32_t pa = desc_lo_mnmajor(smem_u32(sP), 0), dsa = desc_lo_mnmajor(smem_u32(sDS), 0);
      const uint32_t dsk = desc_lo_kmajor(smem_u32(sDS)), ka = desc_lo_mnmajor(smem_u32(sK), kKeys * 128);
#pragma unroll
      for (int kk = 0; kk < kRows / 16; ++kk)        // contraction over the 128 rows, 16 (two 8-row groups) a step
        mma_ss(tmem + kColDV, desc_at_sbo(da, kk * 2 * q_sbo, q_sbo), desc_at(pa, kk * 2048), kIdescT, 1);
#pragma unroll
      for (int kk = 0; kk < kRows / 16; ++kk)
        mma_ss(tmem + kColDK, desc_at_sbo(qa, kk * 2 * q_sbo, q_sbo), desc_at(dsa, kk * 2048), kIdescT, 1);
#pragma unroll
      for (int kk = 0; kk < kKeys / 16; ++kk)        // contraction over the 64 keys
        mma_ss(tmem + colDQ, desc_at(dsk, kk * 32), desc_at(ka, kk * 2048), kIdescDQ, kk > 0);
      tc_commit(bar_acc);
    }
    // row of the partial buffer that takes this row's dQ
    if (half == 0) {
      uint32_t prow = 0xffffffffu;
      if (t_cur >= 0) {
        const int slot = p.kind == 0 ? j % p.n_slots : j;
        prow = (uint32_t)((((size_t)bh * p.T + t_cur) * p.n_slots + slot) * p.G + g);
      }
      s_prow[row] = prow;
    }
    mbar_wait(bar_acc, phase, p.status, s_abort, 128);
    tc_fence_after();
    if (p.dq_acc_mode) {
      // dQ: TMEM -> fp32 staging -> TMA reduce-add into the accumulator.  The fp32 tile is D / 32
      // slabs of 128 rows x 128 bytes (128B swizzle): the first two lie over the P / dS tiles, the
      // other two (D = 128) over the dO tile, whose refill therefore waits until the reduction has
      // read them; Q is refilled at once.
      constexpr bool kTwoStep = D > 64;
      if (i + 2 < rt_end) { gather(s_rowt + (buf ^ 1) * kMaxNq, kTwoStep ? 1 : 0); g_pending = true; }
      __syncwarp();
#pragma unroll
      for (int cc = 0; cc < D / 64; ++cc) {          // this thread's half of the D columns
        const int col0 = half * (D / 2) + cc * 32;
        const int slab = col0 >> 5;
        uint8_t* sbase = slab < 2 ? sP + slab * (kRows * 128) : sDO + (slab - 2) * (kRows * 128);
        uint32_t r32[32];
        tmem_ld32(lane_base + colDQ + col0, r32);
        tmem_wait_ld();
        const uint32_t rbase = smem_u32(sbase) + row * 128;
#pragma unroll
        for (int c = 0; c < 8; ++c)
          st_shared_v4(rbase + (((uint32_t)c ^ (uint32_t)(row & 7)) << 4), r32[c * 4], r32[c * 4 + 1],
                       r32[c * 4 + 2], r32[c * 4 + 3]);
      }
      fence_proxy_async();
      tc_fence_before();
      group_sync(grp);
      if (lt == 0) {
        // rows of queries past the tile's range carry zeros (p = 0 there); rows past T are dropped
        const int t_tile = t_lo + i * p.nq;
#pragma unroll
        for (int sl = 0; sl < D / 32; ++sl) {
          const uint8_t* sbase = sl < 2 ? sP + sl * (kRows * 128) : sDO + (sl - 2) * (kRows * 128);
          tma_reduce_add_4d(&tm_dqacc, sbase, sl * 32, 0, t_tile, bh);
        }
        bulk_commit();
        if (kTwoStep && i + 2 < rt_end) {
          bulk_wait_read();
          gather(s_rowt + (buf ^ 1) * kMaxNq, 2);
        }
      }
    } else {
      // the row tiles are free again: fetch this group's next tile
      if (i + 2 < rt_end) { gather(s_rowt + (buf ^ 1) * kMaxNq); g_pending = true; }
      __syncwarp();
      // dQ: TMEM -> bf16 -> staging tile (the P / dS region): one slab of 128-byte rows per 64
      // columns, 16-byte chunks XOR row, which is the layout of a 128B-swizzled TMA box
      {
#pragma unroll
        for (int cc = 0; cc < D / 64; ++cc) {          // this thread's half of the D columns
          const int col0 = half * (D / 2) + cc * 32;
          uint32_t r32[32];
          tmem_ld32(lane_base + colDQ + col0, r32);
          tmem_wait_ld();
#pragma unroll
          for (int v4 = 0; v4 < 4; ++v4) {
            const uint32_t chunk = (uint32_t)((col0 >> 3) + v4);
            st_shared_v4(smem_u32(sP) + (chunk >> 3) * (kRows * 128) + row * 128 + (((chunk & 7) ^ (row & 7)) << 4),
                         pack_bf16(__uint_as_float(r32[v4 * 8 + 0]), __uint_as_float(r32[v4 * 8 + 1])),
                         pack_bf16(__uint_as_float(r32[v4 * 8 + 2]), __uint_as_float(r32[v4 * 8 + 3])),
                         pack_bf16(__uint_as_float(r32[v4 * 8 + 4]), __uint_as_float(r32[v4 * 8 + 5])),
                         pack_bf16(__uint_as_float(r32[v4 * 8 + 6]), __uint_as_float(r32[v4 * 8 + 7])));
          }
        }
      }
      fence_proxy_async();
      tc_fence_before();
      group_sync(grp);
      if ((i + 1) * p.nq <= n_q) {
        // a full tile: its rows are consecutive in the partial buffer, one TMA store per slab
        if (lt == 0) {
          const int slot = p.kind == 0 ? j % p.n_slots : j;
          const int mid = t_lo + i * p.nq, outer = bh;
#pragma unroll
          for (int sl = 0; sl < kSlabs; ++sl)
            tma_store_5d(&tm_dq, sP + sl * (kRows * 128), sl * 64, 0, slot, mid, outer);
          bulk_commit();
        }
      } else {   // the ragged last tile: 16 lanes write the 256 (D = 128) or 128 bytes of one row
        constexpr int kChunks = D / 8;
        constexpr int kRowsPerPass = kGroupThreads / kChunks;
        const int c = lt % kChunks;
#pragma unroll 4
        for (int r = lt / kChunks; r < kRows; r += kRowsPerPass) {
          const uint32_t prow = s_prow[r];
          if (prow != 0xffffffffu) {
            const uint4 v = *reinterpret_cast<const uint4*>(sP + (c >> 3) * (kRows * 128) + r * 128 +
                                                            (((c & 7) ^ (r & 7)) << 4));
            *reinterpret_cast<uint4*>((__nv_bfloat16*)p.dq_part + (size_t)prow * D + c * 8) = v;
          }
        }
      }
    }
    t_cur = t_nxt; t_nxt = t_nn; lse_cur = lse_nxt; delta_cur = delta_nxt; gate_cur = gate_nxt;
  }

  if (lt == 0) bulk_wait_all();
  tc_fence_before();
  if (__syncthreads_or(*s_abort)) {
    // Give-up path: dK / dV are not written.  Each group's issuing thread waits (bounded) for the
    // gather still on its way into shared memory and for the MMAs it has issued; then the tensor
    // memory goes back.
    if (lt == 0) {
      if (grp == 0) mbar_wait_drain(bar_kv, 0);
      if (g_pending) mbar_wait_drain(bar_g, phase);
      tc_commit(bar_drain);
      mbar_wait_drain(bar_drain, 0);
    }
    tc_fence_before();
    __syncthreads();
    if (tid < 32) tmem_dealloc(tmem, kTmemCols);
    return;
  }
  // ---- dK^T, dV^T: lane = d, column = key; group 0 writes dV, group 1 writes dK ---------------
  tc_fence_after();
  if (half == 0) {
    const uint32_t col = grp == 0 ? kColDV : kColDK;
    const int d = row;
#pragma unroll
    for (int hc = 0; hc < 2; ++hc) {
      uint32_t r32[32];
      tmem_ld32(lane_base + col + hc * 32, r32);
      tmem_wait_ld();
      if (d < D) {
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          const int key = key0 + hc * 32 + c;
          if (key < p.Lk) {
            const size_t o = ((size_t)bh * p.Lk + key) * D + d;
            if (split) atomicAdd((grp == 0 ? p.dv_acc : p.dk_acc) + o, __uint_as_float(r32[c]));
            else (grp == 0 ? p.dv : p.dk)[o] = __float2bfloat16_rn(__uint_as_float(r32[c]));
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid < 32) tmem_dealloc(tmem, kTmemCols);
}

// ---- the same backward with the issuing taken out of the compute groups ---------------------------
// Roles: producer warps fill a ring of Q / dO tiles, one warp issues whichever batch of MMAs is ready next (dP and S of
// a tile that has landed; dV and dK of a tile whose P / dS are written, which give its dO and Q back one after the other;
// dQ behind them), eight compute warps (two per TMEM lane quadrant, half of the key columns each) turn S, dP into P, dS,
// and four warps move dQ from TMEM to a staging tile (the tile's P / dS, which the MMAs are done with) and send it off.
// Each hand-over is an mbarrier with a bounded wait, and each resource is a ring of its own: Q / dO stages, S / dP
// columns, P / dS tiles, dQ columns.
//
// What bounds it.  At D = 128 shared memory: the five products read 224 KB of operands per row tile, the gathered rows,
// P / dS and the staging tile add 160 KB, 3.1 k cycles at 128 bytes a clock; the 36 MMAs take 2.4 k by themselves (65 to
// 70 each, N = 64 or 128 alike).  A row tile takes 3.8 k; with groups that did their own tile's dQ between two tiles'
// arithmetic it was 4.7 k.  At D = 64 (112 + 80 KB, 1.4 k of MMAs) a selection tile takes as long as its gather: 64 to 84
// boxes for groups of 4 and 3, and a warp gets one out every 65 cycles, so seven warps do it (8 x 4096 tokens, 12 heads of
// 64: 604 us, 658 with three; copies of 16 bytes by all lanes instead: 746; with masks as bits 520).  That leaves 96 registers a thread, which
// costs the compute warps more than it gives where the rows are consecutive or two slabs come in one box: three
// producers there.  D = 64 computes dV^T and dK^T in one product, [dO | Q]^T [P | dS] (their tiles are neighbours): the two
// off-diagonal quarters are wasted, but the operands are read once, 8 KB a step instead of 12.
// The issuing warp shares its scheduler with compute warps (mma_ss_by, tc_common.cuh): issued by one thread of it the
// MMAs came out every 85 to 100 cycles.  Sending dQ from registers straight to global memory (32 bytes a lane) took
// 10.8 ms instead of 9.3 at 8 x 32768 tokens, 16 heads of 128: its stores hold up those of P and dS.
constexpr int kB2Compute = 8;     // compute warps
constexpr int kB2Dq = 4;          // dQ warps; then the producers and one MMA warp

// kThreeTerm: selection on 16- and 32-token blocks, whose results are fp32 arithmetic rounded once.  P and dS go to
// the tensor cores as three bf16 terms each, all 24 bits of the fp32 values (two more of each of the three products they
// enter), the dQ partials stay fp32, a block listed twice counts twice and what comes out non-finite is done again row by
// row (sel_row.cuh).  P and dS take 96 KB of a slot, so one slot fits.  The whole op on 16-token blocks, forward + backward (2 x 1024 tokens, 16 heads of 128, 8 blocks a
// list): selection backward with its plan and dQ sum 199 us (then a pass of 345) against 799 on the CUDA cores (182 with two terms), forward
// 42 against 360, the pass 302 against 1300.
template <int D, bool kThreeTerm, bool kGather> struct Bwd2 {
  static constexpr int kSlabs = D / 64;
  static constexpr int kTerms = kThreeTerm ? 3 : 1;
  static constexpr int kProducers = kGather ? 7 : 3;
  static constexpr int kThreads = (kB2Compute + kB2Dq + kProducers + 1) * 32;
  static constexpr int kStages = kThreeTerm ? (D == 64 ? 2 : 1) : (D == 64 ? 3 : 2);    // Q / dO tiles in shared memory
  static constexpr int kSets = kThreeTerm ? 1 : (D == 64 ? 3 : 2);                      // P / dS tiles
  static constexpr int kScores = kStages > 1 ? 2 : 1;                                   // S / dP column sets
  static constexpr int kDqBufs = D == 64 ? 2 : 1;                                       // dQ column sets
  static constexpr int kKVBytes = kKeys * 128 * kSlabs;
  static constexpr int kRowBytes = kRows * 128 * kSlabs;            // Q or dO
  static constexpr int kStageBytes = 2 * kRowBytes;                 // dO, Q
  static constexpr int kSetBytes = 2 * kTerms * kPBytes;            // P, dS (and P, dS: further terms)
  static constexpr int kBars = 2 + 4 * kStages + kScores + 2 * kSets + 2 * kDqBufs;
  static constexpr size_t kSmem = 2 * kKVBytes + (size_t)kStages * kStageBytes + (size_t)kSets * kSetBytes + 256 /*barriers*/ +
                                  128 * 4 /*partial rows of a ragged tile*/ + 1024 /*alignment slack*/;
};

// dK and dV of one work item in scalar fp32, into acc [dV, dK][64 keys][D] in shared memory, for a tile whose sums are
// not finite (three-term selection).  A warp has four keys, their K and V rows and their sums in registers, and goes
// through the rows.
template <int D>
__device__ __noinline__ void sel_tile_dkdv(const BwdArgs& p, float* acc, int bh, int j, int pair_first, int n_rows) {
  constexpr int N = D / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = bh / p.Hkv, hkv = bh % p.Hkv, key0 = j * kKeys, c0 = 4 * warp;
  if (c0 < kKeys) {
    const bool repeats = ld_plain(&p.plan.hdr->repeats) != 0ull;
    float k[4][N], v[4][N], dk[4][N], dv[4][N];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const size_t at = ((size_t)bh * p.Lk + min(key0 + c0 + c, p.Lk - 1)) * D + lane + 32 * e;
        k[c][e] = to_float(p.k[at]);
        v[c][e] = to_float(p.v[at]);
        dk[c][e] = dv[c][e] = 0.f;
      }
    int pair_l = 0;
    long long row_l = 0;
    float lse2_l = 0.f, delta_l = 0.f;
#pragma unroll 1
    for (int r = 0; r < n_rows; ++r) {
      // a lane fetches what 32 rows need before their vectors: one trip to memory for them all
      if ((r & 31) == 0) {
        const int rr = min(r + lane, n_rows - 1);
        pair_l = ld_plain(p.plan.pairs + pair_first + rr / p.G);
        row_l = (b * p.Hq + hkv * p.G + rr % p.G) * (long long)p.T + (pair_l & (int)kPairPosMask);
        lse2_l = ld_plain(p.lse + row_l) * kLog2e - (p.row_scale ? __log2f(ld_plain(p.row_scale + row_l)) : 0.f);
        delta_l = ld_plain(p.delta + row_l);
      }
      const int pair = __shfl_sync(0xffffffffu, pair_l, r & 31);
      const int t = pair & (int)kPairPosMask;
      if (!(((uint32_t)pair >> (kPairPosBits + (c0 >> 4))) & 1u) || key0 + c0 > t) continue;
      const long long row = __shfl_sync(0xffffffffu, row_l, r & 31);
      const float lse2 = __shfl_sync(0xffffffffu, lse2_l, r & 31), delta = __shfl_sync(0xffffffffu, delta_l, r & 31);
      const float times = repeats ? (float)times_listed(p.block_idx + ((size_t)bh * p.T + t) * p.S, p.S, (key0 + c0) / p.block_size) : 1.f;
      float q[N], g[N];
#pragma unroll
      for (int e = 0; e < N; ++e) {
        q[e] = to_float(p.q[row * D + lane + 32 * e]);
        g[e] = to_float(p.d_o[row * D + lane + 32 * e]);
      }
      float x[4], y[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        x[c] = y[c] = 0.f;
#pragma unroll
        for (int e = 0; e < N; ++e) {
          x[c] = fmaf(q[e], k[c][e], x[c]);
          y[c] = fmaf(g[e], v[c][e], y[c]);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          x[c] += __shfl_xor_sync(0xffffffffu, x[c], o);
          y[c] += __shfl_xor_sync(0xffffffffu, y[c], o);
        }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float pr = times * exp2f(fmaf(x[c], p.scale_log2, -lse2));
        const float ds = pr * (y[c] - delta) * p.scale;
        if (key0 + c0 + c <= t) {                          // what is not attended may be infinite or NaN
#pragma unroll
          for (int e = 0; e < N; ++e) {
            dv[c][e] = fmaf(pr, g[e], dv[c][e]);
            dk[c][e] = fmaf(ds, q[e], dk[c][e]);
          }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int e = 0; e < N; ++e) {
        acc[(c0 + c) * D + lane + 32 * e] = dv[c][e];
        acc[(kKeys + c0 + c) * D + lane + 32 * e] = dk[c][e];
      }
  }
  __syncthreads();
}

// 32 columns of a row's dQ against one key tile in scalar fp32 (three-term selection, result not finite).
template <int D>
__device__ __noinline__ void sel_row_dq(const BwdArgs& p, float* out, int bh, int head, int pair, int key0, int col0) {
  const int t = pair & (int)kPairPosMask;
  const size_t row = ((size_t)(bh / p.Hkv) * p.Hq + head) * p.T + t;
  const float gate = p.row_scale ? p.row_scale[row] : 1.f;
  const float lse2 = p.lse[row] * kLog2e - __log2f(gate), delta = p.delta[row];
  const int32_t* list = p.block_idx + ((size_t)bh * p.T + t) * p.S;
  float acc[32];
#pragma unroll
  for (int e = 0; e < 32; ++e) acc[e] = 0.f;
#pragma unroll 1
  for (int c = 0; c < kKeys && key0 + c <= t; ++c) {
    if (!(((uint32_t)pair >> (kPairPosBits + (c >> 4))) & 1u)) continue;
    const size_t key = ((size_t)bh * p.Lk + key0 + c) * D;
    const float x = dot_rows<D>(p.q + row * D, p.k + key), y = dot_rows<D>(p.d_o + row * D, p.v + key);
    const float pr = (float)times_listed(list, p.S, (key0 + c) / p.block_size) * exp2f(fmaf(x, p.scale_log2, -lse2));
    const float ds = pr * (y - delta) * p.scale;
    add32_row(ds, p.k + key + col0, acc);
  }
#pragma unroll
  for (int e = 0; e < 32; ++e) out[e] = acc[e];
}

template <int D, bool kCluster, bool kThreeTerm, bool kGather>
__global__ void __launch_bounds__(Bwd2<D, kThreeTerm, kGather>::kThreads, 1)
tc_bwd2_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
               const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
               const __grid_constant__ CUtensorMap tm_q_run, const __grid_constant__ CUtensorMap tm_do_run,
               const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ BwdArgs p) {
  using L = Bwd2<D, kThreeTerm, kGather>;
  constexpr int kSlabs = L::kSlabs, kStages = L::kStages, kSets = L::kSets, kScores = L::kScores, kDqBufs = L::kDqBufs;
  constexpr int kKVBytes = L::kKVBytes, kProducers = L::kProducers, kThreads = L::kThreads;
  constexpr uint32_t kTmemCols = 512;
  // scores i: S at 128 i, dP at 128 i + 64; then dV^T and dK^T: at D = 128 64 columns each, at D = 64
  // the diagonal quarters of one 128 x 128 product (dV^T: lanes 0-63, columns 0-63; dK^T: lanes 64-127,
  // columns 64-127); then dQ
  constexpr uint32_t kColDV = 256, kColDK = kColDV + 64, kColDQ = 384;
  constexpr uint32_t kIdescS = idesc_bf16(128, kKeys, 0, 0);
  constexpr uint32_t kIdescT = idesc_bf16(128, D == 64 ? 128 : kKeys, 1, 1);
  constexpr uint32_t kIdescDQ = idesc_bf16(128, D, 0, 1);

  extern __shared__ uint8_t smem_raw[];
  chain_wait();
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sK = smem;
  uint8_t* sV = sK + kKVBytes;
  uint8_t* sRow = sV + kKVBytes;                  // [kStages] dO, Q
  uint8_t* sPds = sRow + kStages * L::kStageBytes;    // [kSets] P, dS
  uint64_t* bars = (uint64_t*)(sPds + kSets * L::kSetBytes);
  uint64_t* bar_kv = bars + 0;
  uint64_t* bar_drain = bars + 1;
  uint64_t* do_full = bars + 2;                   // [kStages] dO has landed
  uint64_t* q_full = do_full + kStages;           // [kStages] Q has landed
  uint64_t* do_free = q_full + kStages;           // [kStages] the dV MMAs are done: dO may be refilled
  uint64_t* q_free = do_free + kStages;           // [kStages] the dK MMAs are done: Q may be refilled
  uint64_t* sp_full = q_free + kStages;           // [kScores] S / dP are in TMEM
  uint64_t* pds_full = sp_full + kScores;         // [kSets] P / dS are in shared memory, S / dP have been read (256 arrivals)
  uint64_t* pds_free = pds_full + kSets;          // [kSets] dQ has left its staging tile: P / dS may be written
  uint64_t* acc_full = pds_free + kSets;          // [kDqBufs] all MMAs of the tile are done
  uint64_t* dq_read = acc_full + kDqBufs;         // [kDqBufs] dQ has left TMEM (128 arrivals)
  uint32_t* s_tmem = (uint32_t*)(bars + L::kBars);
  volatile int* s_abort = (volatile int*)(s_tmem + 1);
  uint32_t* s_prow = (uint32_t*)(bars + 32);      // [128] partial row of each tile row (ragged tile)
  static_assert(L::kBars * 8 + 8 <= 256, "barrier region");

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // one key tile (or selection work item) per cluster of csize CTAs, which share its row tiles out
  const int csize = kCluster ? p.csize : 1, rank = kCluster ? (int)blockIdx.x % csize : 0;
  const int work = kCluster ? (int)blockIdx.x / csize : (int)blockIdx.x;
  int4 item = make_int4((int)blockIdx.y, work, 0, 1);
  if (p.kind == 2) {
    if (work % p.plan.max_items >= p.plan.n_items[work / p.plan.max_items]) return;
    item = p.plan.items[work];
  }
  const int j = item.y;                              // key tile
  const int bh = item.x;
  const int b = bh / p.Hkv, hkv = bh % p.Hkv;
  const int key0 = j * kKeys;

  // ---- the queries that attend this key tile ---------------------------------------------
  int t_lo = 0, n_q = 0, pair_base = 0;
  if (p.kind == 0) {
    t_lo = key0;
    n_q = min(p.T - 1, key0 + kKeys - 1 + p.window - 1) - t_lo + 1;
  } else if (p.kind == 1) {
    t_lo = key0 * p.window + p.block_size - 1;       // first query that sees summary key0 (window: the stride)
    n_q = p.T - t_lo;
  } else {
    pair_base = ld_plain(p.plan.offsets + (size_t)bh * (p.n_ktiles + 1) + j);
    n_q = ld_plain(p.plan.offsets + (size_t)bh * (p.n_ktiles + 1) + j + 1) - pair_base;
  }
  n_q = max(n_q, 0);
  const int n_rt_all = (n_q + p.nq - 1) / p.nq;
  const int chunk = p.kind == 2 ? kSelChunkTiles : ((int)gridDim.z > 1 ? p.split_chunk : n_rt_all);
  const int rt_first = p.kind == 2 ? item.z : (int)blockIdx.z * chunk;
  const int rt_last = min(n_rt_all, rt_first + chunk);
  const bool split = p.kind == 2 ? item.w > 1 : gridDim.z > 1;
  const int per_cta = kCluster ? (max(0, rt_last - rt_first) + csize - 1) / csize : rt_last - rt_first;
  const int rt_begin = rt_first + rank * per_cta;
  int n_tiles = max(0, min(rt_last, rt_begin + per_cta) - rt_begin);

  if (rt_last <= rt_first) {
    if (!split && n_rt_all == 0) {   // nobody attends these keys: their gradients are zero
      for (int i = tid; i < kKeys * D / 8; i += blockDim.x) {
        const int key = key0 + i / (D / 8);
        if (key < p.Lk) {
          const size_t off = ((size_t)bh * p.Lk + key) * D + (i % (D / 8)) * 8;
          if ((((uintptr_t)p.dk | (uintptr_t)p.dv) & 15) == 0) {
            *reinterpret_cast<uint4*>(p.dk + off) = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(p.dv + off) = make_uint4(0, 0, 0, 0);
          } else {                       // a caller's tensor may start anywhere
            for (int e = 0; e < 8; ++e) p.dk[off + e] = p.dv[off + e] = __float2bfloat16_rn(0.f);
          }
        }
      }
    }
    return;
  }

  if (tid == 0) {
    int bad = (*(volatile int*)p.status != 0) ? 1 : 0;
    if ((size_t)((uint8_t*)(s_prow + 128) - smem_raw) > L::kSmem) {
      atomicOr(p.status, 256);   // the shared-memory window is less aligned than assumed
      bad = 1;
    }
    *s_abort = bad;
    mbar_init(bar_kv, 1);
    mbar_init(bar_drain, 1);
    for (int s = 0; s < 4 * kStages; ++s) mbar_init(do_full + s, 1);
    for (int s = 0; s < kScores; ++s) mbar_init(sp_full + s, 1);
    for (int s = 0; s < kSets; ++s) { mbar_init(pds_full + s, kB2Compute * 32); mbar_init(pds_free + s, 1); }
    for (int s = 0; s < kDqBufs; ++s) { mbar_init(acc_full + s, 1); mbar_init(dq_read + s, kB2Dq * 32); }
    fence_barrier_init();
    prefetch_tensormap(&tm_k); prefetch_tensormap(&tm_v);
    prefetch_tensormap(&tm_q); prefetch_tensormap(&tm_do); prefetch_tensormap(&tm_dq);
  }
  __syncthreads();
  if (*s_abort) {
    if (!kCluster) return;
    n_tiles = 0;             // the cluster's other CTAs read this one's flag at the end: it stays
  }
  uint32_t tmem = 0;
  const bool producer = warp >= kB2Compute + kB2Dq && warp < kB2Compute + kB2Dq + kProducers;
  if (!producer) {           // the first loads are on their way meanwhile
    // rows past nq * G of a tile are never loaded, and dV / dK sum over all 128: keep them zero
    if (warp < kB2Compute + kB2Dq) {
      // (merged boxes lay the two slabs of a row side by side: one run of 256-byte rows)
      const int r0 = p.nq * p.G, row_bytes = p.merged ? 256 : 128;
      const int n = (kRows - r0) * row_bytes / 16, runs = 2 * L::kRowBytes / (kRows * row_bytes);
      for (int i = tid; i < runs * kStages * n; i += (kB2Compute + kB2Dq) * 32) {
        const int part = i / n;                        // (stages lie one behind the other)
        uint8_t* base = sRow + part * (kRows * row_bytes);
        *reinterpret_cast<uint4*>(base + r0 * row_bytes + (i % n) * 16) = make_uint4(0, 0, 0, 0);
      }
      // nor are P and dS of such rows written, nor dQ over them: times a key that is not finite anything that came of their S
      // would be NaN (zeros stored over them in the last place cost 1 to 2 % at D = 128)
      for (int i = tid; i < kSets * (L::kSetBytes / kPBytes) * (kRows - r0) * 8; i += (kB2Compute + kB2Dq) * 32)
        *reinterpret_cast<uint4*>(sPds + i / ((kRows - r0) * 8) * kPBytes + r0 * 128 + i % ((kRows - r0) * 8) * 16) = make_uint4(0, 0, 0, 0);
    }
    fence_proxy_async();
    if (warp == 0) {
      tmem_alloc(s_tmem, kTmemCols);
      tmem_relinquish();
    }
    tc_fence_before();
    named_sync_b(2, kThreads - kProducers * 32);
    tc_fence_after();
    tmem = *s_tmem;
    // dK^T / dV^T start at zero so that every MMA into them accumulates
    if (warp < 4) {
      uint32_t z[32];
#pragma unroll
      for (int c = 0; c < 32; ++c) z[c] = 0u;
      const uint32_t lb = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) tmem_st32(lb + kColDV + cc * 32, z);
      tmem_wait_st();
    }
    tc_fence_before();
    named_sync_b(2, kThreads - kProducers * 32);
    tc_fence_after();
  }

  if (producer) {
    // ---- producers: K / V once, then Q and dO of every tile.  A warp gets a TMA box out every
    // 60-100 cycles whatever its size, so the boxes of a tile are dealt out over three warps
    // (box o to warp o % 3) and, where the shape allows, one box brings both column slabs ---------
    const int pw = warp - kB2Compute - kB2Dq;
    if (pw == 0 && lane == 0) {
      mbar_expect_tx(bar_kv, 2 * kKVBytes);
#pragma unroll
      for (int s = 0; s < kSlabs; ++s) {
        tma_load_3d(sK + s * (kKeys * 128), &tm_k, bar_kv, s * 64, key0, bh);
        tma_load_3d(sV + s * (kKeys * 128), &tm_v, bar_kv, s * 64, key0, bh);
      }
    }
    const uint32_t tile_bytes = (uint32_t)(p.nq * p.G * 128 * kSlabs);     // of Q or dO
    const int per_q = p.merged ? 1 : kSlabs;         // boxes per query and tensor: one per slab unless merged
    const int n_ops = p.nq * per_q;                  // selection: the boxes of a tile, for Q and for dO
    constexpr int kRounds = (kMaxNq * kSlabs + 32 * kProducers - 1) / (32 * kProducers);
    auto box_of = [&](int r) -> int { return (r * 32 + lane) * kProducers + pw; };
    auto tq_of = [&](int k, int o) -> int {          // pair of box o of tile k (none: past T, zeros)
      const int qi = (rt_begin + k) * p.nq + o / per_q;
      return (o < n_ops && qi < n_q) ? ld_plain(p.plan.pairs + pair_base + qi) : p.T;
    };
    int tq[kRounds];
    if (p.kind == 2) {
#pragma unroll
      for (int r = 0; r < kRounds; ++r) tq[r] = tq_of(0, box_of(r));
    }
    const uint64_t pol_keep = l2_policy_evict_normal();   // gathered q / dO rows: read again by other blocks
    bool ok = true;
    int issued = 0;                                  // halves of tiles whose loads this warp has sent off
    for (int k = 0; k < n_tiles; ++k) {
      const int sb = k % kStages, u = k / kStages;
      // dO, which the dV MMAs give back before the dK MMAs do Q (dQ reads dS and K only), then Q
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint64_t* full = (half ? q_full : do_full) + sb;
        if (u > 0) ok = mbar_wait((half ? q_free : do_free) + sb, (u - 1) & 1, p.status, s_abort, 128);
        if (!(ok = __all_sync(0xffffffffu, ok))) break;       // the whole warp leaves together
        uint8_t* dst = sRow + sb * L::kStageBytes + half * L::kRowBytes;
        if (pw == 0 && lane == 0) mbar_expect_tx(full, tile_bytes);
        __syncwarp();
        if (p.kind != 2) {
          // window / compression: the tile's queries are consecutive tokens, one box per slab
          if (pw == 0 && lane == 0) {
            const int qi = (rt_begin + k) * p.nq;
            const int t0 = qi < n_q ? t_lo + qi : p.T;
#pragma unroll
            for (int s = 0; s < kSlabs; ++s)
              tma_load_3d(dst + s * (kRows * 128), half ? &tm_q_run : &tm_do_run, full, s * 64, b * p.Hq + hkv * p.G, t0);
          }
        } else {
#pragma unroll
          for (int r = 0; r < kRounds; ++r) {
            const int o = box_of(r);
            const int t_box = (int)(tq[r] & kPairPosMask);   // here: not where the load would be waited for
            if (o >= n_ops) continue;
            if (p.merged) {
              tma_load_5d_hint(dst + o * (p.G / 8) * 2048, half ? &tm_q : &tm_do, full, 0, 0, 0, t_box,
                               (b * p.Hq + hkv * p.G) >> 3, pol_keep);
            } else {
              const int qq = o / kSlabs, s = o % kSlabs;
              tma_load_3d(dst + s * (kRows * 128) + qq * p.G * 128, half ? &tm_q : &tm_do, full, s * 64,
                          b * p.Hq + hkv * p.G, t_box);
            }
          }
        }
        issued = 2 * k + half + 1;
      }
      if (!ok) break;
      if (p.kind == 2 && k + 1 < n_tiles) {
#pragma unroll
        for (int r = 0; r < kRounds; ++r) tq[r] = tq_of(k + 1, box_of(r));
      }
    }
    if (lane == 0) {
      // The loads that this warp has sent land before it goes to the teardown barrier (bounded wait on the last phase of
      // each stage), whether the CTA has given up, gives up later or not: none may be on its way when the CTA ends.
      // A stage that not every warp has sent its boxes of, or the first has not armed, runs into the limit
      mbar_wait_drain(bar_kv, 0);
      for (int h = max(0, issued - 2 * kStages); h < issued; ++h)
        mbar_wait_drain((h & 1 ? q_full : do_full) + (h >> 1) % kStages, ((h >> 1) / kStages) & 1);
    }
  } else if (warp == kB2Compute + kB2Dq + kProducers) {
    // ---- MMA issuer: whichever batch is ready next ---------------------------------------------
    {
      const uint32_t lead = elect_one(), tmem_u = uniform(tmem);
      auto seen = [](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_test_wait(bar, parity)); };
      mbar_wait(bar_kv, 0, p.status, s_abort, 32);
      __syncwarp();
      const uint32_t ka = desc_lo_kmajor(smem_u32(sK)), va = desc_lo_kmajor(smem_u32(sV));
      const uint32_t kb = desc_lo_mnmajor(smem_u32(sK), kKeys * 128);
      const uint32_t q_slab = p.merged ? 1024u : (uint32_t)(kRows * 128), q_sbo = p.merged ? 2048u : 1024u;
      int next_a = 0, next_b = 0, next_c = 0;        // next tile for S / dP, for dV / dK, for dQ
      int ga = 0, gb = 0;                            // stages of next_a and next_b
      int pb = 0, pc = 0, dc = 0;                    // P / dS set of next_b and next_c, dQ columns of next_c
      uint32_t ph_ga = 0, ph_pb = 0, ph_dc = 0;      // phases to wait for (dq_read: of its last use)
      bool dp_sent = false;                          // dP of next_a is on its way, S not yet
      long long idle_since = clock64();
      uint32_t polls = 0;
      while (next_c < n_tiles) {
        bool progressed = false;
        // (P / dS of tile next_a - kScores are written: its S / dP have been read)
        if (next_a < n_tiles && next_a < next_b + kScores) {
          const uint8_t* sDO = sRow + ga * L::kStageBytes;
          const uint32_t colS = tmem_u + (next_a % kScores) * 128, colDP = colS + 64;
          if (!dp_sent && seen(do_full + ga, ph_ga)) {
            tc_fence_after();
            const uint32_t da = desc_lo_kmajor(smem_u32(sDO));
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
              const uint32_t slab = kk >> 2, in = (kk & 3) * 32;
              mma_ss_by(lead, colDP, desc_at_sbo(da, slab * q_slab + in, q_sbo), desc_at(va, slab * (kKeys * 128) + in),
                     kIdescS, kk > 0);
            }
            dp_sent = progressed = true;
          }
          if (dp_sent && seen(q_full + ga, ph_ga)) {
            tc_fence_after();
            const uint32_t qa = desc_lo_kmajor(smem_u32(sDO + L::kRowBytes));
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
              const uint32_t slab = kk >> 2, in = (kk & 3) * 32;
              mma_ss_by(lead, colS, desc_at_sbo(qa, slab * q_slab + in, q_sbo), desc_at(ka, slab * (kKeys * 128) + in),
                     kIdescS, kk > 0);
            }
            tc_commit_by(lead, sp_full + next_a % kScores);
            ++next_a;
            if (++ga == kStages) { ga = 0; ph_ga ^= 1; }
            dp_sent = false;
            progressed = true;
          }
        }
        if (next_b < next_a && seen(pds_full + pb, ph_pb)) {
          tc_fence_after();
          const uint8_t* sDO = sRow + gb * L::kStageBytes;
          const uint8_t* sP = sPds + pb * L::kSetBytes;
          const uint8_t* sDS = sP + kPBytes;         // (three-term: P, dS, then their further terms)
#pragma unroll
          for (uint32_t term = 0; term < L::kTerms * 2 * kPBytes; term += 2 * kPBytes) {
            if (D == 64) {
              // A: the dO and Q tiles as two 64-column slabs, B: the P and dS tiles likewise
              const uint32_t da = desc_lo_mnmajor(smem_u32(sDO), L::kRowBytes);
              const uint32_t pa = desc_lo_mnmajor(smem_u32(sP), kPBytes);
#pragma unroll
              for (int kk = 0; kk < kRows / 16; ++kk)        // contraction over the 128 rows, 16 a step
                mma_ss_by(lead, tmem_u + kColDV, desc_at(da, kk * 2048), desc_at(pa, term + kk * 2048), kIdescT, 1);
            } else {
              const uint32_t da = desc_lo_mnmajor(smem_u32(sDO), q_slab);
              const uint32_t qa = desc_lo_mnmajor(smem_u32(sDO + L::kRowBytes), q_slab);
              const uint32_t pa = desc_lo_mnmajor(smem_u32(sP), 0), dsa = desc_lo_mnmajor(smem_u32(sDS), 0);
#pragma unroll
              for (int kk = 0; kk < kRows / 16; ++kk)
                mma_ss_by(lead, tmem_u + kColDV, desc_at_sbo(da, kk * 2 * q_sbo, q_sbo), desc_at(pa, term + kk * 2048), kIdescT, 1);
              if (term == (L::kTerms - 1) * 2 * kPBytes) tc_commit_by(lead, do_free + gb);
#pragma unroll
              for (int kk = 0; kk < kRows / 16; ++kk)
                mma_ss_by(lead, tmem_u + kColDK, desc_at_sbo(qa, kk * 2 * q_sbo, q_sbo), desc_at(dsa, term + kk * 2048), kIdescT, 1);
            }
          }
          if (D == 64) tc_commit_by(lead, do_free + gb);
          tc_commit_by(lead, q_free + gb);
          ++next_b;
          if (++gb == kStages) gb = 0;
          if (++pb == kSets) { pb = 0; ph_pb ^= 1; }
          progressed = true;
        }
        if (next_c < next_b && (next_c < kDqBufs || seen(dq_read + dc, ph_dc ^ 1))) {
          tc_fence_after();
          const uint32_t dsk = desc_lo_kmajor(smem_u32(sPds + pc * L::kSetBytes + kPBytes));
#pragma unroll
          for (uint32_t term = 0; term < L::kTerms * 2 * kPBytes; term += 2 * kPBytes)
#pragma unroll
            for (int kk = 0; kk < kKeys / 16; ++kk)          // contraction over the 64 keys
              mma_ss_by(lead, tmem_u + kColDQ + dc * D, desc_at(dsk, term + kk * 32), desc_at(kb, kk * 2048), kIdescDQ, term > 0 || kk > 0);
          tc_commit_by(lead, acc_full + dc);
          ++next_c;
          if (++pc == kSets) pc = 0;
          if (++dc == kDqBufs) { dc = 0; ph_dc ^= 1; }
          progressed = true;
        }
        if (progressed) {
          idle_since = clock64();
          continue;
        }
        if ((++polls & 0xffu) == 0) {
          bool leave = *s_abort != 0;
          if (!leave && *(volatile int*)p.status != 0) leave = true;
          if (!leave && clock64() - idle_since > kWaitLimitCycles) { atomicOr(p.status, 2048); leave = true; }
          if (__any_sync(0xffffffffu, leave)) { *s_abort = 1; break; }
        }
      }
      // the tensor pipe is idle before TMEM is read for dK / dV and given back, whatever happened
      tc_commit_by(lead, bar_drain);
      if (!mbar_wait(bar_drain, 0, p.status, s_abort, 4096)) mbar_wait_drain(bar_drain, 0);
    }
  } else if (warp < kB2Compute) {
    // ---- compute warps: S, dP -> P, dS, tile after tile -------------------------------------------
    // Two columns an instruction in the arithmetic around the exponentials, the same bits: selection at D = 64, 8 x 4096 tokens of 12
    // heads 528 -> 519 us, 3 x 3001 172 -> 168.5, 8192 of 16 182 -> 180.5.  Elsewhere it was slower: compression
    // at D = 64 72 -> 74, selection at D = 128, which spills then, 8.6 -> 9.1 ms (8 x 32768 tokens), key tiles shared by a cluster
    // (D = 64, 16 heads on 1, 5000 tokens 84 -> 88 us, 2048 49 -> 51; 64 on 4, 1000 tokens 78 -> 81).
    constexpr bool kPacked = D == 64 && kGather && !kCluster;
    const int quad = warp & 3, half = warp >> 2;       // TMEM lane quadrant, key-column half
    const int row = quad * 32 + lane;
    const int ql = row / p.G, g = row % p.G;
    const int head = hkv * p.G + g;
    const bool row_slot_ok = ql < p.nq;
    // query of this thread's row in tile k (selection: with the tile's column groups it attends in
    // the bits above the position), -1: no row
    auto row_query = [&](int k) -> int {
      const int qi = (rt_begin + k) * p.nq + ql;
      if (!row_slot_ok || qi >= n_q) return -1;
      if (p.kind == 2) return ld_plain(p.plan.pairs + pair_base + qi);
      return t_lo + qi;
    };
    auto row_index = [&](int t) -> size_t { return (size_t)(b * p.Hq + head) * p.T + (t & (int)kPairPosMask); };
    int t_cur = row_query(0);
    int t_nxt = n_tiles > 1 ? row_query(1) : -1;
    float lse_cur = 0.f, delta_cur = 0.f, gate_cur = 1.f;
    if (t_cur >= 0) {
      lse_cur = ld_plain(p.lse + row_index(t_cur));
      delta_cur = ld_plain(p.delta + row_index(t_cur));
      if (p.row_scale) gate_cur = ld_plain(p.row_scale + row_index(t_cur));
    }
    const bool repeats = kThreeTerm && ld_plain(&p.plan.hdr->repeats) != 0ull;
    for (int k = 0; k < n_tiles; ++k) {
      uint8_t* sP = sPds + (k % kSets) * L::kSetBytes;
      uint8_t* sDS = sP + kPBytes;
      const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16) + (k % kScores) * 128;
      const int t_nn = k + 2 < n_tiles ? row_query(k + 2) : -1;
      float lse_nxt = 0.f, delta_nxt = 0.f, gate_nxt = 1.f;
      if (t_nxt >= 0) {
        lse_nxt = ld_plain(p.lse + row_index(t_nxt));
        delta_nxt = ld_plain(p.delta + row_index(t_nxt));
        if (p.row_scale) gate_nxt = ld_plain(p.row_scale + row_index(t_nxt));
      }
      int lo = 0, hi = -1;                           // valid key columns of this row: one range [lo, hi]
      uint32_t groups = 0x3u;                        // and, for selection, the 16-column groups of this thread's half
      if (t_cur >= 0) {
        if (p.kind == 0) {
          lo = max(0, t_cur - p.window + 1 - key0);
          hi = min(kKeys - 1, t_cur - key0);
        } else if (p.kind == 1) {
          hi = min(kKeys - 1, cmp_visible(t_cur, p.block_size, p.window, p.Lk) - 1 - key0);
        } else {
          hi = min(kKeys - 1, (t_cur & (int)kPairPosMask) - key0);
          groups = ((uint32_t)t_cur >> (kPairPosBits + 2 * half)) & 0x3u;
        }
      }
      // gate * p = 2^(s * scale * log2e - lse * log2e + log2(gate)): the branch's dO is gate * dO, so dV takes
      // (gate p)^T dO; dS = scale * gate * p * (dP - delta), the constant factors folded once per row
      const float lse2 = lse_cur * kLog2e - __log2f(gate_cur);
      const float dscale = p.scale, ddelta = delta_cur * p.scale;
      // the columns of this thread's half that are attended, a bit each: all of them away from the diagonal.  Rows past
      // nq * G of a tile count as attending all, and their rows of P and dS stay the zeros they start as: two
      // of them in the last quarter of every tile of three heads had its warps mask every element, 1.7 k cycles a tile
      // behind the others
      const int lo_h = min(max(lo - half * 32, 0), 32), hi_h = min(max(hi + 1 - half * 32, 0), 32);
      uint32_t attended = (hi_h == 32 ? ~0u : (1u << hi_h) - 1u) & ~((lo_h == 32) ? ~0u : (1u << lo_h) - 1u);
      if (!(groups & 1u)) attended &= 0xffff0000u;
      if (!(groups & 2u)) attended &= 0x0000ffffu;
      if (!row_slot_ok) attended = ~0u;
      const bool all_cols = attended == ~0u && !repeats;
      float times[2] = {1.f, 1.f};                   // how often the row's list names the blocks of its column groups
      if (kThreeTerm && repeats && t_cur >= 0) {
        const int32_t* list = p.block_idx + ((size_t)bh * p.T + (t_cur & (int)kPairPosMask)) * p.S;
#pragma unroll
        for (int e = 0; e < 2; ++e) times[e] = (float)times_listed(list, p.S, (key0 + half * 32 + 16 * e) / p.block_size);
      }
      bool ok = mbar_wait(sp_full + k % kScores, (k / kScores) & 1, p.status, s_abort, 64);
      if (!__all_sync(0xffffffffu, ok)) break;                 // the whole warp leaves together
      tc_fence_after();
      {
        uint32_t rs[32], rp[32];
        tmem_ld32(lane_base + half * 32, rs);
        tmem_ld32(lane_base + 64 + half * 32, rp);
        tmem_wait_ld();
        uint32_t pp[16], pd[16];
        // the values as bf16; three-term: they stay in fp32 where S and dP were, for the terms to be taken off
        auto put = [&](int c2, float p0, float p1, float d0, float d1) {
          if (kThreeTerm) {
            rs[c2 * 2] = __float_as_uint(p0); rs[c2 * 2 + 1] = __float_as_uint(p1);
            rp[c2 * 2] = __float_as_uint(d0); rp[c2 * 2 + 1] = __float_as_uint(d1);
            return;
          }
          pp[c2] = pack_bf16(p0, p1);
          pd[c2] = pack_bf16(d0, d1);
        };
        if (kPacked && __all_sync(0xffffffffu, all_cols)) {
          const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2), neg_lse2 = pack_f32x2(-lse2, -lse2);
          const uint64_t dscale2 = pack_f32x2(dscale, dscale), neg_ddelta2 = pack_f32x2(-ddelta, -ddelta);
#pragma unroll
          for (int c2 = 0; c2 < 16; ++c2) {
            float x0, x1, y0, y1;
            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(rs[c2 * 2]), __uint_as_float(rs[c2 * 2 + 1])), scale2, neg_lse2), x0, x1);
            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(rp[c2 * 2]), __uint_as_float(rp[c2 * 2 + 1])), dscale2, neg_ddelta2), y0, y1);
            const float p0 = ex2(x0), p1 = ex2(x1);
            put(c2, p0, p1, p0 * y0, p1 * y1);
          }
        } else if (!kPacked && __all_sync(0xffffffffu, all_cols)) {
#pragma unroll
          for (int c2 = 0; c2 < 16; ++c2) {
            const float p0 = ex2(fmaf(__uint_as_float(rs[c2 * 2]), p.scale_log2, -lse2));
            const float p1 = ex2(fmaf(__uint_as_float(rs[c2 * 2 + 1]), p.scale_log2, -lse2));
            put(c2, p0, p1, p0 * fmaf(__uint_as_float(rp[c2 * 2]), dscale, -ddelta),
                p1 * fmaf(__uint_as_float(rp[c2 * 2 + 1]), dscale, -ddelta));
          }
        } else {
#pragma unroll
          for (int c2 = 0; c2 < 16; ++c2) {
            float pv[2], dv[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const bool in = (attended >> (c2 * 2 + e)) & 1u;
              float pr = in ? ex2(fmaf(__uint_as_float(rs[c2 * 2 + e]), p.scale_log2, -lse2)) : 0.f;
              if (kThreeTerm) pr *= times[c2 >> 3];
              pv[e] = pr;
              dv[e] = pr * fmaf(__uint_as_float(rp[c2 * 2 + e]), dscale, -ddelta);
              if (kThreeTerm && !in) dv[e] = 0.f;      // (dP of a key that is not attended may be infinite)
            }
            put(c2, pv[0], pv[1], dv[0], dv[1]);
          }
        }
        // the P / dS tiles double as the dQ staging tile: the store of the set's last tile has read it
        if (k >= kSets) ok = mbar_wait(pds_free + k % kSets, ((k / kSets) - 1) & 1, p.status, s_abort, 64);
        if (!__all_sync(0xffffffffu, ok)) break;
        const uint32_t p_row = smem_u32(sP) + row * 128, ds_row = smem_u32(sDS) + row * 128;
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
          const uint32_t chunk16 = (uint32_t)((half * 4 + k4) ^ (row & 7)) << 4;
          if (kThreeTerm) {
            auto terms = [&](uint32_t at, uint32_t* v) {         // eight fp32 values; what a term leaves is exact
#pragma unroll
              for (int term = 0; term < L::kTerms; ++term) {
                uint32_t b[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  b[e] = pack_bf16(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));
                  v[2 * e] = __float_as_uint(__uint_as_float(v[2 * e]) - __uint_as_float(b[e] << 16));
                  v[2 * e + 1] = __float_as_uint(__uint_as_float(v[2 * e + 1]) - __uint_as_float(b[e] & 0xffff0000u));
                }
                if (row_slot_ok) st_shared_v4(at + term * 2 * kPBytes, b[0], b[1], b[2], b[3]);
              }
            };
            terms(p_row + chunk16, rs + k4 * 8);
            terms(ds_row + chunk16, rp + k4 * 8);
            continue;
          }
          if (row_slot_ok) {
            st_shared_v4(p_row + chunk16, pp[k4 * 4], pp[k4 * 4 + 1], pp[k4 * 4 + 2], pp[k4 * 4 + 3]);
            st_shared_v4(ds_row + chunk16, pd[k4 * 4], pd[k4 * 4 + 1], pd[k4 * 4 + 2], pd[k4 * 4 + 3]);
          }
        }
      }
      fence_proxy_async();
      tc_fence_before();
      mbar_arrive(pds_full + k % kSets);
      t_cur = t_nxt; t_nxt = t_nn; lse_cur = lse_nxt; delta_cur = delta_nxt; gate_cur = gate_nxt;
    }
  } else {
    // ---- dQ of every tile: TMEM -> bf16 -> staging tile (its P / dS, which the MMAs are done with) -> partial buffer ----
    const int quad = warp & 3, lt = tid - kB2Compute * 32;
    const int row = quad * 32 + lane;
    const int ql = row / p.G, g = row % p.G;
    const bool row_slot_ok = ql < p.nq;
    for (int k = 0; k < n_tiles; ++k) {
      const int dc = k % kDqBufs;
      const int i = rt_begin + k, qi = i * p.nq + ql;
      uint8_t* stage = sPds + (k % kSets) * L::kSetBytes;
      const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16) + kColDQ + dc * D;
      const bool ok = mbar_wait(acc_full + dc, (k / kDqBufs) & 1, p.status, s_abort, 128);
      __syncwarp();
      tc_fence_after();
#pragma unroll
      for (int cc = 0; cc < D / 32; ++cc) {
        const int col0 = cc * 32;
        uint32_t r32[32];
        tmem_ld32(lane_base + col0, r32);
        tmem_wait_ld();
        if (cc == D / 32 - 1) {            // dQ is in registers: the columns' next dQ may land
          tc_fence_before();
          mbar_arrive(dq_read + dc);
        }
        if (kThreeTerm) {                    // fp32 staging: slabs of 128 rows x 32 columns
          float z = 0.f;                   // x * 0: 0 or NaN
#pragma unroll
          for (int e = 0; e < 32; ++e) z = fmaf(__uint_as_float(r32[e]), 0.f, z);
          if (z != 0.f && row_slot_ok && qi < n_q) {
            const int head = hkv * p.G + g, pair = ld_plain(p.plan.pairs + pair_base + qi);
            const size_t at = (size_t)(b * p.Hq + head) * p.T + (pair & (int)kPairPosMask);
            const float lse2 = ld_plain(p.lse + at) * kLog2e - (p.row_scale ? __log2f(ld_plain(p.row_scale + at)) : 0.f);
            const float ddelta = ld_plain(p.delta + at) * p.scale;
            if (lse2 == lse2 && ddelta == ddelta) {      // (NaN statistics: NaN in every column, here as there)
              float again[32];
              sel_row_dq<D>(p, again, bh, head, pair, key0, col0);
#pragma unroll
              for (int e = 0; e < 32; ++e) r32[e] = __float_as_uint(again[e]);
            }
          }
          __syncwarp();
          const uint32_t rbase = smem_u32(stage) + (col0 >> 5) * (kRows * 128) + row * 128;
#pragma unroll
          for (int c = 0; c < 8; ++c)
            if (row_slot_ok)
              st_shared_v4(rbase + (((uint32_t)c ^ (uint32_t)(row & 7)) << 4), r32[c * 4], r32[c * 4 + 1], r32[c * 4 + 2], r32[c * 4 + 3]);
          continue;
        }
#pragma unroll
        for (int v4 = 0; v4 < 4; ++v4) {
          const uint32_t ch = (uint32_t)((col0 >> 3) + v4);
          if (row_slot_ok)
            st_shared_v4(smem_u32(stage) + (ch >> 3) * (kRows * 128) + row * 128 + (((ch & 7) ^ (row & 7)) << 4),
                         pack_bf16(__uint_as_float(r32[v4 * 8 + 0]), __uint_as_float(r32[v4 * 8 + 1])),
                         pack_bf16(__uint_as_float(r32[v4 * 8 + 2]), __uint_as_float(r32[v4 * 8 + 3])),
                         pack_bf16(__uint_as_float(r32[v4 * 8 + 4]), __uint_as_float(r32[v4 * 8 + 5])),
                         pack_bf16(__uint_as_float(r32[v4 * 8 + 6]), __uint_as_float(r32[v4 * 8 + 7])));
        }
      }
      const bool full_tile = (i + 1) * p.nq <= n_q;
      if (!full_tile) {
        uint32_t prow = 0xffffffffu;
        if (row_slot_ok && qi < n_q) {
          if (p.kind == 2) {
            prow = (uint32_t)((size_t)(pair_base + qi) * p.G + g);
          } else {
            const int slot = p.kind == 0 ? j % p.n_slots : j;
            prow = (uint32_t)((((size_t)bh * p.T + t_lo + qi) * p.n_slots + slot) * p.G + g);
          }
        }
        s_prow[row] = prow;
      }
      fence_proxy_async();
      if (named_or_b(1, kB2Dq * 32, !ok)) break;               // the whole group leaves together
      if (full_tile) {
        // its rows are consecutive in the partial buffer: one TMA store per slab
        if (lt == 0) {
          const int slot = p.kind == 2 ? 0 : (p.kind == 0 ? j % p.n_slots : j);
          const int mid = p.kind == 2 ? pair_base + i * p.nq : t_lo + i * p.nq;
          const int outer = p.kind == 2 ? 0 : bh;
          constexpr int kParts = kThreeTerm ? D / 32 : kSlabs;
#pragma unroll
          for (int sl = 0; sl < kParts; ++sl)
            tma_store_5d_hint(&tm_dq, stage + sl * (kRows * 128), sl * (D / kParts), 0, slot, mid, outer, l2_policy_evict_first());
          bulk_commit();
          bulk_wait_read();
          mbar_arrive(pds_free + k % kSets);
        }
      } else {   // the ragged last tile: whole rows out by hand, 16 bytes a lane
        constexpr int kChunks = kThreeTerm ? D / 4 : D / 8;
        constexpr int kRowsPerPass = kB2Dq * 32 / kChunks;
        const int c = lt % kChunks;
        for (int r = lt / kChunks; r < kRows; r += kRowsPerPass) {
          const uint32_t prow = s_prow[r];
          if (prow != 0xffffffffu) {
            const uint4 v = *reinterpret_cast<const uint4*>(stage + (c >> 3) * (kRows * 128) + r * 128 +
                                                            (((c & 7) ^ (r & 7)) << 4));
            *reinterpret_cast<uint4*>((char*)p.dq_part + ((size_t)prow * kChunks + c) * 16) = v;
          }
        }
      }
    }
  }

  // ---- dK^T, dV^T: lane = d, column = key; warps 0-3 have dV, 4-7 dK.  Through shared memory, so that they leave in
  // rows of a key -----------------------------------------------------------------------------------
  __syncthreads();           // the MMA thread has seen the tensor pipe drain (bar_drain)
  tc_fence_after();
  float* s_acc = reinterpret_cast<float*>(sRow);       // [dV, dK][64 keys][D], over the stages
  float z = 0.f;             // three-term: x * 0 of every sum, 0 or NaN
  if (warp < 8 && !*s_abort) {
    const int which = warp >> 2, quad = warp & 3;
    // D = 64: dV^T sits in lanes 0-63, dK^T in lanes 64-127
    if (D == 128 || (quad >> 1) == which) {
      const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16) + (which ? kColDK : kColDV);
      const int d = (D == 128 ? quad : quad & 1) * 32 + lane;
#pragma unroll
      for (int hc = 0; hc < 2; ++hc) {
        uint32_t r32[32];
        tmem_ld32(lane_base + hc * 32, r32);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          s_acc[(which * kKeys + hc * 32 + c) * D + d] = __uint_as_float(r32[c]);
          if (kThreeTerm) z = fmaf(__uint_as_float(r32[c]), 0.f, z);
        }
      }
    }
  }
  // sums that are not finite are formed again, leaving out what a row does not attend
  if (kThreeTerm && __syncthreads_or(z != 0.f)) {
    const int first = rt_begin * p.nq, rows = max(0, min(n_tiles * p.nq, n_q - first)) * p.G;
    sel_tile_dkdv<D>(p, s_acc, bh, j, pair_base + first, rows);
  }
  // the CTAs of a cluster add their sums, each a share of the keys, in rank order
  int aborted = 0;
  if (kCluster) {
    cluster_sync();
    for (int r = 0; r < csize; ++r) aborted |= ld_peer_s32(const_cast<int*>(s_abort), r);
  } else {
    __syncthreads();
    aborted = *s_abort;
  }
  if (!aborted) {
    const int n = 2 * kKeys * D / 4 / csize;           // float4s per CTA
    for (int i = tid; i < n; i += kThreads) {
      const int e = (rank * n + i) * 4;
      float4 acc;
      if (kCluster) {
        acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = 0; r < csize; ++r) {
          const float4 v = ld_peer_f32x4(s_acc + e, r);
          acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
      } else {
        acc = *reinterpret_cast<const float4*>(s_acc + e);
      }
      const int which = e / (kKeys * D), key = key0 + (e / D) % kKeys, d = e % D;
      if (key < p.Lk) {
        const size_t o = ((size_t)bh * p.Lk + key) * D + d;
        if (split) {
          float* dst = (which == 0 ? p.dv_acc : p.dk_acc) + o;
          if (p.acc_stride) *reinterpret_cast<float4*>(dst + blockIdx.z * p.acc_stride) = acc;
          else { atomicAdd(dst, acc.x); atomicAdd(dst + 1, acc.y); atomicAdd(dst + 2, acc.z); atomicAdd(dst + 3, acc.w); }
        } else {
          __nv_bfloat16* dst = (which == 0 ? p.dv : p.dk) + o;
          if (((uintptr_t)dst & 7) == 0) {
            *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(acc.x, acc.y), pack_bf16(acc.z, acc.w));
          } else {                                     // a caller's tensor may start anywhere
            dst[0] = __float2bfloat16_rn(acc.x); dst[1] = __float2bfloat16_rn(acc.y);
            dst[2] = __float2bfloat16_rn(acc.z); dst[3] = __float2bfloat16_rn(acc.w);
          }
        }
      }
    }
  }
  if (kCluster) cluster_sync();            // nobody leaves while its memory is read
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

// Selection blocks whose row tiles were split over several work items collect dK / dV in the fp32 accumulators.  The rows of
// those blocks are cleared before the backward kernel and turned into the bf16 outputs after it, a CTA to a key tile.
// Where the call has a delta kernel its first CTAs clear them.  Bound by latency: 16 bytes a thread and access (8192 tokens, 16
// heads of 64: the two kernels of scalar loops took 13.1 us, now 6.4 and 0.9 in the delta kernel; 8 x 32768 of 128 88 -> 55).
struct SplitTiles {
  const int32_t* offsets;                // null: no block is split
  float *dk_acc, *dv_acc;
  int n_ktiles, units, nq, Lk, D;
  // elements of key tile `tile` (of all units) if it is split, else 0; base: its first element
  __device__ __forceinline__ int elements(unsigned tile, size_t* base) const {
    const int bh = (int)(tile / (unsigned)n_ktiles), j = (int)(tile % (unsigned)n_ktiles);
    const int32_t* at = offsets + (size_t)bh * (n_ktiles + 1) + j;
    const int n_rt = (ld_plain(at + 1) - ld_plain(at) + nq - 1) / nq;
    *base = ((size_t)bh * Lk + (size_t)j * kKeys) * D;
    return n_rt <= kSelChunkTiles ? 0 : min(kKeys, Lk - j * kKeys) * D;       // one work item: written directly
  }
  __device__ __forceinline__ void clear(unsigned tile) const {
    size_t base;
    const int n = elements(tile, &base);
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = threadIdx.x * 4; i < n; i += blockDim.x * 4) {
      *reinterpret_cast<float4*>(dk_acc + base + i) = z;
      *reinterpret_cast<float4*>(dv_acc + base + i) = z;
    }
  }
};

// delta[b,h,t] = sum_d dO * O (fp32), D / 8 lanes to a row, one 16-byte vector of each: bound by the pass over both (16
// heads x 8192 rows of 64: 6 us, 18 with a warp to a row).
template <int D>
__global__ void delta_kernel(const __nv_bfloat16* d_o, const __nv_bfloat16* o,
                             float* delta, size_t rows, bool vec, const SplitTiles split) {
  chain_wait();
  chain_go();
  if (split.offsets && blockIdx.x < (unsigned)(split.n_ktiles * split.units)) split.clear(blockIdx.x);
  constexpr int kLanes = D / 8;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x, row = i / kLanes;
  float s = 0.f;
  if (row < rows && !vec) {                          // tensors off a 16-byte boundary
    for (int e = 0; e < 8; ++e) s = fmaf(to_float(d_o[i * 8 + e]), to_float(o[i * 8 + e]), s);
  } else if (row < rows) {
    const uint4 x = reinterpret_cast<const uint4*>(d_o)[i], y = reinterpret_cast<const uint4*>(o)[i];
    const uint32_t a[4] = {x.x, x.y, x.z, x.w}, c[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
    for (int e = 0; e < 4; ++e)
      s = fmaf(__uint_as_float(a[e] << 16), __uint_as_float(c[e] << 16),
               fmaf(__uint_as_float(a[e] & 0xffff0000u), __uint_as_float(c[e] & 0xffff0000u), s));
  }
#pragma unroll
  for (int w = kLanes / 2; w > 0; w >>= 1) s += __shfl_xor_sync(0xffffffffu, s, w);
  if (row < rows && i % kLanes == 0) delta[row] = s;
}

// dq of the whole op in one pass: the partials of the compression, selection and window branches
// of query (bh, t) are added in fp32 and rounded once.  A branch whose buffer is null is absent.
struct Reduce3Args {
  const __nv_bfloat16* part_cmp; int slots_cmp, Lk_cmp, cmp_len, cmp_stride;
  int shift_win;               // log2 of the keys of a window tile
  const void* part_slc; const int32_t* pair_of_slot; int S;     // fp32 where the kernel is kF32
  const __nv_bfloat16* part_win; int slots_win, window;
  const float* acc;            // fp32 accumulator [units][T][G][D] holding the window + compression part, or null
  __nv_bfloat16* dq;
  int B, Hq, Hkv, T, G;
};

// One thread adds up 8 columns of a query's dQ for HG heads (g, g + G / HG, ...): the heads of a
// query share the partial rows, so their index loads and address arithmetic are paid once.  The
// kernel moves 32 GB at the benchmark shape and was held back by its instruction count, not by
// memory, when every thread served a single head.
template <int D, int HG, bool kF32>
__global__ void __launch_bounds__(256, 3)
dq_reduce3_kernel(const Reduce3Args a) {
  chain_wait();
  constexpr int kVec = D / 8;
  const int Gp = a.G / HG;                               // head groups per query
  const size_t gid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t total = (size_t)a.B * a.Hkv * a.T * Gp * kVec;
  if (gid >= total) return;
  const int v = (int)(gid % kVec);
  const int g = (int)((gid / kVec) % Gp);
  const int t = (int)((gid / ((size_t)kVec * Gp)) % a.T);
  const size_t bh = gid / ((size_t)kVec * Gp * a.T);
  float acc[HG][8];
#pragma unroll
  for (int h = 0; h < HG; ++h)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[h][e] = 0.f;
  const size_t row_elems = (size_t)a.G * D;              // elements of one partial row (all heads)
  const size_t in_row = (size_t)g * D + v * 8;           // this thread's first head inside a row
  const size_t head_step = (size_t)Gp * D;               // to its next head
  // Rows per trip and CTAs per SM (three: 80 registers, which hold the loads of a bf16 trip, and of half as many fp32
  // rows; without the bound the compiler took 70 and issued them in turns).  fp32 rows in trips as long spilled in
  // groups of 3 and took the same time: 33 us for 4 x 2000 tokens of 12 heads of 64 and 8 slots, 6 TB/s.  An empty place costs as many instructions as a row (a window
  // of 512 touches 9 key tiles, a query sees few tiles of summaries).  Two heads at 8 x 32768 tokens: trips of
  // 8 rows in 5.24 ms, of 4 in 4.90 (5.33 with five CTAs, which spill), unbounded 5.76; groups of 3 at 8 x 4096:
  // 203 us, unbounded 257.
  constexpr int kTripSel = HG == 1 ? 8 : 4, kTripWin = HG == 3 ? 3 : kTripSel, kTripCmp = HG == 3 ? 2 : kTripSel;
  // a trip of N partial rows: their loads are issued before the first is added
  auto add_rows = [&](const __nv_bfloat16* part, const auto& rows) {
    constexpr int kTrip = sizeof(rows) / sizeof(rows[0]);
    uint4 u[kTrip][HG];
#pragma unroll
    for (int k = 0; k < kTrip; ++k) {
      const __nv_bfloat16* src = part + (size_t)(rows[k] >= 0 ? rows[k] : 0) * row_elems + in_row;
#pragma unroll
      for (int h = 0; h < HG; ++h)
        u[k][h] = rows[k] >= 0 ? __ldcs(reinterpret_cast<const uint4*>(src + h * head_step))
                               : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int k = 0; k < kTrip; ++k)
#pragma unroll
      for (int h = 0; h < HG; ++h) {
        const uint32_t w[4] = {u[k][h].x, u[k][h].y, u[k][h].z, u[k][h].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {                    // bf16 -> fp32 is a shift
          acc[h][2 * e] += __uint_as_float(w[e] << 16);
          acc[h][2 * e + 1] += __uint_as_float(w[e] & 0xffff0000u);
        }
      }
  };
  const long long qrow = (long long)(bh * a.T + t);
  if (a.acc) {
#pragma unroll
    for (int h = 0; h < HG; ++h) {
      const float4* src = reinterpret_cast<const float4*>(a.acc + (size_t)qrow * row_elems + in_row + h * head_step);
      const float4 lo = src[0], hi = src[1];
      acc[h][0] = lo.x; acc[h][1] = lo.y; acc[h][2] = lo.z; acc[h][3] = lo.w;
      acc[h][4] = hi.x; acc[h][5] = hi.y; acc[h][6] = hi.z; acc[h][7] = hi.w;
    }
  }
  if (a.part_slc) {
    const int32_t* ps = a.pair_of_slot + (size_t)qrow * a.S;
    constexpr int kTrip = kF32 ? kTripSel / 2 : kTripSel;      // fp32 rows are twice as wide
    for (int s0 = 0; s0 < a.S; s0 += kTrip) {
      long long rows[kTrip];
#pragma unroll
      for (int k = 0; k < kTrip; ++k) rows[k] = s0 + k < a.S ? (long long)ld_plain(ps + s0 + k) : -1;
      if (!kF32) {
        add_rows((const __nv_bfloat16*)a.part_slc, rows);
        continue;
      }
      float4 f[kTrip][HG][2];
#pragma unroll
      for (int k = 0; k < kTrip; ++k) {
        const float* src = (const float*)a.part_slc + (size_t)(rows[k] >= 0 ? rows[k] : 0) * row_elems + in_row;
#pragma unroll
        for (int h = 0; h < HG; ++h)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            f[k][h][e] = rows[k] >= 0 ? __ldcs(reinterpret_cast<const float4*>(src + h * head_step) + e) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int k = 0; k < kTrip; ++k)
#pragma unroll
        for (int h = 0; h < HG; ++h)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            acc[h][4 * e] += f[k][h][e].x; acc[h][4 * e + 1] += f[k][h][e].y;
            acc[h][4 * e + 2] += f[k][h][e].z; acc[h][4 * e + 3] += f[k][h][e].w;
          }
    }
  }
  if (a.part_win) {
    const int first = max(0, t - a.window + 1) >> a.shift_win, last = t >> a.shift_win;
    for (int j0 = first; j0 <= last; j0 += kTripWin) {
      long long rows[kTripWin];
#pragma unroll
      for (int k = 0; k < kTripWin; ++k) rows[k] = j0 + k <= last ? qrow * a.slots_win + (j0 + k) % a.slots_win : -1;
      add_rows(a.part_win, rows);
    }
  }
  if (a.part_cmp) {
    const int n_vis = cmp_visible(t, a.cmp_len, a.cmp_stride, a.Lk_cmp);
    const int last = n_vis > 0 ? (n_vis - 1) >> 6 : -1;
    for (int j0 = 0; j0 <= last; j0 += kTripCmp) {
      long long rows[kTripCmp];
#pragma unroll
      for (int k = 0; k < kTripCmp; ++k) rows[k] = j0 + k <= last ? qrow * a.slots_cmp + j0 + k : -1;
      add_rows(a.part_cmp, rows);
    }
  }
  const int b = (int)(bh / a.Hkv), hkv = (int)(bh % a.Hkv);
#pragma unroll
  for (int h = 0; h < HG; ++h) {
    uint4 u;
    u.x = pack_bf16(acc[h][0], acc[h][1]); u.y = pack_bf16(acc[h][2], acc[h][3]);
    u.z = pack_bf16(acc[h][4], acc[h][5]); u.w = pack_bf16(acc[h][6], acc[h][7]);
    *reinterpret_cast<uint4*>(a.dq + (((size_t)b * a.Hq + hkv * a.G + g + h * Gp) * a.T + t) * D + v * 8) = u;
  }
}

static Reduce3Args reduce_args(const AttnArgs& a, void* dq) {
  Reduce3Args r = {};
  r.slots_cmp = r.slots_win = 1;
  r.shift_win = 6;
  r.dq = (__nv_bfloat16*)dq;
  r.B = a.B; r.Hq = a.Hq; r.Hkv = a.Hkv; r.T = a.T; r.G = a.Hq / a.Hkv;
  return r;
}

// f32: the selection's partials are fp32 (three-term)
static int reduce_launch(const Reduce3Args& r, int D, bool f32, const char* name, cudaStream_t st) {
  const int hg = r.G % 2 == 0 ? 2 : (r.G % 3 == 0 ? 3 : 1);   // heads of a query served by one thread
  const size_t nthreads = (size_t)r.B * r.Hkv * r.T * (r.G / hg) * (D / 8);
  if (nthreads == 0) return NSA_OK;
  const unsigned grid = (unsigned)((nthreads + 255) / 256);
  KernelScope ks(name, st);
  auto go = [&](auto kernel) -> int { NSA_CUDA_OK(launch_chained(kernel, grid, 256, 0, st, r)); return NSA_OK; };
  auto by_heads = [&](auto f32) -> int {
    constexpr bool kF32 = decltype(f32)::value;
    if (D == 128)
      return hg == 2 ? go(dq_reduce3_kernel<128, 2, kF32>) : hg == 3 ? go(dq_reduce3_kernel<128, 3, kF32>) : go(dq_reduce3_kernel<128, 1, kF32>);
    return hg == 2 ? go(dq_reduce3_kernel<64, 2, kF32>) : hg == 3 ? go(dq_reduce3_kernel<64, 3, kF32>) : go(dq_reduce3_kernel<64, 1, kF32>);
  };
  const int rc = f32 ? by_heads(std::true_type()) : by_heads(std::false_type());
  if (rc != NSA_OK) return rc;
  NSA_LAUNCH_OK("dq_reduce3_kernel");
  return NSA_OK;
}

__global__ void __launch_bounds__(256) sel_split_clear_kernel(const SplitTiles x) {
  chain_wait();
  chain_go();
  x.clear(blockIdx.x);
}
__global__ void __launch_bounds__(256) sel_split_finish_kernel(const SplitTiles x, __nv_bfloat16* dk, __nv_bfloat16* dv, bool vec) {
  chain_wait();
  chain_go();
  size_t base;
  const int n = x.elements(blockIdx.x, &base);
#pragma unroll 4
  for (int i = threadIdx.x * 4; i < n; i += 256 * 4) {
    const float4 k = __ldcs(reinterpret_cast<const float4*>(x.dk_acc + base + i)), v = __ldcs(reinterpret_cast<const float4*>(x.dv_acc + base + i));
    const uint2 uk = make_uint2(pack_bf16(k.x, k.y), pack_bf16(k.z, k.w)), uv = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
    if (vec) {
      *reinterpret_cast<uint2*>(dk + base + i) = uk;
      *reinterpret_cast<uint2*>(dv + base + i) = uv;
    } else {                                           // a caller's tensor may start anywhere
      const __nv_bfloat16 *ek = reinterpret_cast<const __nv_bfloat16*>(&uk), *ev = reinterpret_cast<const __nv_bfloat16*>(&uv);
      for (int e = 0; e < 4; ++e) { dk[base + i + e] = ek[e]; dv[base + i + e] = ev[e]; }
    }
  }
}

// dK and dV of the compression branch from the accumulators of up to kOrderedChunks chunks of row tiles, in a fixed order, so
// that they come out the same on every run: the last chunk of a key tile, then the others as they come.  (Any
// order is as exact.  This one is what fp32 atomics mostly gave before, and was kept so that results stayed as they were:
// the gradient of the key pooling's position parameters is the rounding of these sums, and 1e-2 of it moves with the
// order.  More chunks, beyond 192 row tiles of queries, still meet in atomics.)
constexpr int kOrderedChunks = 4;
__global__ void __launch_bounds__(256)
cmp_chunks_kernel(const float* __restrict__ dk_acc, const float* __restrict__ dv_acc, __nv_bfloat16* __restrict__ dk,
                  __nv_bfloat16* __restrict__ dv, size_t n8, size_t stride, int T, int Lk, int D, int cmp_len, int cmp_stride,
                  int nq, int chunk) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  const float* src = (blockIdx.y ? dv_acc : dk_acc) + i * 8;
  const int key0 = (int)((i * 8 / D) % Lk) & ~(kKeys - 1);
  const int n_q = max(0, T - (key0 * cmp_stride + cmp_len - 1));
  const int chunks = ((n_q + nq - 1) / nq + chunk - 1) / chunk;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int k = 0; k < chunks; ++k) {
    const float4* row = reinterpret_cast<const float4*>(src + (size_t)(k == 0 ? chunks - 1 : k - 1) * stride);
    const float4 a = __ldg(row), b = __ldg(row + 1);
    acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
    acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
  }
  *reinterpret_cast<uint4*>((blockIdx.y ? dv : dk) + i * 8) =
      make_uint4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]), pack_bf16(acc[4], acc[5]), pack_bf16(acc[6], acc[7]));
}

static const char* const kBwdNames[3] = {"tc_bwd_win", "tc_bwd_cmp", "tc_bwd_slc"};
static const char* const kRedNames[3] = {"dq_reduce_win", "dq_reduce_cmp", "dq_reduce_slc"};

struct BwdPlan {
  bool wide;                 // window: tiles of 128 keys (tc_bwd_wide.cu)
  int n_ktiles, n_slots, nq, n_splits, split_chunk;
  int csize;                 // CTAs that share the row tiles of one key tile
  bool sel_split;            // selection: a key tile that every query lists would be more than one work item
  size_t off_acc;
  size_t cap_pairs;          // selection: pairs the CSR may hold
  SelPlanLayout layout;      // selection
  size_t off_delta, off_part, off_plan, total;
};

}  // namespace tc
int get_option_merged_boxes();   // api.cu
int get_option_bwd_kernel();
namespace tc {

// Window with more tiles of 64 keys than SMs: tiles of 128 (tc_bwd_wide.cu).  A tile of 128 takes 1.5 to 1.7 times as long
// as one of 64, so it pays where those would need a second wave, and not before: at 32 tiles of 128 keys (64 of 64, in
// clusters) the window took 45 us for 1024 tokens of 16 heads of 64 and 62 for 2048 of 8 heads of 128, 25 and 33 with tiles
// of 64; from 128 tiles on it takes 0.65 to 0.7 of their time.  Compression keeps tiles of 64: the gradient of its key
// pooling's position parameters is the rounding of P and dS, which the products here round in another order.
static bool use_wide(const AttnArgs& a) {
  return a.kind == 0 && a.Lk == a.T && !a.dq_acc && (a.dq || a.wide_dq) && get_option_bwd_kernel() == 1 &&
         (long long)a.B * a.Hkv * ((a.T + kKeys - 1) / kKeys) > sm_count();
}

static BwdPlan plan_bwd(const AttnArgs& a) {
  BwdPlan pl;
  const int G = a.Hq / a.Hkv;
  pl.nq = kRows / G;
  const size_t units = (size_t)a.B * a.Hkv;
  pl.wide = use_wide(a);
  pl.n_ktiles = (a.Lk + kKeys - 1) / kKeys;        // (the wide kernel has its own)
  size_t part_rows;
  if (a.kind == 2) {
    pl.n_slots = a.S;
    pl.cap_pairs = units * a.T * a.S;
    part_rows = pl.cap_pairs;
  } else {
    pl.n_slots = a.kind != 0 ? pl.n_ktiles : pl.wide ? (std::min(a.window, a.T) + kWideKeys - 2) / kWideKeys + 1
                                                     : (std::min(a.window, a.T) + kKeys - 2) / kKeys + 1;
    pl.cap_pairs = 0;
    part_rows = a.dq_acc ? 0 : units * a.T * pl.n_slots;   // accumulator mode: no partial buffer
  }
  size_t off = 0;
  pl.off_delta = off; off += align_up((size_t)a.B * a.Hq * a.T * sizeof(float), 256);
  pl.off_part = off; off += align_up(part_rows * G * a.D * (a.three_term ? 4 : 2), 256);
  pl.off_plan = off;
  if (a.kind == 2) {
    pl.layout = sel_plan_layout((int)units, a.T, a.S, pl.nq);
    off += pl.layout.total;
  }
  // Fewer key tiles than SMs: a cluster of CTAs shares the row tiles of each and adds its dK / dV through
  // distributed shared memory, as long as a CTA keeps 8 row tiles or so (a CTA costs about as much as
  // two before its first).  The line is 20 CTAs above one per SM: key tiles are unequal (the last ones have
  // few queries left), so the CTAs over the line start as the short ones end.  At 76 to 84 key tiles
  // (152 to 168 CTAs in pairs) window and selection take 40 to 61 and 77 to 107 us in pairs, 49 to 66 and 102
  // to 153 without (D of 64 and 128, groups of 4).  More CTAs than that gain nothing, and clusters
  // leave SMs of a GPC over, so big problems do without.  Compression does too: its sums keep one
  // order, row tiles in turn within a chunk and chunks as cmp_chunks_kernel adds them, since the
  // gradient of the key pooling's position parameters is the rounding of those sums (tc.cu), and where a problem is small it
  // runs beside the other branches.
  const int max_rt = a.kind == 0 ? (std::min(a.window, 1 << 30) + kKeys - 2 + pl.nq) / pl.nq : (a.T + pl.nq - 1) / pl.nq;
  const int item_rt = a.kind == 2 ? (max_rt < kSelChunkTiles ? max_rt : kSelChunkTiles) : max_rt;
  const long long base = (long long)units * pl.n_ktiles;
  pl.csize = 1;
  // Three-term row tiles take three times as long as others beside the same cost of a CTA, and early key tiles have most
  // of them: up to two CTAs per SM, as long as a CTA keeps enough of them beside the one it shares its SM with: 8 (D = 64: 10) up to one and a half per SM,
  // beyond that 12 (20).  Key tiles / row tiles of the longest (alone | pairs | fours | eights, us), D = 128: 128 / 8
  // 62 | 68, 128 / 16 103 | 96, 128 / 32 152 | 125 | 130, 96 / 8 60 | 59, 96 / 48 203 | 111 | 111, 64 / 16 100 | 62 | 66, 64 / 32 152 | 84 | 77, 64 / 64
  // 210 | 113 | 76 | 107, 32 / 32 148 | 84 | 51 | 58, 37 / 128 357 | 189 | 103 | 80; D = 64: 128 / 8 41 | 47, 128 / 16 66 | 68, 128 / 32 99 | 78, 96 / 8
  // 39 | 41, 96 / 12 53 | 49, 88 / 11 48 | 43, 64 / 16 64 | 41 | 49, 64 / 32 74 | 44 | 45, 64 / 64 130 | 72 | 53 | 79, 32 / 32 94 | 54 | 35 | 45,
  // 24 / 48 113 | 65 | 41 | 33, 37 / 128 269 | 144 | 80 | 62.
  auto pays = [&](int csize) {
    const long long ctas = base * csize * 2, sms = sm_count();
    if (ctas <= sms + 20) return item_rt >= 8 * csize;
    if (!a.three_term || ctas > 2 * sms) return false;
    return item_rt >= (2 * ctas <= 3 * sms ? (a.D == 128 ? 8 : 10) : a.D == 128 ? 12 : 20) * csize;
  };
  while (a.kind != 1 && !a.dq_acc && !pl.wide && pl.csize < 8 && pays(pl.csize)) pl.csize *= 2;
  // compression: a few key tiles are attended by (almost) every query; they go in chunks of 48 row
  // tiles whose dK / dV meet in fp32 accumulators
  pl.n_splits = 1;
  pl.split_chunk = 0;
  pl.off_acc = off;
  if (a.kind == 1) {
    pl.split_chunk = 48;
    if (max_rt > pl.split_chunk) {
      pl.n_splits = (max_rt + pl.split_chunk - 1) / pl.split_chunk;
      const size_t n_acc = pl.n_splits <= kOrderedChunks ? (size_t)pl.n_splits : 1;
      off += 2 * align_up(n_acc * a.B * a.Hkv * a.Lk * a.D * sizeof(float), 256);
    }
  }
  // selection: blocks split over several work items use the same accumulators (launches and memory that up to
  // kSelChunkTiles row tiles of queries, 4096 tokens at groups of 4, a call does without)
  pl.sel_split = a.kind == 2 && max_rt > kSelChunkTiles;
  if (pl.sel_split) off += 2 * align_up((size_t)a.B * a.Hkv * a.Lk * a.D * sizeof(float), 256);
  pl.total = off;
  return pl;
}

// the kernels with tiles of 64 keys
static int bwd_narrow(const AttnArgs& a, const BwdArgs& p, const BwdPlan& pl, bool roles, cudaStream_t st) {
  const int G = p.G;
  CUtensorMap tm_k, tm_v, tm_q, tm_do;
  int rc = make_map(&tm_k, a.k, a.D, a.Lk, a.B * a.Hkv, kKeys, 1);
  if (rc == NSA_OK) rc = make_map(&tm_v, a.v, a.D, a.Lk, a.B * a.Hkv, kKeys, 1);
  if (rc == NSA_OK) rc = p.merged ? make_map_query_both_slabs(&tm_q, a.q, a.T, a.B * a.Hq, G)
                                  : make_map_query_rows(&tm_q, a.q, a.D, a.T, a.B * a.Hq, G);
  if (rc == NSA_OK) rc = p.merged ? make_map_query_both_slabs(&tm_do, a.d_o, a.T, a.B * a.Hq, G)
                                  : make_map_query_rows(&tm_do, a.d_o, a.D, a.T, a.B * a.Hq, G);
  CUtensorMap tm_q_run, tm_do_run;
  if (rc == NSA_OK) rc = make_map_query_rows(&tm_q_run, a.q, a.D, a.T, a.B * a.Hq, G, pl.nq);
  if (rc == NSA_OK) rc = make_map_query_rows(&tm_do_run, a.d_o, a.D, a.T, a.B * a.Hq, G, pl.nq);
  CUtensorMap tm_dq, tm_dqacc;
  if (rc == NSA_OK && p.dq_acc_mode) {
    rc = make_map_dq_acc(&tm_dqacc, a.dq_acc, a.D, G, (size_t)a.T, (size_t)a.B * a.Hkv, pl.nq);
    tm_dq = tm_dqacc;        // the partial-tile map is not used in this mode
  } else if (rc == NSA_OK) {
    rc = a.kind == 2 ? make_map_partial(&tm_dq, p.dq_part, a.D, G, 1, pl.cap_pairs ? pl.cap_pairs : 1, 1, pl.nq, a.three_term)
                     : make_map_partial(&tm_dq, p.dq_part, a.D, G, pl.n_slots, a.T, (size_t)a.B * a.Hkv, pl.nq);
    tm_dqacc = tm_dq;        // likewise
  }
  if (rc != NSA_OK) return rc;
  const size_t smem = bwd_smem_bytes(a.D);
  dim3 grid(pl.n_ktiles, a.B * a.Hkv, pl.n_splits);
  if (a.kind == 2)
    grid = dim3((unsigned)((size_t)a.B * a.Hkv * pl.layout.max_items));
  if (roles) {
    KernelScope ks(branch_name(kBwdNames, a.kind), st);
    grid.x *= (unsigned)pl.csize;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (pl.csize > 1) {
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)pl.csize;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      cfg.numAttrs = 1;
    }
    if (a.kind == 2 && !a.row_dot) {       // a call of its own: the short kernels before it, and no other branch beside it
      attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    auto go = [&](auto d, auto three_term, auto gather) -> int {
      constexpr int D = decltype(d)::value;
      constexpr bool kThreeTerm = decltype(three_term)::value, kGather = decltype(gather)::value;
      using L = Bwd2<D, kThreeTerm, kGather>;
      const auto kernel = pl.csize > 1 ? tc_bwd2_kernel<D, true, kThreeTerm, kGather> : tc_bwd2_kernel<D, false, kThreeTerm, kGather>;
      cfg.blockDim = dim3(L::kThreads);
      cfg.dynamicSmemBytes = L::kSmem;
      NSA_CUDA_OK(func_smem((const void*)kernel, L::kSmem));
      NSA_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, tm_k, tm_v, tm_q, tm_do, tm_q_run, tm_do_run, tm_dq, p));
      return NSA_OK;
    };
    auto by_form = [&](auto d) -> int {
      if (a.three_term) return go(d, std::true_type(), std::false_type());
      // a box per query and slab: 64 to 256 of them a row tile, more than three warps get out in the time of its MMAs.  Seven warps
      // against three, selection backward: D = 64, 8 x 4096 tokens of 12 / 4 heads 604 us against 658; D = 128, where the compute warps' 96 registers
      // count for more, 8192 tokens of 16 / 4 heads 272 against 327, 2 x 3001 of 8 / 4 152 against 233, 512 of 12 / 4 27.0 against 30.6
      if (a.kind == 2 && !p.merged) return go(d, std::false_type(), std::true_type());
      return go(d, std::false_type(), std::false_type());
    };
    rc = a.D == 128 ? by_form(std::integral_constant<int, 128>()) : by_form(std::integral_constant<int, 64>());
    if (rc != NSA_OK) return rc;
  } else if (a.D == 128) {
    NSA_CUDA_OK(func_smem((const void*)tc_bwd_kernel<128>, smem));
    KernelScope ks(branch_name(kBwdNames, a.kind), st);
    tc_bwd_kernel<128><<<grid, 512, smem, st>>>(tm_k, tm_v, tm_q_run, tm_do_run, tm_dq, tm_dqacc, p);
  } else {
    NSA_CUDA_OK(func_smem((const void*)tc_bwd_kernel<64>, smem));
    KernelScope ks(branch_name(kBwdNames, a.kind), st);
    tc_bwd_kernel<64><<<grid, 512, smem, st>>>(tm_k, tm_v, tm_q_run, tm_do_run, tm_dq, tm_dqacc, p);
  }
  NSA_LAUNCH_OK("tc_bwd_kernel");
  return NSA_OK;
}

}  // namespace tc

int tc_sel_plan_build(const AttnArgs& a, void* plan, size_t plan_bytes, cudaStream_t st);   // tc_fwdpair.cu

size_t tc_attn_bwd_workspace(const AttnArgs& a) { return tc::plan_bwd(a).total; }

int tc_attn_bwd(const AttnArgs& a, void* ws, size_t ws_bytes, cudaStream_t st) {
  using namespace tc;
  const BwdPlan pl = plan_bwd(a);
  if (!ws || ws_bytes < pl.total) {
    set_error("backward workspace too small: need %zu bytes", pl.total);
    return NSA_ERR_WORKSPACE;
  }
  char* base = (char*)ws;
  const int G = a.Hq / a.Hkv;
  BwdArgs p;
  p.q = (const __nv_bfloat16*)a.q;
  p.k = (const __nv_bfloat16*)a.k;
  p.v = (const __nv_bfloat16*)a.v;
  p.block_idx = a.block_idx;
  p.S = a.S;
  p.d_o = (const __nv_bfloat16*)a.d_o;
  p.lse = a.lse;
  p.delta = a.row_dot ? a.row_dot : (float*)(base + pl.off_delta);
  p.row_scale = a.row_scale;
  p.dk = (__nv_bfloat16*)a.dk_acc;     // the API passes the dk / dv outputs through these fields
  p.dv = (__nv_bfloat16*)a.dv_acc;
  p.dq_part = base + pl.off_part;
  p.plan = SelPlan{};
  p.status = device_status_ptr();
  if (!p.status) { set_error("device status word unavailable"); return NSA_ERR_CUDA; }
  p.B = a.B; p.Hq = a.Hq; p.Hkv = a.Hkv; p.T = a.T; p.Lk = a.Lk; p.G = G; p.nq = pl.nq;
  p.kind = a.kind; p.window = a.kind == 0 ? std::min(a.window, a.T) : a.window; p.block_size = a.block_size;
  p.n_ktiles = pl.n_ktiles; p.n_slots = pl.n_slots;
  p.dq_acc_mode = (a.dq_acc && a.kind != 2) ? 1 : 0;
  p.merged = (a.kind == 2 && a.D == 128 && G % 8 == 0 && get_option_merged_boxes()) ? 1 : 0;
  p.scale = a.scale; p.scale_log2 = a.scale * kLog2e;
  p.split_chunk = pl.split_chunk;
  p.csize = pl.csize;
  const size_t n_kv = (size_t)a.B * a.Hkv * a.Lk * a.D;
  const bool roles = (get_option_bwd_kernel() == 1 || a.kind == 2) && !p.dq_acc_mode;   // compute groups relieved of the issuing
  const bool ordered = roles && pl.n_splits > 1 && pl.n_splits <= kOrderedChunks && aligned16(p.dk, p.dv);
  p.acc_stride = ordered ? n_kv : 0;
  p.dk_acc = (float*)(base + pl.off_acc);
  p.dv_acc = (float*)(base + pl.off_acc + align_up((ordered ? (size_t)pl.n_splits : 1) * n_kv * sizeof(float), 256));
  if (pl.n_splits > 1 && !ordered)
    NSA_CUDA_OK(cudaMemsetAsync(base + pl.off_acc, 0, 2 * align_up(n_kv * sizeof(float), 256), st));

  if (a.kind == 2) {
    const void* plan_mem = a.sel_plan;
    if (!plan_mem) {
      plan_mem = base + pl.off_plan;
      int rc = tc_sel_plan_build(a, base + pl.off_plan, pl.layout.total, st);
      if (rc != NSA_OK) return rc;
    } else if (!a.dq && !a.plan_kept) {      // nsa_dq_reduce3 looks the pair map up in the workspace
      NSA_CUDA_OK(cudaMemcpyAsync(base + pl.off_plan + pl.layout.pos, (const char*)plan_mem + pl.layout.pos,
                                  pl.cap_pairs * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
    }
    p.plan = sel_plan_at(plan_mem, pl.layout);
  }
  const SplitTiles split = {pl.sel_split ? p.plan.offsets : nullptr, p.dk_acc, p.dv_acc, pl.n_ktiles, a.B * a.Hkv, pl.nq, a.Lk, a.D};
  const unsigned n_split = (unsigned)(pl.n_ktiles * a.B * a.Hkv);
  const size_t rows = (size_t)a.B * a.Hq * a.T;
  if (!a.row_dot) {
    // (at least two CTAs for each key tile: its first ones clear the accumulators as well)
    KernelScope ks("delta_kernel", st);
    const unsigned dgrid = (unsigned)((rows * (a.D / 8) + 255) / 256);
    const auto *d_o = (const __nv_bfloat16*)a.d_o, *o = (const __nv_bfloat16*)a.o;
    NSA_CUDA_OK(launch_chained(a.D == 128 ? delta_kernel<128> : delta_kernel<64>, std::max(dgrid, split.offsets ? n_split : 0u), 256, 0,
                               st, d_o, o, (float*)(base + pl.off_delta), rows, aligned16(d_o, o), split));
    NSA_LAUNCH_OK("delta_kernel");
  } else if (split.offsets) {
    KernelScope ks("sel_split_clear_kernel", st);
    NSA_CUDA_OK(launch_chained(sel_split_clear_kernel, n_split, 256, 0, st, split));
    NSA_LAUNCH_OK("sel_split_clear_kernel");
  }
  int rc = NSA_OK;
  if (pl.wide) {
    WideArgs w;
    w.lse = p.lse; w.delta = p.delta; w.row_scale = p.row_scale;
    w.dk = p.dk; w.dv = p.dv; w.dq_part = (__nv_bfloat16*)p.dq_part;
    w.status = p.status;
    w.Hq = a.Hq; w.Hkv = a.Hkv; w.T = a.T; w.G = G; w.nq = pl.nq;
    w.window = std::min(a.window, a.T); w.n_slots = pl.n_slots;
    w.scale = p.scale; w.scale_log2 = p.scale_log2;
    rc = bwd_wide_launch(a, w, branch_name(kBwdNames, a.kind), st);
  } else {
    rc = bwd_narrow(a, p, pl, roles, st);
  }
  if (rc != NSA_OK) return rc;
  if (pl.sel_split) {
    KernelScope ks("sel_split_finish_kernel", st);
    NSA_CUDA_OK(launch_chained(sel_split_finish_kernel, n_split, 256, 0, st, split, p.dk, p.dv,
                               (((uintptr_t)p.dk | (uintptr_t)p.dv) & 7) == 0));
    NSA_LAUNCH_OK("sel_split_finish_kernel");
  }
  if (ordered) {
    KernelScope ks("cmp_chunks_kernel", st);
    cmp_chunks_kernel<<<dim3((unsigned)((n_kv / 8 + 255) / 256), 2), 256, 0, st>>>(p.dk_acc, p.dv_acc, p.dk, p.dv, n_kv / 8, n_kv, a.T,
                                                                                  a.Lk, a.D, a.block_size, a.window, pl.nq,
                                                                                  pl.split_chunk);
    NSA_LAUNCH_OK("cmp_chunks_kernel");
  } else if (pl.n_splits > 1) {
    int rc2 = cast_f32_to(p.dk_acc, p.dk, n_kv, NSA_DTYPE_BF16, st);
    if (rc2 == NSA_OK) rc2 = cast_f32_to(p.dv_acc, p.dv, n_kv, NSA_DTYPE_BF16, st);
    if (rc2 != NSA_OK) return rc2;
  }
  if (!a.dq) return NSA_OK;   // the partials stay in the workspace (or the accumulator) for tc_dq_reduce3
  Reduce3Args r = reduce_args(a, a.dq);
  if (a.kind == 0) { r.part_win = (const __nv_bfloat16*)p.dq_part; r.slots_win = pl.n_slots; r.shift_win = pl.wide ? 7 : 6; r.window = a.window; }
  else if (a.kind == 1) {
    r.part_cmp = (const __nv_bfloat16*)p.dq_part; r.slots_cmp = pl.n_slots;
    r.Lk_cmp = a.Lk; r.cmp_len = a.block_size; r.cmp_stride = a.window;
  } else { r.part_slc = p.dq_part; r.pair_of_slot = p.plan.pair_of_slot; r.S = a.S; }
  return reduce_launch(r, a.D, a.three_term, branch_name(kRedNames, a.kind), st);
}

// dq of the whole op from the three branch workspaces (each written by tc_attn_bwd with a null
// dq) and / or the fp32 accumulator: `base` carries B, Hq, Hkv, T, D; a null workspace means the
// branch is absent (or sits in the accumulator).  pos: the pair map of the selection branch where it
// is not the one inside ws_slc.
int tc_dq_reduce3(const AttnArgs& base, int Lk_cmp, int cmp_len, int cmp_stride, int S, int block_size,
                  int window, const void* ws_cmp, const void* ws_slc, const void* ws_win,
                  const int32_t* pos, const float* dq_acc, void* dq, cudaStream_t st) {
  using namespace tc;
  Reduce3Args r = reduce_args(base, dq);
  r.acc = dq_acc;
  r.Lk_cmp = Lk_cmp; r.cmp_len = cmp_len; r.cmp_stride = cmp_stride; r.S = S; r.window = window;
  if (ws_cmp) {
    AttnArgs a = base; a.three_term = false; a.kind = 1; a.Lk = Lk_cmp; a.block_size = cmp_len; a.window = cmp_stride;
    const BwdPlan pl = plan_bwd(a);
    r.part_cmp = (const __nv_bfloat16*)((const char*)ws_cmp + pl.off_part);
    r.slots_cmp = pl.n_slots;
  }
  if (ws_slc) {
    AttnArgs a = base; a.kind = 2; a.Lk = base.T; a.S = S; a.block_size = block_size;
    const BwdPlan pl = plan_bwd(a);
    r.part_slc = (const char*)ws_slc + pl.off_part;
    r.pair_of_slot = pos ? pos : sel_plan_at((const char*)ws_slc + pl.off_plan, pl.layout).pair_of_slot;
  }
  if (ws_win) {
    AttnArgs a = base; a.three_term = false; a.kind = 0; a.Lk = base.T; a.window = window;
    const BwdPlan pl = plan_bwd(a);
    r.part_win = (const __nv_bfloat16*)((const char*)ws_win + pl.off_part);
    r.slots_win = pl.n_slots;
    r.shift_win = pl.wide ? 7 : 6;
  }
  return reduce_launch(r, base.D, base.three_term, "dq_reduce3", st);
}

}  // namespace nsa
