// Selected-block attention forward, key-block outer ("split-K over blocks"): host side, the
// merge of the per-(query, block) partials and the choice of the variant.
//
// When neighbouring queries list unrelated blocks, a query-outer tile wastes most of every MMA
// on rows that do not attend the block.  The block-outer kernel (tc_fwdpair_kernel.cu) instead gives one
// CTA one 64-token block: K and V of the block are loaded once, the (query, head) rows that list
// the block are gathered from the block -> query CSR, 128 rows at a time, and for each row tile
//   S = Q K^T ,  p = exp2(s*scale*log2e - m) with m the row's maximum over this block,  O_part = P V
// are computed; O_part (bf16), m and the sum of p (fp32) are written per (pair, head).
// sel_combine_kernel merges the partials of each query: o = sum_j 2^(m_j-M) O_j / sum_j 2^(m_j-M) l_j.
// The plan of the block list counts the distinct blocks per query tile; both forward variants read
// that on the device and only the cheaper one does the work.
#include "tc_common.cuh"
#include "tc_host.cuh"

namespace nsa {
namespace tc {

// o[b, hkv*G+g, t, :] and lse from the per-(pair, head) partials of query (bh, t).  Bound by the one pass
// over the partials: a thread owns 8 columns of H neighbouring heads, whose partial rows lie side by
// side and share the index loads and the addresses, and has 4 H 16-byte loads in flight.  Three CTAs of 80
// registers share an SM, which is what the pass needs in flight: at 8 x 32768 tokens, 16 heads of 128, 19 GB in
// 3.02 ms, 3.58 with two CTAs of 110; 64 heads x 65536 2.97, 3.43 (3.45 with four CTAs of 64 registers, which spill, 3.36
// and 3.00 with two slots a trip and three or four CTAs, 3.51 with eight).
//
// Where the whole op asks for it (gb.out) the gate blend is done here too: o_slc need not be read back (nor written,
// when no backward follows).
struct GateBlend {
  const __nv_bfloat16 *cmp, *win, *logits;
  __nv_bfloat16* out;
  bool tokens;                             // out is [B, T, Hq, D]
};
template <int D, int H>
__global__ void __launch_bounds__(256, 3)
sel_combine_kernel(const __nv_bfloat16* o_part, const float* ml,
                   const int32_t* pair_of_slot, const SelPlanHeader* hdr,
                   __nv_bfloat16* o, float* lse, const GateBlend gb, int B, int Hq, int Hkv, int T,
                   int G, int S, int nq_union, int force) {
  chain_wait();
  if (!prefer_pairs(hdr, nq_union, force)) return;
  constexpr int kVec = D / 8;
  const int groups = G / H;
  const size_t gid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t total = (size_t)B * Hkv * T * groups * kVec;
  if (gid >= total) return;
  const int v = (int)(gid % kVec);
  const int g = (int)((gid / kVec) % groups) * H;
  const int t = (int)((gid / ((size_t)kVec * groups)) % T);
  const size_t bh = gid / ((size_t)kVec * groups * T);
  const int32_t* ps = pair_of_slot + (bh * T + t) * S;
  // one pass with a running maximum: o = sum_j 2^(m_j - M) O_j / sum_j 2^(m_j - M) l_j
  float M[H], L[H], acc[H][8];
#pragma unroll
  for (int h = 0; h < H; ++h) {
    M[h] = -INFINITY; L[h] = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[h][e] = 0.f;
  }
  // four slots per trip: all loads of a trip are issued before the first is used
  for (int s0 = 0; s0 < S; s0 += 4) {
    int pr[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) pr[j] = s0 + j < S ? ld_plain(ps + s0 + j) : -1;
    float m[H][4], l[H][4];
    uint4 u[H][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int h = 0; h < H; ++h) { m[h][j] = -INFINITY; l[h][j] = 0.f; u[h][j] = make_uint4(0u, 0u, 0u, 0u); }
      if (pr[j] >= 0) {
        const size_t prow = (size_t)pr[j] * G + g;
        if (H == 2) {
          const float4 st = __ldcs(reinterpret_cast<const float4*>(ml + prow * 2));
          m[0][j] = st.x; l[0][j] = st.y;
          m[H - 1][j] = st.z; l[H - 1][j] = st.w;
        } else {
          const float2 st = __ldcs(reinterpret_cast<const float2*>(ml + prow * 2));
          m[0][j] = st.x; l[0][j] = st.y;
        }
#pragma unroll
        for (int h = 0; h < H; ++h) u[h][j] = __ldcs(reinterpret_cast<const uint4*>(o_part + (prow + h) * D + v * 8));
      }
    }
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const float Mn = fmaxf(fmaxf(fmaxf(m[h][0], m[h][1]), fmaxf(m[h][2], m[h][3])), M[h]);
      if (Mn == -INFINITY) continue;                          // nothing in this trip, nothing before
      const float a_old = ex2(M[h] - Mn);                     // M = -inf: 0
      L[h] *= a_old;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[h][e] *= a_old;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float w = ex2(m[h][j] - Mn);                    // absent slot: 0
        L[h] = fmaf(w, l[h][j], L[h]);
        const uint32_t x[4] = {u[h][j].x, u[h][j].y, u[h][j].z, u[h][j].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {                         // bf16 -> fp32 is a shift
          acc[h][2 * e] = fmaf(w, __uint_as_float(x[e] << 16), acc[h][2 * e]);
          acc[h][2 * e + 1] = fmaf(w, __uint_as_float(x[e] & 0xffff0000u), acc[h][2 * e + 1]);
        }
      }
      M[h] = Mn;
    }
  }
  const int b = (int)(bh / Hkv), hkv = (int)(bh % Hkv);
#pragma unroll
  for (int h = 0; h < H; ++h) {
    const float inv = L[h] > 0.f ? 1.f / L[h] : 0.f;
    const size_t orow = ((size_t)b * Hq + hkv * G + g + h) * T + t;
    uint4 u;
    u.x = pack_bf16(acc[h][0] * inv, acc[h][1] * inv); u.y = pack_bf16(acc[h][2] * inv, acc[h][3] * inv);
    u.z = pack_bf16(acc[h][4] * inv, acc[h][5] * inv); u.w = pack_bf16(acc[h][6] * inv, acc[h][7] * inv);
    if (o) *reinterpret_cast<uint4*>(o + orow * D + v * 8) = u;
    if (gb.out) {
      const uint4 c = __ldcs(reinterpret_cast<const uint4*>(gb.cmp + orow * D + v * 8));
      const uint4 w = __ldcs(reinterpret_cast<const uint4*>(gb.win + orow * D + v * 8));
      float gate[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) gate[k] = 1.f / (1.f + expf(-__bfloat162float(gb.logits[orow * 3 + k])));
      const uint32_t xc[4] = {c.x, c.y, c.z, c.w}, xs[4] = {u.x, u.y, u.z, u.w}, xw[4] = {w.x, w.y, w.z, w.w};
      uint32_t r[4];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        r[e] = pack_bf16(gate[0] * __uint_as_float(xc[e] << 16) + gate[1] * __uint_as_float(xs[e] << 16) +
                             gate[2] * __uint_as_float(xw[e] << 16),
                         gate[0] * __uint_as_float(xc[e] & 0xffff0000u) + gate[1] * __uint_as_float(xs[e] & 0xffff0000u) +
                             gate[2] * __uint_as_float(xw[e] & 0xffff0000u));
      const size_t at = gb.tokens ? ((size_t)b * T + t) * Hq + hkv * G + g + h : orow;
      *reinterpret_cast<uint4*>(gb.out + at * D + v * 8) = make_uint4(r[0], r[1], r[2], r[3]);
    }
    if (v == 0) lse[orow] = L[h] > 0.f ? (M[h] + log2f(L[h])) * kLn2 : kLseEmpty;
  }
}

struct PairPlan {
  int nq;
  size_t cap_pairs;
  SelPlanLayout layout;
  size_t off_part, off_ml, off_plan, total;
};

static PairPlan plan_pairs(const AttnArgs& a) {
  PairPlan pl;
  const int G = a.Hq / a.Hkv;
  pl.nq = kRows / G;
  const int units = a.B * a.Hkv;
  pl.layout = sel_plan_layout(units, a.T, a.S, pl.nq);
  pl.cap_pairs = (size_t)units * a.T * a.S;
  size_t off = 0;
  pl.off_part = off; off += align_up(pl.cap_pairs * G * a.D * 2, 256);
  pl.off_ml = off; off += align_up(pl.cap_pairs * G * 2 * 4, 256);
  pl.off_plan = off; off += pl.layout.total;
  pl.total = off;
  return pl;
}

}  // namespace tc

int tc_fwd_union_launch(const AttnArgs& a, const SelPlanHeader* plan, int force, cudaStream_t st);
int get_option_sel_fwd();
int tc_fwdpair_launch(const AttnArgs& a, const SelPlan& plan, void* o_part, float* ml, int force, int nq,
                      int n_ktiles, int nq_union, size_t cap_pairs, unsigned grid, cudaStream_t st);

// A query tile meets at most the key tiles there are, and a full list names S of them: where there
// are no more than 3.5 S key tiles the query-outer kernel is the cheaper one whatever the lists say
// (prefer_pairs), so the call is that one kernel and needs neither plan nor workspace.
// The three-term form exists query-outer only.
static bool query_outer_only(const AttnArgs& a) {
  return a.three_term || (get_option_sel_fwd() == 0 && 2LL * ((a.T + tc::kKeys - 1) / tc::kKeys) <= 7LL * a.S);
}

size_t tc_sel_fwd_workspace(const AttnArgs& a) { return query_outer_only(a) ? 0 : tc::plan_pairs(a).total; }

size_t tc_sel_plan_bytes(const AttnArgs& a) { return tc::plan_pairs(a).layout.total; }

const int32_t* sel_plan_pair_map(const AttnArgs& base, int S, int block_size, const void* plan) {
  AttnArgs a = base;
  a.S = S; a.block_size = block_size;
  return sel_plan_at(plan, tc::plan_pairs(a).layout).pair_of_slot;
}

SelChoice tc_sel_choice(const AttnArgs& a, const void* plan) {
  return {sel_plan_at(plan, tc::plan_pairs(a).layout).hdr, tc::kRows / tc::group_pad(a.Hq / a.Hkv), get_option_sel_fwd()};
}

int tc_sel_plan_build(const AttnArgs& a, void* plan, size_t plan_bytes, cudaStream_t st) {
  using namespace tc;
  const PairPlan pl = plan_pairs(a);
  if (!plan || plan_bytes < pl.layout.total) {
    set_error("selection plan buffer too small: need %zu bytes", pl.layout.total);
    return NSA_ERR_WORKSPACE;
  }
  return sel_plan_build(a.block_idx, plan, pl.layout, a.B * a.Hkv, a.T, a.S, a.block_size, pl.nq,
                        kRows / group_pad(a.Hq / a.Hkv), st);
}

// Selection forward: the plan (the caller's, or built here), then both variants are launched; the
// device-side rule lets exactly one of them do the work.
int tc_sel_fwd(const AttnArgs& a, void* ws, size_t ws_bytes, cudaStream_t st) {
  using namespace tc;
  if (query_outer_only(a)) return tc_fwd_union_launch(a, nullptr, 1, st);
  const PairPlan pl = plan_pairs(a);
  if (!ws || ws_bytes < pl.total) {
    set_error("selection forward workspace too small: need %zu bytes", pl.total);
    return NSA_ERR_WORKSPACE;
  }
  char* base = (char*)ws;
  const int G = a.Hq / a.Hkv;
  const int nq_union = kRows / group_pad(G);
  const void* plan_mem = a.sel_plan;
  int rc = NSA_OK;
  if (!plan_mem) {
    plan_mem = base + pl.off_plan;
    rc = tc_sel_plan_build(a, base + pl.off_plan, pl.layout.total, st);
    if (rc != NSA_OK) return rc;
  }
  const SelPlan plan = sel_plan_at(plan_mem, pl.layout);
  const int force = get_option_sel_fwd();
  rc = tc_fwd_union_launch(a, plan.hdr, force, st);
  if (rc != NSA_OK) return rc;

  const unsigned grid = (unsigned)((size_t)a.B * a.Hkv * pl.layout.max_items);
  rc = tc_fwdpair_launch(a, plan, base + pl.off_part, (float*)(base + pl.off_ml), force, pl.nq, pl.layout.n_ktiles,
                         nq_union, pl.cap_pairs, grid, st);
  if (rc != NSA_OK) return rc;
  const int H = G % 2 == 0 ? 2 : 1;       // two heads: their statistics are one 16-byte load, aligned for even G
  const size_t nthreads = (size_t)a.B * a.Hkv * a.T * (G / H) * (a.D / 8);
  const unsigned cgrid = (unsigned)((nthreads + 255) / 256);
  auto combine = [&](auto kernel) -> int {
    KernelScope ks("sel_combine_kernel", st);
    NSA_CUDA_OK(launch_chained(kernel, cgrid, 256, 0, st, (const __nv_bfloat16*)(base + pl.off_part), (const float*)(base + pl.off_ml),
                               plan.pair_of_slot, plan.hdr, (__nv_bfloat16*)(a.g_out ? a.o_kept : a.o), a.lse,
                               GateBlend{(const __nv_bfloat16*)a.g_cmp, (const __nv_bfloat16*)a.g_win,
                                         (const __nv_bfloat16*)a.g_logits, (__nv_bfloat16*)a.g_out, a.g_tokens},
                               a.B, a.Hq, a.Hkv, a.T, G, a.S, nq_union, force));
    return NSA_OK;
  };
  if (a.D == 128) rc = H == 2 ? combine(sel_combine_kernel<128, 2>) : combine(sel_combine_kernel<128, 1>);
  else rc = H == 2 ? combine(sel_combine_kernel<64, 2>) : combine(sel_combine_kernel<64, 1>);
  if (rc != NSA_OK) return rc;
  NSA_LAUNCH_OK("sel_combine_kernel");
  return NSA_OK;
}

}  // namespace nsa
