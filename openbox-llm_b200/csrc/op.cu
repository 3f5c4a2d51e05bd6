// The whole op in one call each way: pooling -> compression attention -> block scoring and top-n ->
// selection attention, window attention -> gate blend (nsa_model.py:306-370 without the
// projections), and its backward.  Host work is one argument structure and one workspace instead
// of a dozen calls with their own tensors; the branches that do not depend on one another run on
// side streams where the problem is too small to fill the GPU.
#include <string.h>

#include <algorithm>

#include "op.cuh"
#include "pool.cuh"

namespace nsa {
namespace {

constexpr size_t kAlign = 256;

// Two side streams and the events that tie them to the caller's stream, one set per host thread
// and device: an event that two threads record would tie one thread's work to the other's.  They
// are made on first use, hold no work between calls and go with the thread.  The second has the highest
// priority: it takes short kernels in a chain, which would otherwise wait until the CTAs of the long
// kernels beside them have all been placed.
struct SideStreams {
  int dev = -1;
  cudaStream_t st[2] = {nullptr, nullptr};
  cudaEvent_t begin = nullptr, end[2] = {nullptr, nullptr};
  bool make(int device) {
    dev = device;
    int least = 0, greatest = 0;
    if (cudaDeviceGetStreamPriorityRange(&least, &greatest) != cudaSuccess) return false;
    for (int k = 0; k < 2; ++k)
      if (cudaStreamCreateWithPriority(&st[k], cudaStreamNonBlocking, k == 1 ? greatest : least) != cudaSuccess ||
          cudaEventCreateWithFlags(&end[k], cudaEventDisableTiming) != cudaSuccess)
        return false;
    return cudaEventCreateWithFlags(&begin, cudaEventDisableTiming) == cudaSuccess;
  }
  void drop() {
    for (int k = 0; k < 2; ++k) {
      if (st[k]) cudaStreamDestroy(st[k]);
      if (end[k]) cudaEventDestroy(end[k]);
      st[k] = nullptr; end[k] = nullptr;
    }
    if (begin) cudaEventDestroy(begin);
    begin = nullptr;
    dev = -1;
  }
};
struct SidePool {
  SideStreams per_dev[8];
  ~SidePool() { for (SideStreams& s : per_dev) s.drop(); }
};

SideStreams* side_streams() {
  static thread_local SidePool pool;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 8) return nullptr;
  SideStreams& s = pool.per_dev[dev];
  if (s.dev < 0 && !s.make(dev)) {
    cudaGetLastError();
    s.drop();
    return nullptr;
  }
  return &s;
}

// Forks the side streams off `main` and joins them again; a call that fails in between joins them as it
// returns, since its caller gives back the memory they work in.  Off (everything on `main`) when the
// call fills the GPU by itself, when launches are being timed, or when a side stream is inside a
// stream capture that `main` is not part of.
class Fork {
 public:
  Fork(cudaStream_t main, bool want) : main_(main) {
    if (!want || profiling()) return;
    side_ = side_streams();
    if (!side_) return;
    cudaStreamCaptureStatus mine, theirs;
    unsigned long long my_id = 0, their_id = 0;
    if (cudaStreamIsCapturing(main, &mine) != cudaSuccess) { drop(); return; }
    for (int k = 0; k < 2; ++k) {
      if (cudaStreamIsCapturing(side_->st[k], &theirs) != cudaSuccess) { drop(); return; }
      if (theirs == cudaStreamCaptureStatusNone) continue;
      if (cudaStreamGetCaptureInfo(main, &mine, &my_id) != cudaSuccess ||
          cudaStreamGetCaptureInfo(side_->st[k], &theirs, &their_id) != cudaSuccess || mine != theirs || my_id != their_id) {
        drop();
        return;
      }
    }
  }
  ~Fork() {
    if (rejoin(open_) != cudaSuccess) cudaGetLastError();       // the failure that led here is the one to report
  }
  Fork(const Fork&) = delete;
  Fork& operator=(const Fork&) = delete;
  bool active() const { return side_ != nullptr; }
  cudaStream_t stream(int k) const { return side_ ? side_->st[k] : main_; }
  int begin() {                                    // the side streams see what `main` holds so far
    if (!side_) return NSA_OK;
    open_ = 3;
    NSA_CUDA_OK(cudaEventRecord(side_->begin, main_));
    for (int k = 0; k < 2; ++k) NSA_CUDA_OK(cudaStreamWaitEvent(side_->st[k], side_->begin, 0));
    return NSA_OK;
  }
  // What side stream k holds so far is all that a later wait(k) has `main` wait for (no join of k between the two).
  int mark(int k) {
    if (side_) NSA_CUDA_OK(cudaEventRecord(side_->end[k], side_->st[k]));
    return NSA_OK;
  }
  int wait(int k) {
    if (side_) NSA_CUDA_OK(cudaStreamWaitEvent(main_, side_->end[k], 0));
    return NSA_OK;
  }
  int join(int which = 3) {                        // `main` waits for the side streams of the mask
    NSA_CUDA_OK(rejoin(open_ & which));
    return NSA_OK;
  }

 private:
  void drop() { cudaGetLastError(); side_ = nullptr; }
  cudaError_t rejoin(int which) {
    open_ &= ~which;
    cudaError_t rc = cudaSuccess;
    for (int k = 0; k < 2; ++k) {                  // one stream's error does not leave the other unjoined
      if (!(which >> k & 1)) continue;
      cudaError_t e = cudaEventRecord(side_->end[k], side_->st[k]);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(main_, side_->end[k], 0);
      if (e != cudaSuccess) rc = e;
    }
    return rc;
  }
  cudaStream_t main_;
  SideStreams* side_ = nullptr;
  int open_ = 0;            // side streams that are forked and not joined yet
};

struct Carver {
  size_t off = 0;
  size_t take(size_t bytes) { const size_t at = off; off += align_up(bytes, kAlign); return at; }
};

struct OpPlan {
  int n_cmp, S, es;
  bool fused;              // the three backward kernels leave their dQ partials to one reduction
  bool three_term;           // selection on 16- and 32-token blocks on the tensor cores (api.cu), with fp32 partials
  bool acc_mode;           // fused, and window and compression add to one fp32 dQ accumulator
  bool fast_pool;
  size_t n_q, n_kv, n_c, rows;    // elements of q, of one K/V tensor, of one summary tensor; rows of q
  // saved for backward
  size_t k_cmp, v_cmp, o3, lse3, pooled, plan, plan_bytes, saved_total;
  // forward workspace: the selection's
  size_t fwd_ws;
  // backward workspace
  size_t row_stat, dk_cmp, dv_cmp, acc, acc_bytes, d_pooled, ws_pool, ws_pool_bytes, dq_acc, dq3, ws[3], ws_bytes[3], bwd_ws;
};

// impl chooses the attention kernels; lists longer than the tensor-core scorer keeps (16) are scored on
// the CUDA cores even where it names the former
int score_impl(const NsaAttentionDesc* d) { return d->impl == NSA_IMPL_TC ? NSA_IMPL_AUTO : d->impl; }

// the selection branch of a call as the tcgen05 plan sees it
AttnArgs sel_args(const NsaAttentionDesc* d, const int32_t* block_idx) {
  AttnArgs a = base_args(&d->dims, d->dims.T);
  a.block_idx = block_idx; a.kind = 2; a.S = d->n_sel; a.block_size = d->block_size;
  return a;
}

int op_plan(const NsaAttentionDesc* d, OpPlan* p) {
  int rc = check_dims(&d->dims);
  if (rc != NSA_OK) return rc;
  NSA_CHECK_ARG(d->cmp_len > 0 && d->cmp_stride > 0 && d->cmp_stride <= d->cmp_len, "bad summary length or stride");
  NSA_CHECK_ARG(d->learned || (d->cmp_len == d->block_size && d->cmp_stride == d->block_size),
                "mean pooling is defined on the aligned grid only");
  NSA_CHECK_ARG(d->block_size >= 16, "block_size must be >= 16");
  NSA_CHECK_ARG(d->window >= 1, "window must be >= 1");
  NSA_CHECK_ARG(d->n_sel >= (d->given_lists ? 0 : 1), "bad n_sel: the scorer picks at least one block");
  if (!d->given_lists) {
    rc = topn_check(&d->dims, pool_count(d->dims.T, d->cmp_len, d->cmp_stride), d->cmp_len, d->cmp_stride, d->block_size,
                    d->n_sel, d->n_init, d->n_local, score_impl(d));
    if (rc != NSA_OK) return rc;
  }
  const NsaDims& m = d->dims;
  memset(p, 0, sizeof(*p));
  p->es = m.dtype == NSA_DTYPE_BF16 ? 2 : 4;
  p->S = d->n_sel;
  p->n_cmp = pool_count(m.T, d->cmp_len, d->cmp_stride);
  p->rows = (size_t)m.B * m.Hq * m.T;
  p->n_q = p->rows * m.D;
  p->n_kv = (size_t)m.B * m.Hkv * m.T * m.D;
  p->n_c = (size_t)m.B * m.Hkv * p->n_cmp * m.D;
  p->fast_pool = d->learned && pool_learned_ok(m.D, d->cmp_len, m.dtype);
  int err;
  const bool tc = use_tc(&m, d->block_size, d->impl, &err);
  if (err != NSA_OK) return err;
  p->three_term = use_three_term(&m, d->block_size, p->S, d->impl, true);
  p->fused = (tc || p->three_term) && p->S > 0;
  p->acc_mode = tc && p->fused && d->dq_accumulator;
  const bool grad = d->need_grad != 0;

  Carver s;
  p->k_cmp = s.take(p->n_c * p->es);
  p->v_cmp = s.take(p->n_c * p->es);
  p->o3 = s.take(3 * p->n_q * p->es);
  p->lse3 = s.take(3 * p->rows * sizeof(float));
  p->pooled = s.take(grad && p->fast_pool ? 2 * p->n_c * sizeof(float) : 0);
  p->fwd_ws = nsa_selection_fwd_workspace_bytes(&m, p->S, d->block_size, d->impl);
  if (p->fused && (grad || p->fwd_ws > 0)) p->plan_bytes = tc_sel_plan_bytes(sel_args(d, nullptr));
  p->plan = s.take(p->plan_bytes);
  p->saved_total = s.off;
  if (!grad) return NSA_OK;

  Carver w;
  p->row_stat = w.take(6 * p->rows * sizeof(float));
  p->dk_cmp = w.take(p->n_c * p->es);
  p->dv_cmp = w.take(p->n_c * p->es);
  if (p->fast_pool) {
    p->acc_bytes = 2 * pool_acc_floats(m.D, d->cmp_len) * sizeof(float);
    p->acc = w.take(p->acc_bytes);
    p->d_pooled = w.take(d->cmp_stride < d->cmp_len ? 2 * p->n_c * sizeof(float) : 0);
  } else if (d->learned) {
    p->ws_pool_bytes = nsa_block_compress_strided_bwd_workspace_bytes(m.B, m.Hkv, m.T, m.D, d->cmp_len, d->cmp_stride);
    p->ws_pool = w.take(p->ws_pool_bytes);
  }
  const bool acc_mode = p->acc_mode;
  if (acc_mode) p->dq_acc = w.take(p->n_q * sizeof(float));
  if (!p->fused) p->dq3 = w.take(3 * p->n_q * p->es);
  p->ws_bytes[0] = acc_mode ? nsa_range_attn_bwd_acc_workspace_bytes(&m, p->n_cmp, NSA_MODE_COMPRESS_STRIDED, d->cmp_stride)
                            : nsa_range_attn_bwd_workspace_bytes(&m, p->n_cmp, NSA_MODE_COMPRESS_STRIDED, d->cmp_stride, d->impl);
  p->ws_bytes[1] = nsa_selection_bwd_workspace_bytes(&m, p->S, d->block_size, d->impl);
  p->ws_bytes[2] = acc_mode ? nsa_range_attn_bwd_acc_workspace_bytes(&m, m.T, NSA_MODE_WINDOW, d->window)
                            : nsa_range_attn_bwd_workspace_bytes(&m, m.T, NSA_MODE_WINDOW, d->window, d->impl);
  for (int k = 0; k < 3; ++k) p->ws[k] = w.take(p->ws_bytes[k]);
  p->bwd_ws = w.off;
  return NSA_OK;
}

// Overlap pays while one branch leaves SMs idle; beyond a few row tiles per SM every kernel fills
// the GPU alone.
bool small_problem(const NsaAttentionDesc* d) {
  const NsaDims& m = d->dims;
  const long long row_tiles = ((long long)m.B * m.Hq * m.T + 127) / 128;
  return row_tiles <= 8LL * sm_count();
}

PoolSides op_sides(const NsaAttentionDesc* d, const NsaAttentionTensors* t) {
  PoolSides s = {};
  s.n = 2;
  s.x[0] = t->kc; s.x[1] = t->vc;
  for (int k = 0; k < 2; ++k) {
    s.intra[k] = t->comp[3 * k]; s.logits[k] = t->comp[3 * k + 1]; s.proj[k] = t->comp[3 * k + 2];
  }
  (void)d;
  return s;
}

#define NSA_TRY(expr)            \
  do {                           \
    const int _rc = (expr);      \
    if (_rc != NSA_OK) return _rc; \
  } while (0)

}  // namespace
}  // namespace nsa

using namespace nsa;

extern "C" int nsa_attention_sizes(const NsaAttentionDesc* desc, size_t* saved_bytes, size_t* fwd_workspace_bytes,
                                   size_t* bwd_workspace_bytes) {
  NSA_CHECK_ARG(desc && saved_bytes && fwd_workspace_bytes && bwd_workspace_bytes, "null argument");
  OpPlan p;
  NSA_TRY(op_plan(desc, &p));
  *saved_bytes = p.saved_total;
  *fwd_workspace_bytes = p.fwd_ws;
  *bwd_workspace_bytes = p.bwd_ws;
  return NSA_OK;
}

// tokens: `out` is [B, T, Hq, D]
static int attention_fwd(const NsaAttentionDesc* d, const NsaAttentionTensors* t, void* saved, void* workspace,
                         size_t workspace_bytes, bool tokens, void* stream) {
  NSA_CHECK_ARG(d && t, "null argument");
  OpPlan p;
  NSA_TRY(op_plan(d, &p));
  const NsaDims& m = d->dims;
  if (p.rows == 0) return NSA_OK;
  NSA_CHECK_ARG(saved && t->q && t->kc && t->vc && t->ks && t->vs && t->kw && t->vw && t->gate && t->out &&
                (p.S == 0 || t->block_idx), "null tensor");
  NSA_TRY(gate_args_ok(&m, tokens ? nullptr : t->out, tokens ? t->out : nullptr));
  NSA_CHECK_ARG(p.fwd_ws == 0 || (workspace && workspace_bytes >= p.fwd_ws), "forward workspace too small: need %zu bytes", p.fwd_ws);
  if (d->learned)
    for (int k = 0; k < 6; ++k) NSA_CHECK_ARG(t->comp[k], "null compressor parameter");
  cudaStream_t st = (cudaStream_t)stream;
  char* sv = (char*)saved;
  void* k_cmp = sv + p.k_cmp;
  void* v_cmp = sv + p.v_cmp;
  char* o[3];
  float* lse[3];
  for (int k = 0; k < 3; ++k) {
    o[k] = sv + p.o3 + k * p.n_q * p.es;
    lse[k] = (float*)(sv + p.lse3) + k * p.rows;
  }
  void* plan = p.plan_bytes ? sv + p.plan : nullptr;
  Fork fork(st, small_problem(d));
  NSA_TRY(fork.begin());
  auto window = [&]() -> int {
    return nsa_range_attn_fwd(t->q, t->kw, t->vw, o[2], lse[2], &m, m.T, NSA_MODE_WINDOW, d->window, 0, d->impl, fork.stream(0));
  };
  auto build_plan = [&](cudaStream_t s) -> int {
    return plan ? tc_sel_plan_build(sel_args(d, t->block_idx), plan, p.plan_bytes, s) : NSA_OK;
  };
  SelChoice choice = {};
  auto selection = [&](cudaStream_t s) -> int {
    if (plan && p.fwd_ws) {
      AttnArgs a = sel_args(d, t->block_idx);
      a.q = t->q; a.k = t->ks; a.v = t->vs; a.o = o[1]; a.lse = lse[1]; a.sel_plan = plan;
      if (!fork.active()) {              // the other branches lie before this one: its merge can blend them
        a.g_cmp = o[0]; a.g_win = o[2]; a.g_logits = t->gate; a.g_out = t->out;
        a.o_kept = d->need_grad ? o[1] : nullptr;
        a.g_tokens = tokens;
        choice = tc_sel_choice(a, plan);
      }
      return tc_sel_fwd(a, workspace, workspace_bytes, s);
    }
    return nsa_selection_fwd(t->q, t->ks, t->vs, t->block_idx, o[1], lse[1], &m, p.S, d->block_size, workspace,
                             workspace_bytes, d->impl, s);
  };
  // Given lists: their plan, a chain of small kernels, goes ahead of what fills the GPU beside it, and the
  // selection behind that.  Lists of the scorer: the window beside the chain that leads to them.
  if (d->given_lists) NSA_TRY(build_plan(fork.stream(1)));
  else NSA_TRY(window());
  if (p.fast_pool) {
    PoolSides s = op_sides(d, t);
    s.out[0] = k_cmp; s.out[1] = v_cmp;
    if (d->need_grad)
      for (int k = 0; k < 2; ++k) s.pooled[k] = (float*)(sv + p.pooled) + k * p.n_c;
    NSA_TRY(pool_learned_fwd(s, m.B, m.Hkv, m.T, m.D, d->cmp_len, d->cmp_stride, st));
  } else if (d->learned) {
    NSA_TRY(nsa_block_compress_strided_fwd(t->kc, t->comp[0], t->comp[1], t->comp[2], k_cmp, m.B, m.Hkv, m.T, m.D,
                                           d->cmp_len, d->cmp_stride, m.dtype, stream));
    NSA_TRY(nsa_block_compress_strided_fwd(t->vc, t->comp[3], t->comp[4], t->comp[5], v_cmp, m.B, m.Hkv, m.T, m.D,
                                           d->cmp_len, d->cmp_stride, m.dtype, stream));
  } else {
    PoolSides s = op_sides(d, t);
    s.out[0] = k_cmp; s.out[1] = v_cmp;
    NSA_TRY(pool_mean_fwd(s, m.B, m.Hkv, m.T, m.D, d->block_size, m.dtype, st));
  }
  NSA_TRY(compress_fwd(t->q, k_cmp, v_cmp, o[0], lse[0], &m, p.n_cmp, d->cmp_stride, d->cmp_len, d->impl, !d->given_lists, stream));
  if (d->given_lists) {
    NSA_TRY(window());
    NSA_TRY(selection(fork.stream(1)));
    NSA_TRY(fork.join());
  } else {
    NSA_TRY(nsa_topn_blocks_general(t->q, k_cmp, lse[0], t->block_idx, nullptr, &m, p.n_cmp, d->cmp_len, d->cmp_stride,
                                      d->block_size, p.S, d->n_init, d->n_local, score_impl(d), stream));
    if (plan && !p.fwd_ws) {      // only the backward reads the plan: it is built beside the forward kernel
      NSA_TRY(fork.begin());
      NSA_TRY(build_plan(fork.stream(1)));
      NSA_TRY(nsa_selection_fwd(t->q, t->ks, t->vs, t->block_idx, o[1], lse[1], &m, p.S, d->block_size, nullptr, 0,
                                d->impl, stream));
    } else {
      NSA_TRY(build_plan(st));
      NSA_TRY(selection(st));
    }
    NSA_TRY(fork.join(1));
  }
  NSA_TRY(gate_fwd_unless_blended(o[0], o[1], o[2], t->gate, t->out, &m, choice, tokens, stream));
  return fork.join();                    // a plan that only the backward reads
}

extern "C" int nsa_attention_fwd(const NsaAttentionDesc* d, const NsaAttentionTensors* t, void* saved, void* workspace,
                                 size_t workspace_bytes, void* stream) {
  return attention_fwd(d, t, saved, workspace, workspace_bytes, false, stream);
}

extern "C" int nsa_attention_fwd_tokens(const NsaAttentionDesc* d, const NsaAttentionTensors* t, void* saved, void* workspace,
                                        size_t workspace_bytes, void* stream) {
  return attention_fwd(d, t, saved, workspace, workspace_bytes, true, stream);
}

// d_tokens: d_out in [B, T, Hq, D], which this call writes to t->d_out in the order of the heads (null: it is there)
static int attention_bwd(const NsaAttentionDesc* d, const NsaAttentionTensors* t, const void* saved, void* workspace,
                         size_t workspace_bytes, const void* d_tokens, void* stream) {
  NSA_CHECK_ARG(d && t, "null argument");
  OpPlan p;
  NSA_TRY(op_plan(d, &p));
  NSA_CHECK_ARG(d->need_grad, "the forward call did not keep what backward needs");
  const NsaDims& m = d->dims;
  if (p.rows == 0) {         // no tokens: only the parameters have a gradient, zero
    for (int k = 0; k < 6 && d->learned; ++k) {
      NSA_CHECK_ARG(t->d_comp[k], "null compressor gradient");
      const size_t n = k % 3 == 0 ? (size_t)d->cmp_len * m.D : (k % 3 == 1 ? (size_t)d->cmp_len : (size_t)m.D * m.D);
      NSA_CUDA_OK(cudaMemsetAsync(t->d_comp[k], 0, n * sizeof(float), (cudaStream_t)stream));
    }
    return NSA_OK;
  }
  NSA_CHECK_ARG(saved && t->q && t->kc && t->vc && t->ks && t->vs && t->kw && t->vw && t->gate && t->d_out &&
                (p.S == 0 || t->block_idx), "null tensor");
  NSA_TRY(gate_args_ok(&m, t->d_out, d_tokens));
  NSA_CHECK_ARG(t->dq && t->dkc && t->dvc && t->dks && t->dvs && t->dkw && t->dvw && t->d_gate, "null gradient");
  NSA_CHECK_ARG(workspace && workspace_bytes >= p.bwd_ws, "backward workspace too small: need %zu bytes", p.bwd_ws);
  if (d->learned)
    for (int k = 0; k < 6; ++k) NSA_CHECK_ARG(t->comp[k] && t->d_comp[k], "null compressor parameter or gradient");
  cudaStream_t st = (cudaStream_t)stream;
  const char* sv = (const char*)saved;
  char* w = (char*)workspace;
  const void* k_cmp = sv + p.k_cmp;
  const void* v_cmp = sv + p.v_cmp;
  const char* o[3];
  const float* lse[3];
  float *rs[3], *rd[3];
  for (int k = 0; k < 3; ++k) {
    o[k] = sv + p.o3 + k * p.n_q * p.es;
    lse[k] = (const float*)(sv + p.lse3) + k * p.rows;
    rs[k] = (float*)(w + p.row_stat) + k * p.rows;
    rd[k] = (float*)(w + p.row_stat) + (3 + k) * p.rows;
  }
  void* dk_cmp = w + p.dk_cmp;
  void* dv_cmp = w + p.dv_cmp;
  const bool acc_mode = p.acc_mode;
  NSA_CHECK_ARG(!p.three_term || aligned16(t->q, t->ks, t->vs, t->d_out, t->dq),
                "q, ks, vs, d_out and dq have to start on a 16-byte boundary");
  float* dq_acc = (float*)(w + p.dq_acc);
  void* ws[3];
  void* dq[3];             // where a branch puts its own dq (null: partials stay in its workspace)
  for (int k = 0; k < 3; ++k) {
    ws[k] = w + p.ws[k];
    dq[k] = p.fused ? nullptr : w + p.dq3 + k * p.n_q * p.es;
  }
  if (acc_mode) NSA_CUDA_OK(cudaMemsetAsync(dq_acc, 0, p.n_q * sizeof(float), st));
  // gate backward as per-row statistics; the branch kernels apply the gate factor themselves
  NSA_TRY(gate_bwd_rows(o[0], o[1], o[2], t->gate, d_tokens ? d_tokens : t->d_out, rs[0], rd[0], t->d_gate, &m,
                        d_tokens ? const_cast<void*>(t->d_out) : nullptr, (float*)(w + p.acc), p.acc_bytes / sizeof(float), stream));
  Fork fork(st, small_problem(d));
  NSA_TRY(fork.begin());
  cudaStream_t s_win = fork.stream(0), s_cmp = fork.stream(1);
  // compression, then the pooling under it: first in line, since it is the longest
  // chain.  (3 x 3001 tokens, 12 heads of 64, from a graph: 633 us so, 670 with the window before the selection, 703
  // with the chain at the priority of the other two.)
  if (acc_mode && p.n_cmp > 0)
    NSA_TRY(nsa_range_attn_bwd_acc(t->q, k_cmp, v_cmp, o[0], lse[0], t->d_out, dq_acc, dk_cmp, dv_cmp, &m, p.n_cmp,
                                   NSA_MODE_COMPRESS_STRIDED, d->cmp_stride, d->cmp_len, rs[0], rd[0], ws[0], p.ws_bytes[0], s_cmp));
  else if (!acc_mode)
    NSA_TRY(nsa_range_attn_bwd(t->q, k_cmp, v_cmp, o[0], lse[0], t->d_out, dq[0], dk_cmp, dv_cmp, &m, p.n_cmp,
                               NSA_MODE_COMPRESS_STRIDED, d->cmp_stride, d->cmp_len, rs[0], rd[0], ws[0], p.ws_bytes[0],
                               d->impl, s_cmp));
  NSA_TRY(fork.mark(1));
  if (p.fast_pool) {
    PoolSides s = op_sides(d, t);
    s.d_out[0] = dk_cmp; s.d_out[1] = dv_cmp;
    s.dx[0] = t->dkc; s.dx[1] = t->dvc;
    for (int k = 0; k < 2; ++k) {
      s.pooled[k] = (float*)(sv + p.pooled) + k * p.n_c;
      s.d_pooled[k] = (float*)(w + p.d_pooled) + k * p.n_c;
      s.acc[k] = (float*)(w + p.acc) + k * pool_acc_floats(m.D, d->cmp_len);
      s.d_intra[k] = t->d_comp[3 * k]; s.d_logits[k] = t->d_comp[3 * k + 1]; s.d_proj[k] = t->d_comp[3 * k + 2];
    }
    NSA_TRY(pool_learned_bwd(s, m.B, m.Hkv, m.T, m.D, d->cmp_len, d->cmp_stride, s_cmp));
  } else if (d->learned) {
    for (int k = 0; k < 2; ++k)
      NSA_TRY(nsa_block_compress_strided_bwd(k ? t->vc : t->kc, t->comp[3 * k], t->comp[3 * k + 1], t->comp[3 * k + 2],
                                             k ? dv_cmp : dk_cmp, k ? t->dvc : t->dkc, t->d_comp[3 * k], t->d_comp[3 * k + 1],
                                             t->d_comp[3 * k + 2], m.B, m.Hkv, m.T, m.D, d->cmp_len, d->cmp_stride, m.dtype,
                                             w + p.ws_pool, p.ws_pool_bytes, s_cmp));
  } else {
    PoolSides s = op_sides(d, t);
    s.d_out[0] = dk_cmp; s.d_out[1] = dv_cmp;
    s.dx[0] = t->dkc; s.dx[1] = t->dvc;
    NSA_TRY(pool_mean_bwd(s, m.B, m.Hkv, m.T, m.D, d->block_size, m.dtype, s_cmp));
  }
  // selection
  if (p.fused) {
    AttnArgs a = base_args(&m, m.T);
    a.three_term = p.three_term;
    a.q = t->q; a.k = t->ks; a.v = t->vs; a.o = (void*)o[1]; a.lse = (float*)lse[1]; a.d_o = t->d_out; a.dq = nullptr;
    a.block_idx = t->block_idx; a.kind = 2; a.S = p.S; a.block_size = d->block_size;
    a.row_scale = rs[1]; a.row_dot = rd[1];
    a.dk_acc = (float*)t->dks; a.dv_acc = (float*)t->dvs;
    a.sel_plan = sv + p.plan; a.plan_kept = true;
    NSA_TRY(tc_attn_bwd(a, ws[1], p.ws_bytes[1], st));
  } else {
    NSA_TRY(nsa_selection_bwd(t->q, t->ks, t->vs, t->block_idx, o[1], lse[1], t->d_out, dq[1], t->dks, t->dvs, &m, p.S,
                              d->block_size, rs[1], rd[1], ws[1], p.ws_bytes[1], d->impl, st));
  }
  // window
  if (acc_mode)
    NSA_TRY(nsa_range_attn_bwd_acc(t->q, t->kw, t->vw, o[2], lse[2], t->d_out, dq_acc, t->dkw, t->dvw, &m, m.T,
                                   NSA_MODE_WINDOW, d->window, 0, rs[2], rd[2], ws[2], p.ws_bytes[2], s_win));
  else
    NSA_TRY(window_bwd(t->q, t->kw, t->vw, o[2], lse[2], t->d_out, dq[2], t->dkw, t->dvw, &m, d->window, rs[2], rd[2],
                       ws[2], p.ws_bytes[2], d->impl, s_win));
  // the sum of dq needs the compression's attention, not the pooling behind it, which runs beside the sum
  NSA_TRY(fork.join(1));
  NSA_TRY(fork.wait(1));
  if (!p.fused) {
    NSA_TRY(nsa_sum3(dq[0], dq[1], dq[2], t->dq, p.n_q, m.dtype, stream));
    return fork.join();
  }
  // the three branches left their dQ partials in their workspaces (or two of them in the accumulator)
  AttnArgs a = base_args(&m, m.T);
  a.three_term = p.three_term;
  a.wide_dq = true;
  const int32_t* pos = sel_plan_pair_map(a, p.S, d->block_size, sv + p.plan);
  if (acc_mode)
    NSA_TRY(tc_dq_reduce3(a, 0, 0, 0, p.S, d->block_size, 1, nullptr, ws[1], nullptr, pos, dq_acc, t->dq, st));
  else
    NSA_TRY(tc_dq_reduce3(a, p.n_cmp, d->cmp_len, d->cmp_stride, p.S, d->block_size, d->window,
                          p.n_cmp > 0 ? ws[0] : nullptr, ws[1], ws[2], pos, nullptr, t->dq, st));
  return fork.join();
}

extern "C" int nsa_attention_bwd(const NsaAttentionDesc* d, const NsaAttentionTensors* t, const void* saved, void* workspace,
                                 size_t workspace_bytes, void* stream) {
  return attention_bwd(d, t, saved, workspace, workspace_bytes, nullptr, stream);
}

extern "C" int nsa_attention_bwd_tokens(const NsaAttentionDesc* d, const NsaAttentionTensors* t, const void* saved,
                                        void* workspace, size_t workspace_bytes, const void* d_tokens, void* stream) {
  NSA_CHECK_ARG(d_tokens || !t || !t->d_out, "null tensor");
  return attention_bwd(d, t, saved, workspace, workspace_bytes, d_tokens, stream);
}
