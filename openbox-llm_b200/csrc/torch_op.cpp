// Autograd nodes of the whole op and of the projection layer in C++.  What a short call costs is host work: with
// 1024 tokens the op's kernels take 150 us forward + backward, while its Python nodes, their tensors and
// the ctypes calls took 350.  The nodes here do what those of ops.py and module.py do for the usual form of a call
// (dense CUDA tensors of one device and type that start on 16-byte boundaries, no dispatch mode, transform or
// trace under way); for every other form the entry points return None and the Python nodes serve it.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/nsa_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

PyObject* g_error = nullptr;             // NsaError of the Python package

[[noreturn]] void raise_error(int rc) {
  PyGILState_STATE s = PyGILState_Ensure();
  const std::string msg = "libnsa_b200 error " + std::to_string(rc) + ": " + nsa_last_error();
  PyErr_SetString(g_error, msg.c_str());
  python_error err;
  err.persist();
  PyGILState_Release(s);
  throw std::move(err);
}
void check(int rc) {
  if (rc != NSA_OK) raise_error(rc);
}

void* raw_stream(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
// New memory on the device of `t`, without the way through the dispatcher that at::empty takes: a backward makes 15
// tensors, and calls of some 1024 tokens last as long as their host work.  Operator forward + backward at
// T = 1024 199 -> 192 us, the layer's forward on 256 tokens 97 -> 92.
// Where torch fills new memory itself (deterministic algorithms) or something looks on at the calls, it is at::empty.
Tensor fresh(at::IntArrayRef sizes, at::ScalarType dtype, const Tensor& t) {
  if (at::globalContext().deterministicAlgorithms() || c10::impl::TorchDispatchModeTLS::any_modes_set())
    return at::empty(sizes, t.options().dtype(dtype));
  return Tensor(at::detail::empty_cuda(sizes, dtype, t.device(), std::nullopt));
}
Tensor fresh_like(const Tensor& t) { return fresh(t.sizes(), t.scalar_type(), t); }
Tensor bytes_like(size_t n, const Tensor& t) { return fresh({(int64_t)n}, at::kByte, t); }

// A dense CUDA tensor of the given type on device `dev` that starts on a 16-byte boundary and that no Python-side
// dispatch stands behind.
bool plain(const Tensor& t, at::ScalarType dtype, at::Device dev) {
  return t.defined() && t.layout() == at::kStrided && t.device() == dev && t.scalar_type() == dtype && t.numel() > 0 &&
         t.is_contiguous() && !t.is_neg() && !t.unsafeGetTensorImpl()->is_python_dispatch() &&
         (reinterpret_cast<uintptr_t>(t.unsafeGetTensorImpl()->data()) & 15) == 0;
}
// No functorch transform and no dispatch mode sees the tensors of this call.
bool plain_state() {
  return !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

// The tensors of a call in the order of NsaAttentionTensors: q, kc, vc, ks, vs, kw, vw, gate; the compressor's.
struct Call {
  NsaAttentionDesc d;
  Tensor in[8], comp[6], block_idx;
};

// Sizes that belong together; what is refused here gets its message from the Python side.
bool fill_desc(Call& c, int64_t B, int64_t Hq, int64_t Hkv, int64_t T, int64_t D, at::ScalarType dtype, const int* ints,
               bool learned, bool given) {
  if ((dtype != at::kBFloat16 && dtype != at::kFloat) || Hkv < 1 || Hq % Hkv || (D != 16 && D != 32 && D != 64 && D != 128) || ints[0] < 16 || T > INT32_MAX) return false;
  c.d.dims = {(int32_t)B, (int32_t)Hq, (int32_t)Hkv, (int32_t)T, (int32_t)D,
              dtype == at::kBFloat16 ? NSA_DTYPE_BF16 : NSA_DTYPE_F32};
  c.d.block_size = ints[0]; c.d.n_sel = ints[1]; c.d.window = ints[2];
  c.d.n_init = ints[3]; c.d.n_local = ints[4]; c.d.cmp_len = ints[5]; c.d.cmp_stride = ints[6];
  c.d.dq_accumulator = ints[7]; c.d.impl = ints[8];
  c.d.learned = learned; c.d.given_lists = given; c.d.need_grad = 0;
  if (!learned && (ints[5] != ints[0] || ints[6] != ints[0])) return false;
  if (given) {
    const auto s = c.block_idx.sizes();
    if (s.size() != 4 || s[0] != B || s[1] != Hkv || s[2] != T) return false;
    c.d.n_sel = (int32_t)s[3];
  } else if (ints[1] < 1) {
    return false;
  }
  return true;
}
bool comp_ok(const Call& c, at::Device dev) {
  const int64_t n = c.d.cmp_len, D = c.d.dims.D;
  for (int k = 0; k < 6; ++k)
    if (!plain(c.comp[k], at::kFloat, dev) || c.comp[k].numel() != (k % 3 == 0 ? n * D : k % 3 == 1 ? n : D * D)) return false;
  return true;
}

// The eight inputs, or their gradients, by address.  Of the layer the keys and values of the branches are parts of one tensor: views of them
// would cost a dispatch each (forward on 256 tokens, calls in a row, 99.8 -> 95.0 us).
struct Eight {
  void* p[8];
  explicit Eight(const Tensor* t) {
    for (int k = 0; k < 8; ++k) p[k] = t[k].data_ptr();
  }
  Eight(const Tensor& q, const Tensor& kv, const Tensor& gate) {
    const size_t part = kv.nbytes() / 6;
    p[0] = q.data_ptr();
    for (int k = 0; k < 6; ++k) p[1 + k] = (char*)kv.data_ptr() + k * part;
    p[7] = gate.data_ptr();
  }
};
NsaAttentionTensors pointers(const Eight& in, const Tensor* comp, const Tensor& block_idx, bool learned) {
  NsaAttentionTensors t = {};
  const void** p[8] = {&t.q, &t.kc, &t.vc, &t.ks, &t.vs, &t.kw, &t.vw, &t.gate};
  for (int k = 0; k < 8; ++k) *p[k] = in.p[k];
  for (int k = 0; k < 6 && learned; ++k) t.comp[k] = comp[k].data_ptr<float>();
  t.block_idx = block_idx.data_ptr<int32_t>();
  return t;
}

// out; `saved` keeps what backward reads.  Makes c.block_idx where the scorer writes it.
// tokens: the shape of an output in token order ([B, T, Hq, D] elements)
Tensor op_forward(Call& c, const Eight& in, const Tensor& q, bool need_grad, Tensor* saved, at::IntArrayRef tokens = {}) {
  c.d.need_grad = need_grad;
  if (!c.d.given_lists) c.block_idx = fresh({c.d.dims.B, c.d.dims.Hkv, c.d.dims.T, c.d.n_sel}, at::kInt, q);
  size_t keep, fwd, bwd;
  check(nsa_attention_sizes(&c.d, &keep, &fwd, &bwd));
  Tensor out = tokens.empty() ? fresh_like(q) : fresh(tokens, q.scalar_type(), q);
  Tensor mem = bytes_like(keep + (need_grad ? 0 : fwd) + 1, q), ws;
  void* ws_ptr = (char*)mem.data_ptr() + keep;
  if (need_grad && fwd) {
    ws = bytes_like(fwd, q);
    ws_ptr = ws.data_ptr();
  }
  NsaAttentionTensors t = pointers(in, c.comp, c.block_idx, c.d.learned);
  t.out = out.data_ptr();
  check((tokens.empty() ? nsa_attention_fwd : nsa_attention_fwd_tokens)(&c.d, &t, mem.data_ptr(), ws_ptr, fwd, raw_stream(q)));
  *saved = mem;
  return out;
}

// d_in: the eight gradients, allocated by the caller.  d_tokens: the output's gradient in [B, T, Hq, D]; d_out is scratch then.
void op_backward(const NsaAttentionDesc& d, const Eight& in, const Tensor* comp, const Tensor& block_idx, const Tensor& saved,
                 const Tensor& d_out, const Eight& d_in, Tensor* d_comp, const Tensor* d_tokens = nullptr) {
  size_t keep, fwd, bwd;
  check(nsa_attention_sizes(&d, &keep, &fwd, &bwd));
  NsaAttentionTensors t = pointers(in, comp, block_idx, d.learned);
  t.d_out = d_out.data_ptr();
  void** p[8] = {&t.dq, &t.dkc, &t.dvc, &t.dks, &t.dvs, &t.dkw, &t.dvw, &t.d_gate};
  for (int k = 0; k < 8; ++k) *p[k] = d_in.p[k];
  for (int k = 0; k < 6 && d.learned; ++k) {
    d_comp[k] = fresh_like(comp[k]);
    t.d_comp[k] = d_comp[k].data_ptr<float>();
  }
  Tensor ws = bytes_like(bwd + 1, d_out);
  if (d_tokens) check(nsa_attention_bwd_tokens(&d, &t, saved.data_ptr(), ws.data_ptr(), bwd, d_tokens->data_ptr(), raw_stream(d_out)));
  else check(nsa_attention_bwd(&d, &t, saved.data_ptr(), ws.data_ptr(), bwd, raw_stream(d_out)));
}

// A descriptor travels to the backward as a list of integers.
std::vector<int64_t> pack(const NsaAttentionDesc& d) {
  const int32_t* p = reinterpret_cast<const int32_t*>(&d);
  return std::vector<int64_t>(p, p + sizeof(d) / sizeof(int32_t));
}
NsaAttentionDesc unpack(AutogradContext* ctx) {
  NsaAttentionDesc d;
  const auto v = ctx->saved_data["desc"].toIntVector();
  for (size_t k = 0; k < v.size(); ++k) reinterpret_cast<int32_t*>(&d)[k] = (int32_t)v[k];
  return d;
}
// what a saved-tensor hook gave back may lie anywhere
Tensor aligned(const Tensor& t) {
  if (!t.defined()) return t;
  const Tensor c = t.contiguous();
  return (reinterpret_cast<uintptr_t>(c.data_ptr()) & 15) ? c.clone() : c;
}

// The kernels' gradients have no derivative here.  Where a graph of the backward is asked for (create_graph), they
// come out of nodes that say so when they are differentiated, instead of as constants.
struct Once : torch::autograd::Function<Once> {
  static Tensor forward(AutogradContext* ctx, const Tensor& g) { return g.detach(); }
  static variable_list backward(AutogradContext*, variable_list) {
    TORCH_CHECK(false, "libnsa_b200: the gradients of the op cannot be differentiated again");
  }
};
variable_list once(variable_list res) {
  if (at::GradMode::is_enabled())
    for (Tensor& g : res)
      if (g.defined()) g = Once::apply(g.detach().requires_grad_(true));
  return res;
}

// ---- the whole op -------------------------------------------------------------------------------------
struct OpNode {
  template <typename... A>
  static Tensor run(AutogradContext* ctx, Call* c, const A&...) {
    Tensor saved;
    Tensor out = op_forward(*c, Eight(c->in), c->in[0], true, &saved);
    variable_list keep(c->in, c->in + 8);
    keep.push_back(c->block_idx);
    keep.push_back(saved);
    if (c->d.learned) keep.insert(keep.end(), c->comp, c->comp + 6);
    ctx->save_for_backward(std::move(keep));
    ctx->saved_data["desc"] = pack(c->d);
    ctx->set_materialize_grads(false);
    return out;
  }
  static variable_list grads(AutogradContext* ctx, const variable_list& g) {
    const NsaAttentionDesc d = unpack(ctx);
    const int n = d.learned ? 14 : 8;
    variable_list res(1 + n);                   // the call structure has no gradient
    if (!g[0].defined()) return res;
    variable_list kept = ctx->get_saved_variables();
    for (Tensor& t : kept) t = aligned(t);
    TORCH_CHECK(g[0].device() == kept[9].device(), "libnsa_b200: tensors on different devices");
    TORCH_CHECK(g[0].scalar_type() == kept[0].scalar_type(), "libnsa_b200: the gradient's type is not the output's");
    const Tensor d_out = aligned(g[0]);
    Tensor d_in[8], d_comp[6];
    for (int k = 0; k < 8; ++k) d_in[k] = fresh_like(kept[k]);
    op_backward(d, Eight(kept.data()), kept.data() + 10, kept[8], kept[9], d_out, Eight(d_in), d_comp);
    for (int k = 0; k < 8; ++k) res[1 + k] = d_in[k];
    for (int k = 8; k < n; ++k) res[1 + k] = d_comp[k - 8];
    return res;
  }
};
struct OpMean : torch::autograd::Function<OpMean> {
  static Tensor forward(AutogradContext* ctx, Call* c, const Tensor& q, const Tensor& kc, const Tensor& vc, const Tensor& ks,
                        const Tensor& vs, const Tensor& kw, const Tensor& vw, const Tensor& gate) {
    return OpNode::run(ctx, c);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) { return once(OpNode::grads(ctx, g)); }
};
struct OpLearned : torch::autograd::Function<OpLearned> {
  static Tensor forward(AutogradContext* ctx, Call* c, const Tensor& q, const Tensor& kc, const Tensor& vc, const Tensor& ks,
                        const Tensor& vs, const Tensor& kw, const Tensor& vw, const Tensor& gate, const Tensor& c0,
                        const Tensor& c1, const Tensor& c2, const Tensor& c3, const Tensor& c4, const Tensor& c5) {
    return OpNode::run(ctx, c);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) { return once(OpNode::grads(ctx, g)); }
};

// ---- the layer under bf16 autocast: projections, op and out_proj in one node ----------------------------
// One launch casts x and the nine weights, laid out as the GEMMs read them; the gradients of x and the
// weights leave their GEMMs in fp32, the K / V gradients of the six branches land in one buffer and the bias
// row is summed over its own columns.  The op reads and writes the tokens of out_proj's GEMMs itself.  In place of torch's nodes and modules: 8 x 4096 tokens, 12 heads
// of 64, forward + backward 3165 -> 2984 us; 256 tokens, forward, 271 -> 94.
struct Layer {
  Call c;
  Tensor x, w[8], bias, w_out;
  int64_t B, T, dm, width, n_attn;
};
struct LayerNode : torch::autograd::Function<LayerNode> {
  // keep: what the backward reads; a GEMM's operand only where the gradient that reads it is asked for
  static Tensor run(Layer& l, bool need_grad, variable_list* keep) {
    const NsaDims& m = l.c.d.dims;
    const int64_t rows = l.B * l.T, hd = (int64_t)m.Hq * m.D;
    Tensor xb = l.x.scalar_type() == at::kBFloat16 ? l.x.view({rows, l.dm}) : fresh({rows, l.dm}, at::kBFloat16, l.x);
    Tensor w = fresh({l.width, l.dm}, at::kBFloat16, l.x), bias = fresh({l.width}, at::kBFloat16, l.x),
           w_out = fresh({l.dm, hd}, at::kBFloat16, l.x);
    NsaCastSegment s[NSA_MAX_CAST_SEGMENTS];
    int n = 0;
    auto seg = [&](const float* src, void* dst, int64_t e) { s[n++] = NsaCastSegment{src, dst, (size_t)e}; };
    if (l.x.scalar_type() == at::kFloat) seg(l.x.data_ptr<float>(), xb.data_ptr(), xb.numel());
    char* at_w = (char*)w.data_ptr();
    int64_t row = 0;
    for (int k = 0; k < 8; ++k) {
      seg(l.w[k].data_ptr<float>(), at_w + row * l.dm * 2, l.w[k].numel());
      row += l.w[k].size(0);
    }
    seg(nullptr, at_w + row * l.dm * 2, (l.width - row) * l.dm);
    char* at_b = (char*)bias.data_ptr();
    seg(nullptr, at_b, l.n_attn);
    seg(l.bias.data_ptr<float>(), at_b + l.n_attn * 2, l.bias.numel());
    seg(nullptr, at_b + row * 2, l.width - row);
    seg(l.w_out.data_ptr<float>(), w_out.data_ptr(), w_out.numel());
    check(nsa_cast_bf16_segments(s, n, raw_stream(l.x)));
    Tensor y = at::addmm(bias, xb, w.t());
    Call& c = l.c;
    Tensor q = fresh({m.B, m.Hq, m.T, m.D}, at::kBFloat16, l.x);
    Tensor kv = fresh({6, m.B, m.Hkv, m.T, m.D}, at::kBFloat16, l.x);
    Tensor gate = fresh({m.B, m.Hq, m.T, 3}, at::kBFloat16, l.x);
    check(nsa_split_heads(y.data_ptr(), q.data_ptr(), kv.data_ptr(), gate.data_ptr(), m.B, m.T, m.Hq, m.Hkv, m.D,
                          NSA_DTYPE_BF16, raw_stream(l.x)));
    Tensor saved;
    Tensor tokens = op_forward(c, Eight(q, kv, gate), q, need_grad, &saved, {rows, hd});
    Tensor out = at::mm(tokens, w_out.t()).view({l.B, l.T, l.dm});
    if (keep) {
      bool weights = false;
      for (const Tensor& t : l.w) weights |= t.requires_grad();
      *keep = {q, kv, gate, c.block_idx, saved, weights ? xb : Tensor(), l.x.requires_grad() ? w : Tensor(), w_out,
               l.w_out.requires_grad() ? tokens : Tensor()};
      keep->insert(keep->end(), c.comp, c.comp + 6);
    }
    return out;
  }
  static Tensor forward(AutogradContext* ctx, Layer* l, const Tensor& x, const Tensor& w0, const Tensor& w1, const Tensor& w2,
                        const Tensor& w3, const Tensor& w4, const Tensor& w5, const Tensor& w6, const Tensor& w7,
                        const Tensor& bias, const Tensor& w_out, const Tensor& c0, const Tensor& c1, const Tensor& c2,
                        const Tensor& c3, const Tensor& c4, const Tensor& c5) {
    variable_list keep;
    Tensor out = run(*l, true, &keep);
    ctx->save_for_backward(std::move(keep));
    ctx->saved_data["desc"] = pack(l->c.d);
    ctx->saved_data["x_bf16"] = x.scalar_type() == at::kBFloat16;
    ctx->set_materialize_grads(false);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    variable_list res;
    {
      at::NoGradGuard no_grad;
      res = grads(ctx, g);
    }
    return once(std::move(res));
  }
  static variable_list grads(AutogradContext* ctx, const variable_list& g) {
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    variable_list res(18);                      // l, x, w[8], bias, w_out, comp[6]
    if (!g[0].defined()) return res;
    // x: 0, w: 1..8, bias: 9, w_out: 10, comp: 11..16.  Nothing is done for what no one asks for.
    bool dw_any = false, rows_any = ctx->needs_input_grad(0) || ctx->needs_input_grad(9), op_any = false;
    for (int k = 1; k < 9; ++k) dw_any |= ctx->needs_input_grad(k);
    rows_any |= dw_any;
    for (int k = 11; k < 17; ++k) op_any |= ctx->needs_input_grad(k);
    op_any |= rows_any;
    const NsaAttentionDesc d = unpack(ctx);
    const NsaDims& m = d.dims;
    variable_list kept = ctx->get_saved_variables();
    for (Tensor& t : kept) t = aligned(t);
    const Tensor &kv = kept[1], &xb = kept[5], &w = kept[6], &w_out = kept[7], &tokens = kept[8];
    const int64_t rows = (int64_t)m.B * m.T, hd = (int64_t)m.Hq * m.D, dm = w_out.size(0);
    const int64_t width = nsa_fused_projection_width(m.Hq, m.Hkv, m.D);
    const Tensor dy = aligned(g[0].to(at::kBFloat16)).view({rows, dm});
    if (ctx->needs_input_grad(10)) res[11] = at::mm(dy.t(), tokens, at::kFloat);
    if (!op_any) return res;
    Tensor d_tokens = at::mm(dy, w_out), d_out = fresh({m.B, m.Hq, m.T, m.D}, at::kBFloat16, kv);
    Tensor d_comp[6], d_q = fresh_like(kept[0]), d_kv = fresh_like(kv), d_gate = fresh_like(kept[2]);
    op_backward(d, Eight(kept[0], kv, kept[2]), kept.data() + 9, kept[3], kept[4], d_out, Eight(d_q, d_kv, d_gate), d_comp, &d_tokens);
    for (int k = 0; k < 6; ++k) res[12 + k] = d_comp[k];
    if (!rows_any) return res;
    Tensor d_rows = fresh({rows, width}, at::kBFloat16, kv);
    check(nsa_merge_heads(d_q.data_ptr(), d_kv.data_ptr(), d_gate.data_ptr(), d_rows.data_ptr(), m.B, m.T, m.Hq, m.Hkv, m.D,
                          NSA_DTYPE_BF16, raw_stream(dy)));
    if (ctx->needs_input_grad(0)) {
      Tensor dx = ctx->saved_data["x_bf16"].toBool() ? at::mm(d_rows, w) : at::mm(d_rows, w, at::kFloat);
      res[1] = dx.view({m.B, m.T, dm});
    }
    if (dw_any) {
      const Tensor dw = at::mm(d_rows.t(), xb, at::kFloat);
      int64_t row = 0;
      for (int k = 0; k < 8; ++k) {
        const int64_t n = k == 0 ? hd : k < 7 ? (int64_t)m.Hkv * m.D : 3 * m.Hq;
        res[2 + k] = dw.narrow(0, row, n);
        row += n;
      }
    }
    if (ctx->needs_input_grad(9)) res[10] = d_rows.narrow(1, hd + 6 * (int64_t)m.Hkv * m.D, 3 * m.Hq).sum({0}, false, at::kFloat);
    return res;
  }
};

bool tensor_arg(PyObject* o, Tensor* t) {
  if (!THPVariable_CheckExact(o)) return false;
  *t = THPVariable_Unpack(o);
  return true;
}
bool int_args(PyObject* const* a, int n, int* out) {
  for (int k = 0; k < n; ++k) {
    const long v = PyLong_AsLong(a[k]);
    if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    if (v < INT32_MIN || v > INT32_MAX) return false;
    out[k] = (int)v;
  }
  return true;
}
PyObject* none() { Py_RETURN_NONE; }

// op(q, kc, vc, ks, vs, kw, vw, gate, block_idx | None, compressor tuple | None, block_size, n_sel, window, n_init,
//    n_local, cmp_len, cmp_stride, dq_accumulator, impl) -> (out, block_idx), or None where the call is not plain
PyObject* py_op(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 19 || !plain_state()) return none();
  Call c;
  for (int k = 0; k < 8; ++k)
    if (!tensor_arg(a[k], &c.in[k])) return none();
  const bool given = a[8] != Py_None, learned = a[9] != Py_None;
  if (given && !tensor_arg(a[8], &c.block_idx)) return none();
  if (learned) {
    if (!PyTuple_Check(a[9]) || PyTuple_GET_SIZE(a[9]) != 6) return none();
    for (int k = 0; k < 6; ++k)
      if (!tensor_arg(PyTuple_GET_ITEM(a[9], k), &c.comp[k])) return none();
  }
  int ints[9];
  if (!int_args(a + 10, 9, ints)) return none();
  const Tensor& q = c.in[0];
  if (!q.defined() || !q.is_cuda() || q.device().index() != c10::cuda::current_device()) return none();
  for (int k = 0; k < 8; ++k)
    if (!plain(c.in[k], q.scalar_type(), q.device())) return none();
  if (given && !(c.block_idx.device() == q.device() && c.block_idx.scalar_type() == at::kInt && c.block_idx.is_contiguous())) return none();
  if (q.dim() != 4 || c.in[1].dim() != 4 ||
      !fill_desc(c, q.size(0), q.size(1), c.in[1].size(1), q.size(2), q.size(3), q.scalar_type(), ints, learned, given))
    return none();
  const NsaDims& m = c.d.dims;
  for (int k = 1; k < 7; ++k)
    if (c.in[k].sizes() != at::IntArrayRef({m.B, m.Hkv, m.T, m.D})) return none();
  if (c.in[7].sizes() != at::IntArrayRef({m.B, m.Hq, m.T, 3})) return none();
  if (learned && !comp_ok(c, q.device())) return none();
  bool need = false;
  if (at::GradMode::is_enabled()) {
    for (const Tensor& t : c.in) need |= t.requires_grad();
    for (int k = 0; k < 6 && learned; ++k) need |= c.comp[k].requires_grad();
  }
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    if (!need) {
      Tensor saved;
      at::NoGradGuard no_grad;
      out = op_forward(c, Eight(c.in), c.in[0], false, &saved);
    } else if (learned) {
      out = OpLearned::apply(&c, c.in[0], c.in[1], c.in[2], c.in[3], c.in[4], c.in[5], c.in[6], c.in[7], c.comp[0], c.comp[1],
                             c.comp[2], c.comp[3], c.comp[4], c.comp[5]);
    } else {
      out = OpMean::apply(&c, c.in[0], c.in[1], c.in[2], c.in[3], c.in[4], c.in[5], c.in[6], c.in[7]);
    }
  }
  PyObject* o = THPVariable_Wrap(out);
  if (!o) return nullptr;
  PyObject* idx = given ? (Py_INCREF(a[8]), a[8]) : THPVariable_Wrap(c.block_idx);
  if (!idx) { Py_DECREF(o); return nullptr; }
  PyObject* res = PyTuple_Pack(2, o, idx);
  Py_DECREF(o);
  Py_DECREF(idx);
  return res;
  END_HANDLE_TH_ERRORS
}

// layer(x, (q, kc, vc, ks, vs, kw, vw, gate weights), gate bias, out weight, compressor tuple, block_idx | None, Hq, Hkv,
//       then the integers of op()) -> y, or None where the call is not plain
PyObject* py_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 17 || !plain_state()) return none();
  Layer l;
  Call& c = l.c;
  if (!tensor_arg(a[0], &l.x) || !PyTuple_Check(a[1]) || PyTuple_GET_SIZE(a[1]) != 8 || !PyTuple_Check(a[4]) ||
      PyTuple_GET_SIZE(a[4]) != 6 || !tensor_arg(a[2], &l.bias) || !tensor_arg(a[3], &l.w_out))
    return none();
  for (int k = 0; k < 8; ++k)
    if (!tensor_arg(PyTuple_GET_ITEM(a[1], k), &l.w[k])) return none();
  for (int k = 0; k < 6; ++k)
    if (!tensor_arg(PyTuple_GET_ITEM(a[4], k), &c.comp[k])) return none();
  const bool given = a[5] != Py_None;
  if (given && !tensor_arg(a[5], &c.block_idx)) return none();
  int ints[11];
  if (!int_args(a + 6, 11, ints)) return none();
  const int64_t Hq = ints[0], Hkv = ints[1];
  const Tensor& x = l.x;
  if (!x.defined() || !x.is_cuda() || x.device().index() != c10::cuda::current_device() || x.dim() != 3 || Hq < 1 || Hkv < 1) return none();
  const at::Device dev = x.device();
  l.B = x.size(0); l.T = x.size(1); l.dm = x.size(2);
  if (!plain(x, x.scalar_type(), dev) || (x.scalar_type() != at::kFloat && x.scalar_type() != at::kBFloat16)) return none();
  const int64_t D = l.w[0].dim() == 2 ? l.w[0].size(0) / Hq : 0;
  if (D < 16 || D % 8 || l.dm % 8) return none();
  l.n_attn = (Hq + 6 * Hkv) * D;
  l.width = nsa_fused_projection_width((int)Hq, (int)Hkv, (int)D);
  for (int k = 0; k < 8; ++k) {
    const int64_t r = k == 0 ? Hq * D : k < 7 ? Hkv * D : 3 * Hq;
    if (!plain(l.w[k], at::kFloat, dev) || l.w[k].sizes() != at::IntArrayRef({r, l.dm})) return none();
  }
  if (!plain(l.bias, at::kFloat, dev) || l.bias.sizes() != at::IntArrayRef({3 * Hq})) return none();
  if (!plain(l.w_out, at::kFloat, dev) || l.w_out.sizes() != at::IntArrayRef({l.dm, Hq * D})) return none();
  if (given && !(c.block_idx.device() == dev && c.block_idx.scalar_type() == at::kInt && c.block_idx.is_contiguous())) return none();
  if (!fill_desc(c, l.B, Hq, Hkv, l.T, D, at::kBFloat16, ints + 2, true, given) || !comp_ok(c, dev)) return none();
  bool need = false;
  if (at::GradMode::is_enabled()) {
    need = x.requires_grad() || l.bias.requires_grad();
    for (const Tensor& t : l.w) need |= t.requires_grad();
    for (const Tensor& t : c.comp) need |= t.requires_grad();
    if (!need && l.w_out.requires_grad()) return none();      // the op has no backward then: out_proj is a node by itself
  }
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    if (need) {
      out = LayerNode::apply(&l, x, l.w[0], l.w[1], l.w[2], l.w[3], l.w[4], l.w[5], l.w[6], l.w[7], l.bias, l.w_out, c.comp[0],
                             c.comp[1], c.comp[2], c.comp[3], c.comp[4], c.comp[5]);
    } else {
      at::NoGradGuard no_grad;
      out = LayerNode::run(l, false, nullptr);
    }
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

PyObject* py_set_error(PyObject*, PyObject* cls) {
  Py_INCREF(cls);
  g_error = cls;
  return none();
}

PyMethodDef kMethods[] = {
    {"op", (PyCFunction)(void (*)(void))py_op, METH_FASTCALL, "whole op, or None where the call is not plain"},
    {"layer", (PyCFunction)(void (*)(void))py_layer, METH_FASTCALL, "layer under bf16 autocast, or None where the call is not plain"},
    {"set_error", py_set_error, METH_O, "exception class of failed library calls"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_nsa_torch", nullptr, -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit__nsa_torch() {
  PyObject* m = PyModule_Create(&kModule);
  if (m && PyModule_AddStringConstant(m, "torch_version", NSA_TORCH_VERSION) != 0) Py_CLEAR(m);
  return m;
}
