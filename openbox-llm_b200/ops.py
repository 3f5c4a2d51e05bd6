"""Host side of the NSA attention path: the reference's operator interface on top of the
C-ABI library.

Names, argument meaning and error behaviour follow the reference modules they replace:
  selection_forward_triton, selection_forward_reference   nsa_selection_kernel.py:55-213
  selection_backward_triton, SelectionAttnTriton,
  selection_attn_triton                                    nsa_selection_backward.py:156-369
  build_block_to_query_csr                                 nsa_fsa.py:14-64
  _RangeAttn, window_attn_triton, compression_attn_triton,
  block_mean_pool, nsa_fused_forward                       nsa_fused_kernel.py:521-573
`nsa_attention` is the one addition: the whole op (pooling, compression attention, block
scoring + top-n, selection, window, gate) behind one autograd.Function.
"""
import ctypes
import functools

import torch
from torch.autograd import forward_ad

from . import _lib as L

MODE_WINDOW = L.MODE_WINDOW
MODE_COMPRESS = L.MODE_COMPRESS
MODE_COMPRESS_STRIDED = L.MODE_COMPRESS_STRIDED

_impl = "auto"
_dq_accumulator = False


def set_impl(name: str):
    """Choose the kernel family: 'auto' (tcgen05 where the shape fits; selection on 16- and 32-token
    blocks with the probabilities in three bf16 terms, 24 bits as on the CUDA cores; fp32 heads of 64 with every product as six
    products of bf16 terms on the tensor cores), 'simt' (the CUDA cores, products by FFMA), or 'tc' (tcgen05, or an error; takes 16- and
    32-token blocks too, with bf16 probabilities as on 64-token blocks)."""
    global _impl
    assert name in L.IMPL
    _impl = name


def get_impl() -> str:
    return _impl


def set_dq_accumulator(on: bool):
    """Whole-op backward on tcgen05 shapes.  False (default): every branch keeps bf16 dQ partials
    (one slot per key tile a query attends) and one kernel adds them in a fixed order: dq is
    bit-reproducible, at the price of the partial buffers.  True: the window and compression
    branches add their dQ tiles into one fp32 accumulator by TMA reduce-add instead: no partial
    buffers for them (23 GB less at B=8, T=32K; the way to run compression strides that would need
    dozens of slots), but the L2 reduction rate bounds those kernels (they run about 1.7 times
    longer) and the order of the adds, hence the last bits of dq, varies from run to run."""
    global _dq_accumulator
    _dq_accumulator = bool(on)


def get_dq_accumulator() -> bool:
    return _dq_accumulator


def set_option(name: str, value: int):
    """Library tuning switch (see nsa_set_option in include/nsa_b200.h)."""
    L.check(L.lib().nsa_set_option(name.encode(), int(value)))
    _op_desc.cache_clear()            # workspace sizes depend on the switches


def tc_supported(B, Hq, Hkv, T, D, dtype, block_size=64) -> bool:
    code = L.DTYPE_BF16 if dtype == torch.bfloat16 else L.DTYPE_F32
    return bool(L.lib().nsa_tc_supported(L.dims(B, Hq, Hkv, T, D, code), block_size))


def _check_qkv(q, k, v):
    B, Hq, T, D = q.shape
    assert k.shape == v.shape and k.shape[0] == B and k.shape[3] == D
    assert Hq % k.shape[1] == 0, "GQA needs Hq divisible by Hkv"
    assert D in (16, 32, 64, 128), "head dim must be a power of two <= 128"
    assert q.stride(-1) == 1 and k.stride(-1) == 1 and v.stride(-1) == 1
    assert q.dtype == k.dtype == v.dtype
    return B, Hq, k.shape[1], T, D


# ---------------------------------------------------------------------------------------
# raw launch wrappers
# ---------------------------------------------------------------------------------------
@L.on_device
def range_attn_forward(q, k, v, mode, window, block_size, out=None):
    """o, lse of the window (mode 0) or compression (mode 1) branch.  `out` = (o, lse) makes the
    kernel write into existing contiguous tensors (the whole op keeps its three branches' outputs
    and statistics in one tensor each)."""
    B, Hq, Hkv, T, D = _check_qkv(q, k, v)
    q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
    o, lse = out if out is not None else (
        torch.empty_like(q), torch.empty(B, Hq, T, device=q.device, dtype=torch.float32))
    d = L.dims(B, Hq, Hkv, T, D, L.dtype_code(q))
    L.check(L.lib().nsa_range_attn_fwd(L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(o), L.ptr(lse), d,
                                       k.shape[2], mode, int(window), int(block_size),
                                       L.IMPL[_impl], L.stream()))
    return o, lse


@L.on_device
def range_attn_backward(q, k, v, o, lse, do, mode, window, block_size, row_scale=None, row_dot=None,
                        defer_dq=False):
    """dq, dk, dv of a range branch.  With row_scale / row_dot (see nsa_gate_combine_bwd_rows) `do`
    is the whole op's upstream gradient and the gate factor is applied inside the kernel.
    defer_dq (tcgen05 shapes only): returns (workspace, dk, dv), the dQ partials staying in the
    workspace for nsa_dq_reduce3."""
    B, Hq, Hkv, T, D = _check_qkv(q, k, v)
    q, k, v, o, do = (t.contiguous() for t in (q, k, v, o, do))
    dq = None if defer_dq else torch.empty_like(q)
    dk, dv = torch.empty_like(k), torch.empty_like(v)
    d = L.dims(B, Hq, Hkv, T, D, L.dtype_code(q))
    nws = L.lib().nsa_range_attn_bwd_workspace_bytes(d, k.shape[2], mode, int(window), L.IMPL[_impl])
    ws = L.workspace(nws, q.device)
    L.check(L.lib().nsa_range_attn_bwd(L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(o), L.ptr(lse),
                                       L.ptr(do), L.ptr(dq), L.ptr(dk), L.ptr(dv), d, k.shape[2],
                                       mode, int(window), int(block_size), L.ptr(row_scale),
                                       L.ptr(row_dot), L.ptr(ws), nws, L.IMPL[_impl], L.stream()))
    return (ws if defer_dq else dq), dk, dv


@L.on_device
def range_attn_backward_acc(q, k, v, o, lse, do, mode, window, block_size, row_scale, row_dot, dq_acc):
    """dk, dv of a gated range branch on a tcgen05 shape; its dQ is added to dq_acc
    [B*Hkv, T, G, D] float32 (see nsa_range_attn_bwd_acc)."""
    B, Hq, Hkv, T, D = _check_qkv(q, k, v)
    q, k, v, do = (t.contiguous() for t in (q, k, v, do))
    dk, dv = torch.empty_like(k), torch.empty_like(v)
    d = L.dims(B, Hq, Hkv, T, D, L.dtype_code(q))
    nws = L.lib().nsa_range_attn_bwd_acc_workspace_bytes(d, k.shape[2], mode, int(window))
    ws = L.workspace(nws, q.device)
    L.check(L.lib().nsa_range_attn_bwd_acc(L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(o), L.ptr(lse), L.ptr(do),
                                           L.ptr(dq_acc), L.ptr(dk), L.ptr(dv), d, k.shape[2], mode,
                                           int(window), int(block_size), L.ptr(row_scale),
                                           L.ptr(row_dot), L.ptr(ws), nws, L.stream()))
    return dk, dv


@L.on_device
def selection_plan(q, k, block_idx, block_size):
    """The index structures the tcgen05 selection kernels walk (CSR, pair map, work list), built
    once for a block list so that forward and backward need not each build them; None when the
    shape is not served by those kernels.  Opaque uint8 tensor."""
    B, Hq, T, D = q.shape
    S = block_idx.shape[-1]
    if _impl == "simt" or S == 0:
        return None
    d = L.dims(B, Hq, k.shape[1], T, D, L.dtype_code(q))
    n = L.lib().nsa_selection_plan_bytes(d, S, int(block_size))
    if n == 0:
        return None
    idx = block_idx.to(torch.int32).contiguous()
    plan = torch.empty(n, dtype=torch.uint8, device=q.device)
    L.check(L.lib().nsa_selection_plan_build(L.ptr(idx), d, S, int(block_size), L.ptr(plan), n, L.stream()))
    return plan


@L.on_device
def selection_forward_triton(q, k, v, block_idx, block_size, return_lse=False, out=None, plan=None):
    """nsa_selection_kernel.py:175-213.  q [B,Hq,T,D], k/v [B,Hkv,T,D], block_idx [B,Hkv,T,S].
    `out` = (o, lse): write into existing contiguous tensors; `plan`: see selection_plan (neither
    is in the reference's signature)."""
    B, Hq, Hkv, T, D = _check_qkv(q, k, v)
    S = block_idx.shape[-1]
    assert block_idx.shape[:3] == (B, Hkv, T)
    assert block_size >= 16, "block_size must be >= 16 (tl.dot inner dim)"
    q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
    idx = block_idx.to(torch.int32).contiguous()
    o, lse = out if out is not None else (
        torch.empty_like(q), torch.empty(B, Hq, T, device=q.device, dtype=torch.float32))
    d = L.dims(B, Hq, Hkv, T, D, L.dtype_code(q))
    nws = L.lib().nsa_selection_fwd_workspace_bytes(d, S, block_size, L.IMPL[_impl])
    ws = L.workspace(nws, q.device)
    if plan is not None:
        L.check(L.lib().nsa_selection_fwd_planned(L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(idx), L.ptr(o),
                                                  L.ptr(lse), d, S, int(block_size), L.ptr(ws), nws,
                                                  L.ptr(plan), L.stream()))
    else:
        L.check(L.lib().nsa_selection_fwd(L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(idx), L.ptr(o),
                                          L.ptr(lse), d, S, int(block_size), L.ptr(ws), nws,
                                          L.IMPL[_impl], L.stream()))
    return (o, lse) if return_lse else o


@L.on_device
def _selection_backward(q, k, v, block_idx, block_size, do, o, lse, row_scale=None, row_dot=None,
                        defer_dq=False, plan=None):
    B, Hq, Hkv, T, D = _check_qkv(q, k, v)
    S = block_idx.shape[-1]
    assert block_size >= 16
    q, k, v, o, do = (t.contiguous() for t in (q, k, v, o, do))
    idx = block_idx.to(torch.int32).contiguous()
    dq = None if defer_dq else torch.empty_like(q)
    dk, dv = torch.empty_like(k), torch.empty_like(v)
    d = L.dims(B, Hq, Hkv, T, D, L.dtype_code(q))
    nws = L.lib().nsa_selection_bwd_workspace_bytes(d, S, block_size, L.IMPL[_impl])
    ws = L.workspace(nws, q.device)
    if plan is not None:
        L.check(L.lib().nsa_selection_bwd_planned(L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(idx), L.ptr(o),
                                                  L.ptr(lse), L.ptr(do), L.ptr(dq), L.ptr(dk), L.ptr(dv), d, S,
                                                  int(block_size), L.ptr(row_scale), L.ptr(row_dot), L.ptr(ws),
                                                  nws, L.ptr(plan), L.stream()))
    else:
        L.check(L.lib().nsa_selection_bwd(L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(idx), L.ptr(o),
                                          L.ptr(lse), L.ptr(do), L.ptr(dq), L.ptr(dk), L.ptr(dv), d, S,
                                          int(block_size), L.ptr(row_scale), L.ptr(row_dot), L.ptr(ws),
                                          nws, L.IMPL[_impl], L.stream()))
    return (ws if defer_dq else dq), dk, dv


def selection_backward_triton(q, k, v, block_idx, block_size, do, o):
    """nsa_selection_backward.py:156-189: dq, dk, dv from (q,k,v,block_idx,dO,O); the softmax
    statistics are recomputed by a forward pass because this signature carries no LSE."""
    _, lse = selection_forward_triton(q, k, v, block_idx, block_size, return_lse=True)
    return _selection_backward(q, k, v, block_idx, block_size, do, o, lse)


@torch.no_grad()
@L.on_device
def build_block_to_query_csr(block_idx, block_size):
    """nsa_fsa.py:14-64: (q_of_block [P], block_offsets [B,Hkv,n_blk+1], pair_bh [P]), int32."""
    B, Hkv, T, S = block_idx.shape
    idx = block_idx.to(torch.int32).contiguous()
    n_blk = T // block_size
    dev = idx.device
    cap = max(B * Hkv * T * S, 1)
    q_of_block = torch.empty(cap, dtype=torch.int32, device=dev)
    pair_bh = torch.empty(cap, dtype=torch.int32, device=dev)
    offsets = torch.zeros(B, Hkv, n_blk + 1, dtype=torch.int32, device=dev)
    nws = L.lib().nsa_csr_workspace_bytes(B, Hkv, T, S, block_size)
    ws = L.workspace(nws, dev)
    L.check(L.lib().nsa_build_block_to_query_csr(L.ptr(idx), B, Hkv, T, S, int(block_size),
                                                 L.ptr(q_of_block), L.ptr(offsets), L.ptr(pair_bh),
                                                 L.ptr(ws), nws, L.stream()))
    P = int(offsets.view(-1)[-1].item()) if offsets.numel() else 0
    return q_of_block[:P], offsets, pair_bh[:P]


def _pool_dims(x, block_size):
    B, H, T, D = x.shape
    return B, H, T, D, T // block_size


@L.on_device
def _mean_pool_fwd(x, block_size):
    B, H, T, D, n_blk = _pool_dims(x, block_size)
    x = x.contiguous()
    out = torch.empty(B, H, n_blk, D, device=x.device, dtype=x.dtype)
    L.check(L.lib().nsa_block_mean_pool_fwd(L.ptr(x), L.ptr(out), B, H, T, D, int(block_size),
                                            L.dtype_code(x), L.stream()))
    return out


@L.on_device
def _mean_pool_bwd(d_out, T, block_size):
    B, H, n_blk, D = d_out.shape
    d_out = d_out.contiguous()
    dx = torch.empty(B, H, T, D, device=d_out.device, dtype=d_out.dtype)
    L.check(L.lib().nsa_block_mean_pool_bwd(L.ptr(d_out), L.ptr(dx), B, H, T, D, int(block_size),
                                            L.dtype_code(d_out), L.stream()))
    return dx


def n_summaries(T, cmp_len, cmp_stride):
    """Complete windows of cmp_len tokens every cmp_stride tokens inside T tokens."""
    return (T - cmp_len) // cmp_stride + 1 if T >= cmp_len else 0


@L.on_device
def _compress_fwd(x, intra, logits, proj, block_size, stride=None):
    stride = block_size if stride is None else stride
    B, H, T, D = x.shape
    x = x.contiguous()
    out = torch.empty(B, H, n_summaries(T, block_size, stride), D, device=x.device, dtype=x.dtype)
    L.check(L.lib().nsa_block_compress_strided_fwd(L.ptr(x), L.ptr(intra), L.ptr(logits), L.ptr(proj),
                                                   L.ptr(out), B, H, T, D, int(block_size), int(stride),
                                                   L.dtype_code(x), L.stream()))
    return out


@L.on_device
def _compress_bwd(x, intra, logits, proj, d_out, block_size, stride=None):
    stride = block_size if stride is None else stride
    B, H, T, D = x.shape
    x, d_out = x.contiguous(), d_out.contiguous()
    dx = torch.empty_like(x)
    d_intra, d_logits, d_proj = (torch.empty_like(t) for t in (intra, logits, proj))
    nws = L.lib().nsa_block_compress_strided_bwd_workspace_bytes(B, H, T, D, int(block_size), int(stride))
    ws = L.workspace(nws, x.device)
    L.check(L.lib().nsa_block_compress_strided_bwd(
        L.ptr(x), L.ptr(intra), L.ptr(logits), L.ptr(proj), L.ptr(d_out), L.ptr(dx), L.ptr(d_intra),
        L.ptr(d_logits), L.ptr(d_proj), B, H, T, D, int(block_size), int(stride), L.dtype_code(x),
        L.ptr(ws), nws, L.stream()))
    return dx, d_intra, d_logits, d_proj


@torch.no_grad()
@L.on_device
def topn_blocks(q, k_cmp, lse_cmp, block_size, n_sel, return_importance=False, n_init_blocks=0,
                n_local_blocks=0, cmp_len=None, cmp_stride=None):
    """Block scoring + top-n (nsa_model.py:343-355): block_idx [B,Hkv,T,n_sel] int32, ordered by
    (importance descending, index ascending), -1 where fewer than n_sel blocks are causally
    valid.  lse_cmp is the LSE of the compression branch for the same q, k_cmp.
    Not in the reference: n_init_blocks / n_local_blocks put the first blocks and the most
    recent blocks, the one holding t included, ahead of the scored ones; cmp_len / cmp_stride
    (default block_size) say that k_cmp are summaries of cmp_len tokens every cmp_stride tokens
    while the selection blocks stay block_size tokens."""
    B, Hq, T, D = q.shape
    Hkv, n_cmp = k_cmp.shape[1], k_cmp.shape[2]
    cl = int(block_size if cmp_len is None else cmp_len)
    cs = int(cl if cmp_stride is None else cmp_stride)
    aligned = cl == cs == int(block_size)
    q, k_cmp, lse_cmp = q.contiguous(), k_cmp.contiguous(), lse_cmp.contiguous()
    idx = torch.empty(B, Hkv, T, n_sel, device=q.device, dtype=torch.int32)
    cols = n_cmp if aligned else (T + int(block_size) - 1) // int(block_size)
    imp = torch.empty(B, Hkv, T, cols, device=q.device, dtype=torch.float32) if return_importance else None
    d = L.dims(B, Hq, Hkv, T, D, L.dtype_code(q))
    L.check(L.lib().nsa_topn_blocks_general(L.ptr(q), L.ptr(k_cmp), L.ptr(lse_cmp), L.ptr(idx), L.ptr(imp),
                                            d, n_cmp, cl, cs, int(block_size), int(n_sel),
                                            int(n_init_blocks), int(n_local_blocks), L.IMPL[_impl],
                                            L.stream()))
    return (idx, imp) if return_importance else idx


@L.on_device
def _gate_fwd(o_cmp, o_slc, o_win, gate):
    B, Hq, T, D = o_cmp.shape
    out = torch.empty_like(o_cmp)
    d = L.dims(B, Hq, 1, T, D, L.dtype_code(o_cmp))
    L.check(L.lib().nsa_gate_combine_fwd(L.ptr(o_cmp), L.ptr(o_slc), L.ptr(o_win), L.ptr(gate),
                                         L.ptr(out), d, L.stream()))
    return out


@L.on_device
def _gate_bwd(o_cmp, o_slc, o_win, gate, d_out):
    B, Hq, T, D = o_cmp.shape
    d_out = d_out.contiguous()
    dc, ds, dw = (torch.empty_like(o_cmp) for _ in range(3))
    dg = torch.empty_like(gate)
    d = L.dims(B, Hq, 1, T, D, L.dtype_code(o_cmp))
    L.check(L.lib().nsa_gate_combine_bwd(L.ptr(o_cmp), L.ptr(o_slc), L.ptr(o_win), L.ptr(gate),
                                         L.ptr(d_out), L.ptr(dc), L.ptr(ds), L.ptr(dw), L.ptr(dg),
                                         d, L.stream()))
    return dc, ds, dw, dg


# ---------------------------------------------------------------------------------------
# autograd boundary (same classes and callables as the reference)
# ---------------------------------------------------------------------------------------
class _RangeAttn(torch.autograd.Function):
    """nsa_fused_kernel.py:521-534; additionally keeps the LSE so backward is one pass."""

    @staticmethod
    def forward(ctx, q, k, v, mode, window, block_size):
        o, lse = range_attn_forward(q, k, v, mode, window, block_size)
        ctx.save_for_backward(q, k, v, o, lse)
        ctx.mode, ctx.window, ctx.block_size = mode, window, block_size
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse = ctx.saved_tensors
        dq, dk, dv = range_attn_backward(q, k, v, o, lse, do, ctx.mode, ctx.window, ctx.block_size)
        return dq, dk, dv, None, None, None


def window_attn_triton(q, k, v, window):
    return _RangeAttn.apply(q, k, v, MODE_WINDOW, window, 0)


def compression_attn_triton(q, k_cmp, v_cmp, block_size, stride=0):
    """nsa_fused_kernel.py:541-543.  stride (not in the reference): the summaries are windows of
    block_size tokens every `stride` tokens; 0 = block_size."""
    if stride:
        return _RangeAttn.apply(q, k_cmp, v_cmp, MODE_COMPRESS_STRIDED, stride, block_size)
    return _RangeAttn.apply(q, k_cmp, v_cmp, MODE_COMPRESS, 0, block_size)


class SelectionAttnTriton(torch.autograd.Function):
    """nsa_selection_backward.py:337-365: block_idx and block_size get no gradient."""

    @staticmethod
    def forward(ctx, q, k, v, block_idx, block_size):
        # the index structures of the block list are built once for forward and backward (the
        # reference builds its CSR in each: nsa_selection_kernel.py:199-201, nsa_selection_backward.py:356-358)
        plan = None
        if q.is_cuda and q.dtype == torch.bfloat16 and any(ctx.needs_input_grad[:3]):
            plan = selection_plan(q, k, block_idx, block_size)
        o, lse = selection_forward_triton(q, k, v, block_idx, block_size, return_lse=True, plan=plan)
        ctx.save_for_backward(q, k, v, block_idx, o, lse)
        ctx.block_size, ctx.sel_plan = block_size, plan
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, block_idx, o, lse = ctx.saved_tensors
        dq, dk, dv = _selection_backward(q, k, v, block_idx, ctx.block_size, do, o, lse, plan=ctx.sel_plan)
        return dq, dk, dv, None, None


def selection_attn_triton(q, k, v, block_idx, block_size):
    return SelectionAttnTriton.apply(q, k, v, block_idx, block_size)


class _MeanPool(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, block_size):
        ctx.T, ctx.block_size = x.shape[2], block_size
        return _mean_pool_fwd(x, block_size)

    @staticmethod
    def backward(ctx, d_out):
        return _mean_pool_bwd(d_out, ctx.T, ctx.block_size), None


def block_mean_pool(x, block_size):
    """nsa_fused_kernel.py:549-554: [B,Hkv,T,D] -> [B,Hkv,n_blk,D]."""
    return _MeanPool.apply(x, block_size)


class _BlockCompress(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, intra_pos, pool_logits, proj_weight, block_size, stride):
        intra, logits, proj = (t.detach().float().contiguous() for t in (intra_pos, pool_logits, proj_weight))
        ctx.save_for_backward(x, intra, logits, proj)
        ctx.block_size, ctx.stride = block_size, stride
        ctx.param_dtypes = (intra_pos.dtype, pool_logits.dtype, proj_weight.dtype)
        return _compress_fwd(x, intra, logits, proj, block_size, stride)

    @staticmethod
    def backward(ctx, d_out):
        x, intra, logits, proj = ctx.saved_tensors
        dx, di, dl, dp = _compress_bwd(x, intra, logits, proj, d_out, ctx.block_size, ctx.stride)
        a, b, c = ctx.param_dtypes
        return dx, di.to(a), dl.to(b), dp.to(c), None, None


def block_compress(x, intra_pos, pool_logits, proj_weight, block_size, stride=None):
    """BlockCompressor.forward (nsa_model.py:118-123) on the block view of x [B,Hkv,T,D];
    with stride < block_size on overlapping windows (not in the reference)."""
    return _BlockCompress.apply(x, intra_pos, pool_logits, proj_weight, block_size, stride)


class _GateCombine(torch.autograd.Function):
    @staticmethod
    def forward(ctx, o_cmp, o_slc, o_win, gate_logits):
        o_cmp, o_slc, o_win = (t.contiguous() for t in (o_cmp, o_slc, o_win))
        gate = gate_logits.to(o_cmp.dtype).contiguous()
        ctx.save_for_backward(o_cmp, o_slc, o_win, gate)
        ctx.gate_dtype = gate_logits.dtype
        return _gate_fwd(o_cmp, o_slc, o_win, gate)

    @staticmethod
    def backward(ctx, d_out):
        o_cmp, o_slc, o_win, gate = ctx.saved_tensors
        dc, ds, dw, dg = _gate_bwd(o_cmp, o_slc, o_win, gate, d_out)
        return dc, ds, dw, dg.to(ctx.gate_dtype)


def gate_combine(o_cmp, o_slc, o_win, gate_logits):
    """sigmoid(gate)[...,0]*o_cmp + [...,1]*o_slc + [...,2]*o_win (nsa_model.py:366-368)."""
    return _GateCombine.apply(o_cmp, o_slc, o_win, gate_logits)


# ---------------------------------------------------------------------------------------
# projection glue of the layer (nsa_model.py:192-194, 325-329, 358-359, 366-369)
# ---------------------------------------------------------------------------------------
def fused_projection_width(Hq, Hkv, D):
    """Row width of the fused projection: q, six K/V projections, 3*Hq gate logits padded to 8."""
    return int(L.lib().nsa_fused_projection_width(Hq, Hkv, D))


@L.on_device
def _split_heads_launch(y, q, kv, gate, Hq, Hkv, D, merge):
    B, T = y.shape[0], y.shape[1]
    fn = L.lib().nsa_merge_heads if merge else L.lib().nsa_split_heads
    if merge:
        L.check(fn(L.ptr(q), L.ptr(kv), L.ptr(gate), L.ptr(y), B, T, Hq, Hkv, D, L.dtype_code(y), L.stream()))
    else:
        L.check(fn(L.ptr(y), L.ptr(q), L.ptr(kv), L.ptr(gate), B, T, Hq, Hkv, D, L.dtype_code(y), L.stream()))


class _SplitHeads(torch.autograd.Function):
    """Rows [B,T,W] of the fused projection -> q [B,Hq,T,D], kv [6,B,Hkv,T,D] (kc, vc, ks, vs, kw,
    vw), gate logits [B,Hq,T,3], in one pass; backward assembles the gradient rows in one pass."""

    @staticmethod
    def forward(ctx, y, Hq, Hkv, D):
        B, T, W = y.shape
        assert W == fused_projection_width(Hq, Hkv, D), "row width does not match the head counts"
        y = y.contiguous()
        q = torch.empty(B, Hq, T, D, device=y.device, dtype=y.dtype)
        kv = torch.empty(6, B, Hkv, T, D, device=y.device, dtype=y.dtype)
        gate = torch.empty(B, Hq, T, 3, device=y.device, dtype=y.dtype)
        _split_heads_launch(y, q, kv, gate, Hq, Hkv, D, False)
        ctx.cfg = (Hq, Hkv, D, W)
        return q, kv, gate

    @staticmethod
    def backward(ctx, dq, dkv, dgate):
        Hq, Hkv, D, W = ctx.cfg
        B, _, T, _ = dq.shape
        dq, dkv, dgate = dq.contiguous(), dkv.contiguous(), dgate.contiguous()
        dy = torch.empty(B, T, W, device=dq.device, dtype=dq.dtype)
        _split_heads_launch(dy, dq, dkv, dgate, Hq, Hkv, D, True)
        return dy, None, None, None


def split_heads(y, Hq, Hkv, D):
    return _SplitHeads.apply(y, Hq, Hkv, D)


@L.on_device
def _swap_heads_tokens(x, to_tokens):
    if to_tokens:
        B, H, T, D = x.shape
        out = torch.empty(B, T, H, D, device=x.device, dtype=x.dtype)
    else:
        B, T, H, D = x.shape
        out = torch.empty(B, H, T, D, device=x.device, dtype=x.dtype)
    L.check(L.lib().nsa_swap_heads_tokens(L.ptr(x), L.ptr(out), B, H, T, D, L.dtype_code(x), int(to_tokens),
                                          L.stream()))
    return out


class _HeadsToTokens(torch.autograd.Function):
    """[B,H,T,D] -> [B,T,H*D] (what out_proj reads, nsa_model.py:369); backward the other way."""

    @staticmethod
    def forward(ctx, x):
        ctx.D = x.shape[3]
        out = _swap_heads_tokens(x.contiguous(), True)
        return out.view(out.shape[0], out.shape[1], -1)

    @staticmethod
    def backward(ctx, d_out):
        B, T, HD = d_out.shape
        return _swap_heads_tokens(d_out.contiguous().view(B, T, HD // ctx.D, ctx.D), False)


def heads_to_tokens(x):
    return _HeadsToTokens.apply(x)


def nsa_fused_forward(q, kc, vc, ks, vs, kw, vw, gate_logits, block_idx, block_size, window):
    """nsa_fused_kernel.py:560-573: the three branches with a given block_idx, mean pooling."""
    bs = int(block_size)
    assert q.stride(-1) == 1
    return _op(q, (kc, vc, ks, vs, kw, vw), gate_logits, block_idx, bs, 0, window, (0, 0, bs, bs), None)[0]


@functools.lru_cache(maxsize=512)
def _op_desc(B, Hq, Hkv, T, D, dtype, block_size, n_sel, window, n_init, n_local, cmp_len, cmp_stride, learned,
             given_lists, need_grad, dq_accumulator, impl):
    """Descriptor of a whole-op call and the bytes it keeps and needs (saved, forward, backward)."""
    d = L.NsaAttentionDesc(L.dims(B, Hq, Hkv, T, D, dtype), block_size, n_sel, window, n_init, n_local, cmp_len,
                           cmp_stride, int(learned), int(given_lists), int(need_grad), int(dq_accumulator), impl)
    sizes = [ctypes.c_size_t() for _ in range(3)]
    L.check(L.lib().nsa_attention_sizes(d, *sizes))
    return (d, *(x.value for x in sizes))


def _aligned(t):
    """t, or a copy of it where it does not start on a 16-byte boundary."""
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _op_forward(q, kv, gate_logits, block_idx, block_size, n_sel, window, forced, comp, need_grad):
    """Forward of the whole op: (out, block_idx, what backward needs).  forced = (n_init, n_local,
    summary length, summary stride); comp: the six compressor parameters, or None for mean pooling."""
    B, Hq, T, D = q.shape
    Hkv = kv[0].shape[1]
    dtype = L.dtype_code(q)
    assert q.is_cuda, "libnsa_b200 needs CUDA tensors; there is no CPU path"
    assert Hq % Hkv == 0, "GQA needs Hq divisible by Hkv"
    assert D in (16, 32, 64, 128), "head dim must be a power of two <= 128"
    assert block_size >= 16, "block_size must be >= 16 (tl.dot inner dim)"
    dev = q.device
    tensors = [q, *kv]
    assert kv[0].shape == (B, Hkv, T, D)          # and the other five like it (_op)
    for t in kv:
        assert t.dtype == q.dtype
    gate = gate_logits if gate_logits.dtype == q.dtype else gate_logits.to(q.dtype)
    tensors.append(gate)
    given = block_idx is not None
    if given:
        assert block_idx.shape[:3] == (B, Hkv, T)
        n_sel = block_idx.shape[3]
        block_idx = block_idx.to(torch.int32).contiguous()
        tensors.append(block_idx)
    cp = [] if comp is None else [t.detach().float().contiguous() for t in comp]
    for t in (*tensors, *cp):
        if t.device != dev:
            raise L.NsaError(f"libnsa_b200: tensors on different devices ({dev} and {t.device})")
    if comp is None:
        assert forced[2] == forced[3] == block_size, "mean pooling is defined on the aligned grid only"
    if torch.cuda.current_device() != dev.index:
        with torch.cuda.device(dev):
            return _op_forward(q, kv, gate_logits, block_idx, block_size, n_sel, window, forced, comp, need_grad)
    for i, t in enumerate(tensors[:8]):
        if not t.is_contiguous():
            # as _check_qkv: the rows of the attention calls are dense (the pooling takes any kc, vc)
            assert i not in (3, 4, 5, 6) or t.stride(-1) == 1
            tensors[i] = t.contiguous()
    tensors = tensors[:8]
    in_ptrs, cp_ptrs = [t.data_ptr() for t in tensors], [t.data_ptr() for t in cp]
    # the pooling reads these as 16-byte vectors; a view may start anywhere
    if any(p % 16 for p in (in_ptrs[1], in_ptrs[2], *cp_ptrs)):
        tensors[1:3] = map(_aligned, tensors[1:3])
        cp = [_aligned(t) for t in cp]
        in_ptrs, cp_ptrs = [t.data_ptr() for t in tensors], [t.data_ptr() for t in cp]
    if not given:
        block_idx = torch.empty(B, Hkv, T, n_sel, device=dev, dtype=torch.int32)
    desc, saved_bytes, fwd_bytes, bwd_bytes = _op_desc(
        B, Hq, Hkv, T, D, dtype, int(block_size), int(n_sel), int(window), *forced, comp is not None, given, need_grad,
        _dq_accumulator, L.IMPL[_impl])
    out = torch.empty(B, Hq, T, D, device=dev, dtype=q.dtype)
    saved = torch.empty(saved_bytes + (0 if need_grad else fwd_bytes) + 1, device=dev, dtype=torch.uint8)
    ws, ws_ptr = None, saved.data_ptr() + saved_bytes
    if need_grad and fwd_bytes:
        ws = L.workspace(fwd_bytes, dev)
        ws_ptr = ws.data_ptr()
    ptrs = L.OP_TENSORS(*in_ptrs, *(cp_ptrs or (None,) * 6), block_idx.data_ptr(), out.data_ptr())
    L.check(L.lib().nsa_attention_fwd(desc, ptrs, saved.data_ptr(), ws_ptr, fwd_bytes, L.raw_stream(dev)))
    if L.CHECK_STATUS_EVERY_CALL:
        L.check_device_status()
    return out, block_idx, (tensors, cp, saved, desc, bwd_bytes)


class _Once(torch.autograd.Function):
    """Gradients that cannot be differentiated again, where a graph of the backward is asked for."""

    @staticmethod
    def forward(ctx, g):
        return g.detach()

    @staticmethod
    def backward(ctx, _):
        raise RuntimeError("libnsa_b200: the gradients of the op cannot be differentiated again")


class _NSAAttention(torch.autograd.Function):
    """The whole op in one node: pooling -> compression attention (+LSE) -> block scoring and
    top-n -> selection attention -> window attention -> gate combine.  Saves q once."""

    @staticmethod
    def forward(ctx, q, kc, vc, ks, vs, kw, vw, gate_logits, block_size, n_sel, window, block_idx, forced, *comp):
        out, block_idx, (tensors, cp, saved, desc, bwd_bytes) = _op_forward(
            q, (kc, vc, ks, vs, kw, vw), gate_logits, block_idx, block_size, n_sel, window, forced, comp or None, True)
        ctx.save_for_backward(*tensors, block_idx, saved, *cp)
        ctx.cfg = (desc, bwd_bytes, gate_logits.dtype, tuple(t.dtype for t in comp))
        ctx.mark_non_differentiable(block_idx)
        ctx.set_materialize_grads(False)
        return out, block_idx

    @staticmethod
    def backward(ctx, d_out, _d_idx):
        desc, bwd_bytes, gate_dtype, comp_dtypes = ctx.cfg
        if d_out is None:
            return (None,) * (13 + len(comp_dtypes))
        kept = ctx.saved_tensors
        if any(t.data_ptr() % 16 for t in kept):
            kept = [_aligned(t) for t in kept]
        tensors, block_idx, saved, cp = kept[:8], kept[8], kept[9], kept[10:]
        dev = saved.device
        if torch.cuda.current_device() != dev.index:
            with torch.cuda.device(dev):
                return _NSAAttention.backward(ctx, d_out, _d_idx)
        if d_out.device != dev:
            raise L.NsaError(f"libnsa_b200: tensors on different devices ({dev} and {d_out.device})")
        assert d_out.dtype == tensors[0].dtype
        d_out = _aligned(d_out.contiguous())
        grads = [torch.empty_like(t) for t in tensors]
        d_cp = [torch.empty_like(t) for t in cp]
        ws = L.workspace(bwd_bytes, dev)
        ptrs = L.OP_TENSORS(*[t.data_ptr() for t in tensors], *([t.data_ptr() for t in cp] or (None,) * 6),
                            block_idx.data_ptr(), None, d_out.data_ptr(), *[t.data_ptr() for t in grads],
                            *[t.data_ptr() for t in d_cp])
        L.check(L.lib().nsa_attention_bwd(desc, ptrs, saved.data_ptr(), ws.data_ptr(), bwd_bytes, L.raw_stream(dev)))
        if L.CHECK_STATUS_EVERY_CALL:
            L.check_device_status()
        if gate_dtype != d_out.dtype:
            grads[7] = grads[7].to(gate_dtype)
        d_cp = [g if g.dtype == t else g.to(t) for g, t in zip(d_cp, comp_dtypes)]
        if torch.is_grad_enabled():
            grads, d_cp = ([_Once.apply(g.requires_grad_(True)) for g in gs] for gs in (grads, d_cp))
        return (*grads, None, None, None, None, None, *d_cp)


def _op_in_parts(q, kv, gate_logits, block_idx, block_size, n_sel, window, forced, comp):
    """The op out of the calls of its parts, for K / V tensors that do not share one shape: a pooled or windowed
    pair of another length, branches with other numbers of kv heads."""
    kc, vc, ks, vs, kw, vw = kv
    n_init, n_local, cl, cs = forced
    if comp is None:
        assert cl == cs == block_size, "mean pooling is defined on the aligned grid only"
        k_cmp, v_cmp = block_mean_pool(kc, block_size), block_mean_pool(vc, block_size)
    else:
        k_cmp, v_cmp = (block_compress(x, *comp[3 * i:3 * i + 3], cl, cs) for i, x in enumerate((kc, vc)))
    o_cmp = compression_attn_triton(q, k_cmp, v_cmp, cl, cs)
    if block_idx is None:
        with torch.no_grad():
            _, lse = range_attn_forward(q, k_cmp, v_cmp, MODE_COMPRESS_STRIDED, cs, cl)
        block_idx = topn_blocks(q, k_cmp, lse, block_size, n_sel, n_init_blocks=n_init, n_local_blocks=n_local,
                                cmp_len=cl, cmp_stride=cs)
    else:
        block_idx = block_idx.to(torch.int32).contiguous()
    assert ks.shape[2] == q.shape[2], "selection keys and queries are the same tokens"
    o_slc = selection_attn_triton(q, ks, vs, block_idx, block_size)
    return gate_combine(o_cmp, o_slc, window_attn_triton(q, kw, vw, window), gate_logits), block_idx


def _dual_level():
    return getattr(forward_ad, "_current_level", 0) >= 0


def one_node_ok():
    """Whether the nodes in C++ may serve a call: where they are built, outside of forward-mode levels and traces, and
    without a look at the device status after every call."""
    return (not _dual_level() and not L.CHECK_STATUS_EVERY_CALL and torch._C._get_tracing_state() is None
            and L.torch_op() is not None)


def switches():
    """The process-wide choices a call goes by: dQ accumulator, kernel family."""
    return int(_dq_accumulator), L.IMPL[_impl]


def _op(q, kv, gate_logits, block_idx, block_size, n_sel, window, forced, comp):
    """The whole op.  The usual form of a call goes to the node in C++ (csrc/torch_op.cpp, which says what that form is);
    every other one through the Python node where a gradient is asked for, and inside a forward-mode level,
    where the node refuses a tangent that the bare call would drop."""
    kc, vc, ks, vs, kw, vw = kv
    if one_node_ok():
        res = L.torch_op().op(q, kc, vc, ks, vs, kw, vw, gate_logits, block_idx, comp, block_size, n_sel, window, *forced,
                              *switches())
        if res is not None:
            return res
    if not (kc.shape == vc.shape == ks.shape == vs.shape == kw.shape == vw.shape and kc.shape[2] == q.shape[2]):
        return _op_in_parts(q, kv, gate_logits, block_idx, block_size, n_sel, window, forced, comp)
    if (torch.is_grad_enabled() and any(t.requires_grad for t in (q, *kv, gate_logits, *(comp or ())))) or _dual_level():
        return _NSAAttention.apply(q, *kv, gate_logits, block_size, n_sel, window, block_idx, forced, *(comp or ()))
    return _op_forward(q, kv, gate_logits, block_idx, block_size, n_sel, window, forced, comp, False)[:2]


@torch.no_grad()
def select_blocks(q, kc, vc, block_size, n_sel, compressor=None, n_init_blocks=0, n_local_blocks=0,
                  cmp_len=None, cmp_stride=None):
    """The block lists [B,Hkv,T,n_sel] the whole op picks for q (pooling, compression attention,
    block scoring + top-n; nsa_model.py:336-355), without the rest of the op.  The scores sum over
    all query heads of a kv head, so a caller that deals the query heads of one group out over
    several devices computes the lists from the whole group on each and passes them to
    nsa_attention(..., block_idx=...) with its share of the heads."""
    cl = int(block_size if cmp_len is None else cmp_len)
    cs = int(cl if cmp_stride is None else cmp_stride)
    if compressor is not None:
        cp = [compressor[n].detach().float().contiguous()
              for n in ("k_intra", "k_logits", "k_proj", "v_intra", "v_logits", "v_proj")]
        k_cmp = _compress_fwd(kc, cp[0], cp[1], cp[2], cl, cs)
        v_cmp = _compress_fwd(vc, cp[3], cp[4], cp[5], cl, cs)
    else:
        assert cl == cs == block_size, "mean pooling is defined on the aligned grid only"
        k_cmp, v_cmp = _mean_pool_fwd(kc, block_size), _mean_pool_fwd(vc, block_size)
    _, lse_cmp = range_attn_forward(q, k_cmp, v_cmp, MODE_COMPRESS_STRIDED, cs, cl)
    return topn_blocks(q, k_cmp, lse_cmp, block_size, n_sel, n_init_blocks=n_init_blocks,
                       n_local_blocks=n_local_blocks, cmp_len=cl, cmp_stride=cs)


def nsa_attention(q, kc, vc, ks, vs, kw, vw, gate_logits, block_size, n_sel, window,
                  block_idx=None, compressor=None, return_block_idx=False, n_init_blocks=0,
                  n_local_blocks=0, cmp_len=None, cmp_stride=None):
    """Full NSA attention (pre out_proj) as one differentiable op.

    q [B,Hq,T,D]; kc..vw [B,Hkv,T,D]; gate_logits [B,Hq,T,3].  `compressor` is None for mean
    pooling or a dict k_intra,k_logits,k_proj,v_intra,v_logits,v_proj holding the parameters
    of the two BlockCompressor modules (nsa_model.py:180-181).  With block_idx=None the blocks
    are picked by the scorer (nsa_model.py:343-355 semantics, deterministic tie order);
    n_init_blocks / n_local_blocks force the first blocks and the most recent blocks into every
    list ahead of the scored ones (the published NSA recipe; the reference has no such option).
    cmp_len / cmp_stride (learned pooling only; default block_size, the reference's grid) make
    the summaries windows of cmp_len tokens every cmp_stride tokens, e.g. 32 / 16 with 64-token
    selection blocks; the compressor parameters then have cmp_len positions.
    With NSA_B200_CHECK_STATUS=1 in the environment the device status word is read (one stream
    synchronisation) after every forward and backward and a give-up raises NsaError."""
    cp = None
    if compressor is not None:
        cp = tuple(compressor[n] for n in ("k_intra", "k_logits", "k_proj", "v_intra", "v_logits", "v_proj"))
    cl = int(block_size if cmp_len is None else cmp_len)
    cs = int(cl if cmp_stride is None else cmp_stride)
    out, idx = _op(q, (kc, vc, ks, vs, kw, vw), gate_logits, block_idx, block_size, n_sel, window,
                   (int(n_init_blocks), int(n_local_blocks), cl, cs), cp)
    return (out, idx) if return_block_idx else out
