"""The whole-op call and its side streams: captures, callers' streams, threads."""
import ctypes
import importlib
import threading

import pytest
import torch

from tests.test_refused_calls import _inputs
from tests.util import pkg

pytestmark = pytest.mark.gpu


def _forward_call(ins, S=4, W=128, bs=64):
    """A forward through the C ABI on memory of its own: (launch(stream) -> return code, output)."""
    L = importlib.import_module("openbox-llm_b200._lib")
    q, k = ins[0], ins[1]
    B, Hq, T, D = q.shape
    desc = L.NsaAttentionDesc(L.dims(B, Hq, k.shape[1], T, D, L.DTYPE_BF16), bs, S, W, 0, 0, bs, bs, 0, 0, 0, 0, 0)
    n = [ctypes.c_size_t() for _ in range(3)]
    L.check(L.lib().nsa_attention_sizes(desc, *n))
    saved, ws = (torch.empty(x.value + 1, dtype=torch.uint8, device="cuda") for x in n[:2])
    idx = torch.empty(B, k.shape[1], T, S, dtype=torch.int32, device="cuda")
    out = torch.zeros_like(q)
    ptrs = L.OP_TENSORS(*[x.data_ptr() for x in ins], *(None,) * 6, idx.data_ptr(), out.data_ptr())
    keep = (saved, ws, idx)

    def launch(stream):
        return L.lib().nsa_attention_fwd(desc, ptrs, keep[0].data_ptr(), keep[1].data_ptr(), n[1], stream)

    return launch, out


def test_two_captures_open_in_one_thread():
    """A thread's side streams belong to one capture at a time: a call in another capture goes without them.  The
    thread is new, so its side streams are also made inside the first capture."""
    nsa = pkg()
    rt = ctypes.CDLL("libcudart.so.12")
    ins = [_inputs(1, 8, 2, 512, 64, seed=s) for s in (1, 2)]
    want = [nsa.nsa_attention(*x, 64, 4, 128) for x in ins]
    calls = [_forward_call(x) for x in ins]
    streams = [torch.cuda.Stream() for _ in ins]
    torch.cuda.synchronize()
    codes, graphs = [], [ctypes.c_void_p() for _ in ins]
    execs = [ctypes.c_void_p() for _ in ins]

    def body():
        torch.cuda.set_device(0)
        for s, (launch, _) in zip(streams, calls):
            codes.append(rt.cudaStreamBeginCapture(ctypes.c_void_p(s.cuda_stream), 1))   # thread-local mode
            codes.append(launch(s.cuda_stream))
        for s, g in zip(streams, graphs):
            codes.append(rt.cudaStreamEndCapture(ctypes.c_void_p(s.cuda_stream), ctypes.byref(g)))
        for g, e in zip(graphs, execs):
            codes.append(rt.cudaGraphInstantiateWithFlags(ctypes.byref(e), g, ctypes.c_ulonglong(0)))
        for s, e in zip(streams, execs):
            codes.append(rt.cudaGraphLaunch(e, ctypes.c_void_p(s.cuda_stream)))

    t = threading.Thread(target=body)
    t.start()
    t.join()
    assert codes == [0] * 10, codes
    torch.cuda.synchronize()
    for (_, out), w, g, e in zip(calls, want, graphs, execs):
        assert torch.equal(out, w)
        rt.cudaGraphExecDestroy(e)
        rt.cudaGraphDestroy(g)
    assert nsa.lib().nsa_device_status(None) == 0


def _train(ins, do, **kw):
    nsa = pkg()
    xs = [x.detach().requires_grad_(True) for x in ins]
    out = nsa.nsa_attention(*xs, 64, 4, 128, **kw)
    return [out.detach(), *torch.autograd.grad(out, xs, do)]


def _same(got, want):
    """out, dq and d_gate are the same bits; the rest may meet in another order: one bf16 step of the largest."""
    for i, (a, b) in enumerate(zip(got, want)):
        if i in (0, 1, 8):
            assert torch.equal(a, b), i
        else:
            assert (a.float() - b.float()).abs().max() <= 2.0 ** -7 * b.float().abs().max(), i


def test_op_on_callers_streams_with_memory_going_round():
    """Calls on a stream of the caller's, each on inputs made on that stream just before and given back right after:
    what the side streams read and write is the call's own memory, whatever is allocated next."""
    want = []
    for seed in range(6):
        ins = _inputs(1, 8, 2, 448, 64, seed=seed)
        want.append(_train(ins, torch.ones_like(ins[0])))
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    for seed in [0, 1, 2, 3, 4, 5] * 4:
        with torch.cuda.stream(stream):
            ins = _inputs(1, 8, 2, 448, 64, seed=seed)
            got = _train(ins, torch.ones_like(ins[0]))
            del ins
            torch.full((1 << 22,), float("nan"), device="cuda")     # takes over freed memory on this stream
        stream.synchronize()
        _same(got, want[seed])
    assert pkg().lib().nsa_device_status(None) == 0


def test_op_from_two_threads():
    """Every thread has side streams of its own; two threads on two streams get what one gets alone."""
    ins = [_inputs(1, 8, 2, 512, 64, seed=s) for s in (1, 2)]
    want = [_train(x, torch.ones_like(x[0])) for x in ins]
    torch.cuda.synchronize()
    got, errors = [[], []], []

    def body(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    got[k].append(_train(ins[k], torch.ones_like(ins[k][0])))
                torch.cuda.current_stream().synchronize()
        except Exception as e:      # noqa: BLE001 (reported by the assertion below)
            errors.append(e)

    threads = [threading.Thread(target=body, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k in range(2):
        for g in got[k]:
            _same(g, want[k])
    assert pkg().lib().nsa_device_status(None) == 0


@pytest.mark.parametrize("over", [0, 1])
def test_op_on_both_sides_of_the_overlap_line(over):
    """The branches run on side streams up to 8 row tiles of 128 rows per SM: the forward is bit for bit what the
    entry points of the parts give, at the last size that overlaps and at the next one."""
    nsa = pkg()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    T = 64 * sms + 64 * over                # 16 heads: T / 8 row tiles
    ins = _inputs(1, 16, 1, T, 64)
    q, kc, vc, ks, vs, kw, vw, gate = ins
    with torch.no_grad():
        out, idx = nsa.nsa_attention(*ins, 64, 4, 128, return_block_idx=True)
        k_cmp, v_cmp = nsa.block_mean_pool(kc, 64), nsa.block_mean_pool(vc, 64)
        o_cmp, lse = nsa.range_attn_forward(q, k_cmp, v_cmp, nsa.MODE_COMPRESS, 0, 64)
        assert torch.equal(idx, nsa.topn_blocks(q, k_cmp, lse, 64, 4))
        parts = nsa.gate_combine(o_cmp, nsa.selection_attn_triton(q, ks, vs, idx, 64), nsa.window_attn_triton(q, kw, vw, 128), gate)
    assert torch.equal(out, parts)
    got = _train(ins, torch.ones_like(q))
    assert torch.equal(got[0], out)
    # gradients against the parts through autograd: three roundings of dq instead of one
    xs = [x.detach().requires_grad_(True) for x in ins]
    q, kc, vc, ks, vs, kw, vw, gate = xs
    out = nsa.gate_combine(nsa.compression_attn_triton(q, nsa.block_mean_pool(kc, 64), nsa.block_mean_pool(vc, 64), 64),
                           nsa.selection_attn_triton(q, ks, vs, idx, 64), nsa.window_attn_triton(q, kw, vw, 128), gate)
    for a, b in zip(got[1:], torch.autograd.grad(out, xs, torch.ones_like(q))):
        assert (a.float() - b.float()).norm() <= 2.0 ** -6 * b.float().norm()
    assert nsa.lib().nsa_device_status(None) == 0


def test_dq_of_three_deferred_branches():
    """Backward calls with dq = NULL and one nsa_dq_reduce3 over their workspaces: the sum of the three branches'
    own dq, each of which is rounded to bf16 by itself (half a step each)."""
    nsa = pkg()
    L = importlib.import_module("openbox-llm_b200._lib")
    for B, Hq, Hkv, T, D, bs, S, W in ((1, 8, 2, 700, 64, 64, 4, 130), (2, 16, 2, 512, 128, 64, 3, 200)):
        q, kc, vc, ks, vs, kw, vw, _ = _inputs(B, Hq, Hkv, T, D)
        do = torch.randn_like(q)
        n_cmp = T // bs
        kc, vc = kc[:, :, :n_cmp].contiguous(), vc[:, :, :n_cmp].contiguous()
        o, lse = nsa.range_attn_forward(q, kc, vc, nsa.MODE_COMPRESS, 0, bs)
        idx = nsa.topn_blocks(q, kc, lse, bs, S)
        cmp = [nsa.range_attn_backward(q, kc, vc, o, lse, do, nsa.MODE_COMPRESS, 0, bs, defer_dq=d) for d in (False, True)]
        o, lse = nsa.selection_forward_triton(q, ks, vs, idx, bs, return_lse=True)
        slc = [nsa.ops._selection_backward(q, ks, vs, idx, bs, do, o, lse, defer_dq=d, plan=p)
               for d, p in ((False, None), (True, None), (True, nsa.ops.selection_plan(q, ks, idx, bs)))]
        o, lse = nsa.range_attn_forward(q, kw, vw, nsa.MODE_WINDOW, W, 0)
        win = [nsa.range_attn_backward(q, kw, vw, o, lse, do, nsa.MODE_WINDOW, W, 0, defer_dq=d) for d in (False, True)]
        parts = [x[0][0].float() for x in (cmp, slc, win)]
        bound = 2.0 ** -9 * sum(x.abs() for x in parts) * 2 + 2.0 ** -8 * sum(parts).abs() + 1e-6
        for ws in slc[1:]:
            dq = torch.empty_like(q)
            L.check(L.lib().nsa_dq_reduce3(L.dims(B, Hq, Hkv, T, D, L.DTYPE_BF16), n_cmp, bs, bs, S, bs, W, L.ptr(cmp[1][0]),
                                           L.ptr(ws[0]), L.ptr(win[1][0]), L.ptr(dq), L.stream()))
            assert ((dq.float() - sum(parts)).abs() <= bound).all()
    assert nsa.lib().nsa_device_status(None) == 0
