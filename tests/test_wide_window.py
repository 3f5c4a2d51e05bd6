"""Window backward on tiles of 128 keys (csrc/tc_bwd_wide.cu) against 64-bit arithmetic, at the edges of its key tiles,
row tiles and windows.

The kernel serves windows with more tiles of 64 keys than the GPU has SMs, so the sequences here are short and many.
What is rounded to bf16 (relative 2^-9 at most) on the way to a gradient: P, O in delta, dS, the partial rows of dQ, the gradient itself,
four of them for each of dq, dk and dv at most, independent of one another: relative L2 of 2 x 2^-9.  Measured: 1.7e-3 to 2.9e-3."""
import importlib

import pytest
import torch

nsa = importlib.import_module("openbox-llm_b200")
TOL = 2 * 2.0 ** -9
pytestmark = pytest.mark.gpu


def reference(q, k, v, do, window, gate=None):
    """dq, dk, dv in 64 bits, of do * gate where a gate (per row) is given."""
    q, k, v, do = (x.detach().double() for x in (q, k, v, do))
    B, Hq, T, D = q.shape
    G = Hq // k.shape[1]
    for x in (q, k, v):
        x.requires_grad_(True)
    kk, vv = k.repeat_interleave(G, 1), v.repeat_interleave(G, 1)
    t = torch.arange(T, device=q.device)
    seen = (t[None, :] <= t[:, None]) & (t[None, :] > t[:, None] - window)
    s = (q @ kk.transpose(-1, -2) * D ** -0.5).masked_fill(~seen, float("-inf"))
    o = s.softmax(-1) @ vv
    return torch.autograd.grad(o, (q, k, v), do if gate is None else do * gate[..., None])


def rel(x, y):
    return ((x.double() - y).norm() / y.norm()).item()


CASES = [  # B, Hq, Hkv, T, D, window
    (40, 8, 4, 65, 64, 512), (40, 12, 4, 127, 64, 64), (40, 12, 4, 128, 64, 1), (40, 16, 4, 129, 64, 127), (40, 16, 2, 130, 128, 128),
    (24, 6, 2, 300, 64, 129), (24, 32, 2, 257, 128, 200), (24, 8, 4, 383, 128, 512), (24, 12, 4, 385, 128, 2 ** 31 - 1),
    (40, 256, 2, 129, 64, 100), (3, 12, 4, 3001, 64, 512),
]


@pytest.mark.parametrize("B,Hq,Hkv,T,D,window", CASES)
def test_against_64_bits(B, Hq, Hkv, T, D, window):
    assert B * Hkv * ((T + 63) // 64) > 148
    g = torch.Generator("cuda").manual_seed(T + Hq)
    q, do = (torch.randn(B, Hq, T, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Hkv, T, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    leaves = [x.clone().requires_grad_(True) for x in (q, k, v)]
    o = nsa.window_attn_triton(*leaves, min(window, 2 ** 31 - 1))
    got = torch.autograd.grad(o, leaves, do)
    sums = [torch.zeros(2, dtype=torch.float64, device="cuda") for _ in range(3)]
    step = max(1, 2 ** 26 // (Hq * T * T))
    for b in range(0, B, step):
        part = slice(b, b + step)
        for s, x, y in zip(sums, got, reference(q[part], k[part], v[part], do[part], window)):
            d = x[part].double() - y
            s += torch.stack([(d * d).sum(), (y * y).sum()])
    for name, s in zip(("dq", "dk", "dv"), sums):
        e = (s[0] / s[1]).sqrt().item()
        assert e <= TOL or (window == 1 and name != "dv"), (name, e)
    if window == 1:
        # p = 1 and O = V: dP = delta, two fp32 sums of the same D products, each off by D 2^-23 of their absolute sum at most,
        # in any order.  That is all there is in dS, and dq and dk are dS times a row of k and G rows of q.
        G = Hq // Hkv
        ds = 2 * D * 2.0 ** -23 * D ** -0.5 * (do.float() * v.float().repeat_interleave(G, 1)).abs().sum(-1).max().item() * 1.01
        assert got[0].abs().max().item() <= ds * k.abs().max().item() and got[1].abs().max().item() <= G * ds * q.abs().max().item()
    assert all(torch.isfinite(x.float()).all() for x in got)


def test_gates_that_underflow():
    """Rows whose gate is 0 in fp32 leave nothing behind, in dK and dV of their keys neither."""
    B, Hq, Hkv, T, D = 40, 16, 4, 200, 64
    g = torch.Generator("cuda").manual_seed(5)
    q, do = (torch.randn(B, Hq, T, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    kv = [torch.randn(B, Hkv, T, D, generator=g, device="cuda").bfloat16() for _ in range(6)]
    logits = torch.randn(B, Hq, T, 3, generator=g, device="cuda").bfloat16()
    logits[:, :, ::3, 2] = -300.0
    idx = torch.full((B, Hkv, T, 16), -1, dtype=torch.int32, device="cuda")
    idx[:, :, 63:, 0] = 0
    leaves = [x.clone().requires_grad_(True) for x in (q, *kv, logits)]
    out = nsa.nsa_fused_forward(*leaves, idx, 64, 128)
    got = torch.autograd.grad(out, leaves, do)
    assert all(torch.isfinite(x.float()).all() for x in got)
    gate = torch.sigmoid(logits[..., 2].double())
    _, dk, dv = reference(q[:4], kv[4][:4], kv[5][:4], do[:4], 128, gate[:4])
    assert rel(got[5][:4], dk) <= TOL and rel(got[6][:4], dv) <= TOL
    # dq of these rows is that of the other two branches: bit for bit the same beside other keys in the window
    others = leaves[:5] + [torch.flip(x.detach(), [2]).requires_grad_(True) for x in leaves[5:7]] + leaves[7:]
    dq = torch.autograd.grad(nsa.nsa_fused_forward(*others, idx, 64, 128), others[0], do)[0]
    assert torch.equal(dq[:, :, ::3], got[0][:, :, ::3]) and not torch.equal(dq[:, :, 1::3], got[0][:, :, 1::3])


def test_gradients_that_start_anywhere():
    """dk and dv of the C entry point need no alignment, and nothing is written around them."""
    ops, L = nsa.ops, importlib.import_module("openbox-llm_b200._lib")
    B, Hq, Hkv, T, D, window = 20, 8, 4, 200, 64, 77
    g = torch.Generator("cuda").manual_seed(3)
    q, do, k, v = (torch.randn(B, h, T, D, generator=g, device="cuda").bfloat16() for h in (Hq, Hq, Hkv, Hkv))
    o, lse = ops.range_attn_forward(q, k, v, L.MODE_WINDOW, window, 0)
    dims = L.dims(B, Hq, Hkv, T, D, L.DTYPE_BF16)
    n = L.lib().nsa_range_attn_bwd_workspace_bytes(dims, T, L.MODE_WINDOW, window, 0)
    want = None
    for off in (8, 1, 4):
        ws = torch.empty(n, dtype=torch.uint8, device="cuda")
        dq = torch.empty_like(q)
        bufs = [torch.full((k.numel() + 16,), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
        dk, dv = (b[off:off + k.numel()] for b in bufs)
        L.check(L.lib().nsa_range_attn_bwd(L.ptr(q), L.ptr(k), L.ptr(v), L.ptr(o), L.ptr(lse), L.ptr(do), L.ptr(dq), L.ptr(dk),
                                           L.ptr(dv), dims, T, L.MODE_WINDOW, window, 0, None, None, L.ptr(ws), n, 0, L.stream()))
        assert all((b[:off] == 7.0).all() and (b[off + k.numel():] == 7.0).all() for b in bufs)
        got = [dq, dk.clone(), dv.clone()]
        want = want or got
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert L.lib().nsa_device_status(None) == 0


@pytest.mark.parametrize("B,Hq,Hkv,T,Lk,D,window", [(40, 8, 4, 130, 200, 64, 100), (24, 12, 4, 385, 385, 128, 200), (40, 8, 4, 130, 129, 64, 2 ** 31 - 1)])
def test_partials_for_a_sum_by_hand(B, Hq, Hkv, T, Lk, D, window):
    """Partials that a caller has added up by nsa_dq_reduce3 lie where that looks for them, whatever the number of keys and
    the options at that time.  Bound: two bf16 partials' roundings apart."""
    L = importlib.import_module("openbox-llm_b200._lib")
    g = torch.Generator("cuda").manual_seed(T + Lk)
    q, do = (torch.randn(B, Hq, T, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Hkv, Lk, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    o, lse = nsa.range_attn_forward(q, k, v, nsa.MODE_WINDOW, window, 0)
    want = nsa.range_attn_backward(q, k, v, o, lse, do, nsa.MODE_WINDOW, window, 0)
    ws, dk, dv = nsa.range_attn_backward(q, k, v, o, lse, do, nsa.MODE_WINDOW, window, 0, defer_dq=True)
    dq = torch.empty_like(q)
    try:
        L.check(L.lib().nsa_set_option(b"bwd_kernel", 0))
        L.check(L.lib().nsa_dq_reduce3(L.dims(B, Hq, Hkv, T, D, L.DTYPE_BF16), 0, 0, 0, 0, 64, window, None, None, ws.data_ptr(), dq.data_ptr(),
                                       L.stream()))
    finally:
        L.check(L.lib().nsa_set_option(b"bwd_kernel", 1))
    for x, y in zip((dq, dk, dv), want):
        assert rel(x, y.double()) < 2.0 ** -7
