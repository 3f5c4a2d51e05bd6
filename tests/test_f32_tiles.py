"""fp32 attention at D = 64 on the tensor cores: every product as six products of bf16 terms."""
import pytest
import torch

from tests.util import pkg

pytestmark = pytest.mark.gpu


def _dense(q, k, v, do, keep):
    """o, dq, dk, dv in 64 bits; keep [B, Hkv, T, L] counts how often a row attends a key."""
    B, Hq, T, D = q.shape
    G = Hq // k.shape[1]
    q, k, v, do = (x.double() for x in (q, k, v, do))
    kk, vv, n = (x.repeat_interleave(G, 1) for x in (k, v, keep.double()))
    s = (q @ kk.transpose(-1, -2) * D ** -0.5).masked_fill(n == 0, float("-inf"))
    p = (s - s.amax(-1, keepdim=True).nan_to_num(0, 0, 0)).exp() * n
    p = p / p.sum(-1, keepdim=True).clamp_min(1e-300)
    o = p @ vv
    ds = p * (do @ vv.transpose(-1, -2) - (do * o).sum(-1, keepdim=True)) * D ** -0.5
    fold = lambda x: x.view(B, -1, G, *x.shape[2:]).sum(2)
    return o, ds @ kk, fold(ds.transpose(-1, -2) @ q), fold(p.transpose(-1, -2) @ do)


def _lists(B, Hkv, T, bs, S, repeat, g):
    """Block lists and how often each row attends each token."""
    n_blk = (T + bs - 1) // bs
    t = torch.arange(T, device="cuda")
    idx = torch.randint(0, n_blk, (B, Hkv, T, S), generator=g, device="cuda")
    idx = torch.where(idx * bs <= t[:, None], idx, torch.full_like(idx, -1))
    if not repeat:
        first = (idx[..., :, None] == idx[..., None, :]).int().argmax(-1) == torch.arange(S, device="cuda")
        idx = torch.where(first, idx, torch.full_like(idx, -1))
    n = torch.zeros(B, Hkv, T, n_blk + 1, device="cuda")
    n.scatter_add_(3, torch.where(idx < 0, n_blk, idx), torch.ones_like(idx, dtype=torch.float32))
    keep = n[..., :n_blk].repeat_interleave(bs, 3)[..., :T] * (t[:, None] >= t)
    return idx.int().contiguous(), keep


def _run(nsa, kind, q, k, v, do, idx, bs, W):
    if kind == "selection":
        o, lse = nsa.selection_forward_triton(q, k, v, idx, bs, return_lse=True)
        return o, *nsa.ops._selection_backward(q, k, v, idx, bs, do, o, lse)
    mode, w = (nsa.MODE_WINDOW, W) if kind == "window" else (nsa.MODE_COMPRESS, 0)
    o, lse = nsa.range_attn_forward(q, k, v, mode, w, bs)
    return o, *nsa.range_attn_backward(q, k, v, o, lse, do, mode, w, bs)


# the last row tile with 1, 63 and all of its rows, key tiles of 1, 64 and 65 keys, one to eight heads on a kv head; clusters of four, two
# and one (row tiles per SM: below 0.5, between, above 3); blocks that end within a key tile, and longer ones than it
@pytest.mark.parametrize("B,Hq,Hkv,T,W,bs,S,repeat", [
    (1, 8, 2, 481, 2, 64, 8, False), (2, 3, 3, 575, 64, 16, 24, True), (1, 12, 4, 704, 65, 24, 20, True), (2, 8, 1, 1000, 133, 64, 16, False),
    (1, 4, 4, 4097, 512, 64, 16, False), (6, 16, 2, 640, 200, 32, 12, True), (2, 16, 1, 300, 70, 17, 9, True), (1, 8, 2, 705, 63, 40, 9, False),
    (3, 6, 2, 901, 30, 100, 5, True)])
def test_f32_tiles_are_fp32_arithmetic(B, Hq, Hkv, T, W, bs, S, repeat):
    """Against 64 bits, whole tensors.  A dot product of 64 terms is good to 2^-23 of its norm, and o and the gradients are chains of two to
    five such steps and of sums of up to 40 tiles, each rounded to 2^-24: 2^-20 of a tensor's norm (measured: up to 3.4e-7; 4.8e-7 with
    chains of FFMAs)."""
    nsa = pkg()
    g = torch.Generator(device="cuda").manual_seed(1)
    q, do = (torch.randn(B, Hq, T, 64, generator=g, device="cuda") for _ in range(2))
    k, v = (torch.randn(B, Hkv, T, 64, generator=g, device="cuda") for _ in range(2))
    do *= 2.0 ** -20                                       # (small gradients keep their bits)
    t = torch.arange(T, device="cuda")
    idx, keep = _lists(B, Hkv, T, bs, S, repeat, g)
    cases = {"selection": (k, v, keep), "window": (k, v, ((t[:, None] >= t) & (t[:, None] - t < W)).expand(B, Hkv, T, T)),
             "compression": (k[:, :, :T // bs].contiguous(), v[:, :, :T // bs].contiguous(),
                             ((t[:, None] + 1) // bs > torch.arange(T // bs, device="cuda")).expand(B, Hkv, T, T // bs))}
    for kind, (kk, vv, n) in cases.items():
        got = _run(nsa, kind, q, kk, vv, do, idx, bs, W)
        for name, x, y in zip(("o", "dq", "dk", "dv"), got, _dense(q, kk, vv, do, n)):
            assert (x.double() - y).norm() <= 2.0 ** -20 * y.norm(), (kind, name, ((x.double() - y).norm() / y.norm()).item())


def test_f32_values_that_cannot_be_split():
    """Values from 2^60 on (products of whose terms could overflow), infinities and NaN go by FFMA: a huge value gives what it
    gives in fp32, and what is not finite stays with the rows and keys that it belongs to."""
    nsa = pkg()
    T, W = 700, 100
    g = torch.Generator(device="cuda").manual_seed(2)
    q, do = (torch.randn(1, 8, T, 64, generator=g, device="cuda") for _ in range(2))
    k, v = (torch.randn(1, 2, T, 64, generator=g, device="cuda") for _ in range(2))
    clean = _run(nsa, "window", q, k, v, do, None, 0, W)
    t = torch.arange(T, device="cuda")
    attends = (t[:, None] >= t) & (t[:, None] - t < W)
    for at, where, bad in ((300, "v", float("inf")), (300, "k", float("nan")), (64, "q", float("nan")), (500, "do", float("inf"))):
        x = {"q": q, "k": k, "v": v, "do": do}
        x[where] = x[where].clone()
        x[where][:, :, at, 3] = bad
        got = _run(nsa, "window", x["q"], x["k"], x["v"], x["do"], None, 0, W)
        rows = ~attends[:, at] if where in "kv" else t != at
        keys = ~(attends & ~rows[:, None]).any(0)
        for i, keep in enumerate((rows, rows, keys, keys)):
            a, b = got[i][:, :, keep], clean[i][:, :, keep]
            assert torch.isfinite(a).all() and (a - b).norm() <= 2.0 ** -20 * b.norm(), (where, i)
        assert not torch.isfinite(got[1 if where != "v" else 0]).all()
    # v = 2^100 in one column: o of the rows that attend it is 2^100 times their probability, and dv is as without it
    big = v.clone()
    big[:, :, 300, 5] = 2.0 ** 100
    o, dq, dk, dv = _run(nsa, "window", q, k, big, do * 2.0 ** -100, None, 0, W)
    ref = _dense(q, k, big, do * 2.0 ** -100, attends.expand(1, 2, T, T))
    for x, y in zip((o, dq, dk, dv), ref):
        assert (x.double() - y).norm() <= 2.0 ** -20 * y.norm()
    assert nsa.lib().nsa_device_status(None) == 0


def _attended(kind, B, Hkv, T, bs, S, W, repeat, g):
    """How often each row attends each key, what _run takes for it, and the number of keys."""
    t = torch.arange(T, device="cuda")
    if kind == "selection":
        idx, keep = _lists(B, Hkv, T, bs, S, repeat, g)
        return keep, idx, T
    if kind == "window":
        return ((t[:, None] >= t) & (t[:, None] - t < W)).float().expand(B, Hkv, T, T), None, T
    n = (T - bs) // W + 1                                  # summaries of bs tokens every W
    return ((t[:, None] - bs + 1) // W >= torch.arange(n, device="cuda")).float().expand(B, Hkv, T, n), None, n


# row tiles that clusters of four (up to half a row tile per SM; selection 0.87), of two (1.3; 3) and none share; lists that repeat blocks; blocks
# of 24, 40 and 48 tokens; summaries of 16 tokens every W
@pytest.mark.parametrize("kind,B,Hq,Hkv,T,bs,S,W,repeat", [
    ("selection", 1, 8, 2, 700, 64, 6, 0, False), ("selection", 1, 4, 2, 1300, 24, 14, 0, True), ("selection", 3, 8, 2, 800, 48, 5, 0, True),
    ("selection", 6, 8, 2, 700, 40, 5, 0, True), ("compression", 1, 4, 1, 500, 16, 0, 1, False), ("compression", 1, 8, 2, 900, 16, 0, 2, False),
    ("compression", 2, 8, 2, 1000, 16, 0, 16, False), ("window", 1, 8, 2, 500, 0, 0, 480, False), ("window", 1, 8, 2, 700, 0, 0, 300, False),
    ("window", 3, 8, 2, 700, 0, 0, 300, False)])
def test_f32_values_that_cannot_be_split_in_every_branch(kind, B, Hq, Hkv, T, bs, S, W, repeat):
    """The repairs by FFMA where a key tile is a union of listed blocks, counts blocks twice, or is shared out over a cluster: what is not
    finite stays with the rows that attend it and their keys, huge values are exact to the same 2^-20."""
    nsa = pkg()
    g = torch.Generator(device="cuda").manual_seed(5)
    n, idx, L = _attended(kind, B, Hkv, T, bs, S, W, repeat, g)
    q, do = (torch.randn(B, Hq, T, 64, generator=g, device="cuda") for _ in range(2))
    k, v = (torch.randn(B, Hkv, L, 64, generator=g, device="cuda") for _ in range(2))

    def run(q, k, v, do):
        if kind != "compression":
            return _run(nsa, kind, q, k, v, do, idx, bs, W)
        o, lse = nsa.range_attn_forward(q, k, v, nsa.MODE_COMPRESS_STRIDED, W, bs)
        return o, *nsa.range_attn_backward(q, k, v, o, lse, do, nsa.MODE_COMPRESS_STRIDED, W, bs)

    clean = run(q, k, v, do)
    for name, a, b in zip(("o", "dq", "dk", "dv"), clean, _dense(q, k, v, do, n)):
        assert (a.double() - b).norm() <= 2.0 ** -20 * b.norm(), name
    hit = lambda where, at: (n[..., at] > 0) if where in "kv" else (torch.arange(T, device="cuda") == at).expand(B, Hkv, T)
    same = lambda a, b: torch.isfinite(a).all() and (a - b).norm() <= 2.0 ** -20 * b.norm()

    def stays(got, where, at):
        rows = hit(where, at)
        keys = ((n > 0) & rows[..., None]).any(2)
        far = (~rows).repeat_interleave(Hq // Hkv, 1), ~keys
        for i, (x, y) in enumerate(zip(got, clean)):
            assert same(x[far[i > 1]], y[far[i > 1]]), (where, at, i)

    for at, where, bad in ((L // 3, "v", float("inf")), (L // 2, "k", float("nan")), (T - 70, "q", float("nan")), (T // 2 + 1, "do", float("-inf"))):
        x = {"q": q, "k": k, "v": v, "do": do}
        x[where] = x[where].clone()
        x[where][:, :, at, 3] = bad
        got = run(**x)
        stays(got, where, at)
        assert hit(where, at).any() and not torch.isfinite(got[0 if where == "v" else 1]).all(), where
    for at, where, scale in ((L // 3, "v", 2.0 ** -100), (T // 2 + 1, "do", 1.0)):
        x = {"q": q, "k": k, "v": v, "do": do * scale}
        x[where] = x[where].clone()
        x[where][:, :, at, 5] = 2.0 ** 100
        got = run(**x)
        for name, a, b in zip(("o", "dq", "dk", "dv"), got, _dense(*x.values(), n)):
            assert (a.double() - b).norm() <= 2.0 ** -20 * b.norm(), (where, name)
        if where == "do":
            stays(got, where, at)
    assert nsa.lib().nsa_device_status(None) == 0


def test_simt_is_the_cuda_cores():
    """Who asks for the CUDA cores gets FFMA tiles; by default fp32 heads of 64 go by bf16 terms.  Both to 2^-20 of the norm, as above."""
    nsa = pkg()
    L, lib = nsa._lib, nsa.lib()
    g = torch.Generator(device="cuda").manual_seed(3)
    T, bs = 700, 64
    q, do = (torch.randn(1, 8, T, 64, generator=g, device="cuda") for _ in range(2))
    k, v = (torch.randn(1, 2, T, 64, generator=g, device="cuda") for _ in range(2))
    idx, keep = _lists(1, 2, T, bs, 6, False, g)
    want = _dense(q, k, v, do, keep)
    for impl, name in (("auto", "f32_tile"), ("simt", "simt_tile")):
        nsa.set_impl(impl)
        lib.nsa_profile_enable(1)
        try:
            got = _run(nsa, "selection", q, k, v, do, idx, bs, 0)
            _run(nsa, "window", q, k, v, do, None, 0, 100)
            _run(nsa, "compression", q, k[:, :, :T // bs].contiguous(), v[:, :, :T // bs].contiguous(), do, None, bs, 0)
            torch.cuda.synchronize()
            seen = {n for n in L.profile_summary() if "_fwd_" in n or "_bwd_" in n}
        finally:
            lib.nsa_profile_enable(0)
            nsa.set_impl("auto")
        assert seen == {f"{name}_{way}_{kind}" for way in ("fwd", "bwd") for kind in ("slc", "win", "cmp")}, seen
        for x, y in zip(got, want):
            assert (x.double() - y).norm() <= 2.0 ** -20 * y.norm()
