"""Forms of a call that choose a path without changing the mathematics: block sizes, views, streams,
refused arguments, non-finite values where nothing attends them."""
import pytest
import torch

from oracle import nsa_oracle as O
from tests.test_small_blocks_and_tiles import TILES, _branch
from tests.util import cfg_id, check, dev, make_inputs, pkg

pytestmark = pytest.mark.gpu


def _shifted(t, by=1):
    """The same values in a contiguous view that starts `by` elements into its buffer."""
    view = t.new_empty(t.numel() + by)[by:].view(t.shape)
    return view.copy_(t)


def _selection_64(t, idx, bs):
    """Selection attention and its gradients in 64-bit arithmetic, dense, on the CPU."""
    q, k, v, do = (t[n].double() for n in ("q", "ks", "vs", "do"))
    B, Hq, T, D = q.shape
    G = Hq // k.shape[1]
    kk, vv = k.repeat_interleave(G, 1), v.repeat_interleave(G, 1)
    keep = torch.zeros(B, k.shape[1], T, T + bs, dtype=torch.bool)
    for s in range(idx.shape[-1]):
        for e in range(bs):
            pos = idx[..., s].long() * bs + e
            ok = (idx[..., s] >= 0) & (pos <= torch.arange(T))
            keep.scatter_(3, torch.where(ok, pos, T + e % bs)[..., None], True)
    keep = keep[..., :T].repeat_interleave(G, 1)
    s = (q @ kk.transpose(-1, -2) * D ** -0.5).masked_fill(~keep, float("-inf"))
    lse = torch.logsumexp(s, -1)
    p = torch.where(keep, (s - lse[..., None]).exp(), torch.zeros(()).double())
    o = p @ vv
    delta = (do * o).sum(-1)
    ds = p * (do @ vv.transpose(-1, -2) - delta[..., None]) * D ** -0.5
    fold = lambda x: x.view(B, k.shape[1], G, T, D).sum(2)
    return o, lse, delta, ds @ kk, fold(ds.transpose(-1, -2) @ q), fold(p.transpose(-1, -2) @ do)


@pytest.mark.parametrize("c", [dict(B=1, Hq=4, Hkv=2, D=64, T=200, block_size=16, S=3),
                               dict(B=1, Hq=8, Hkv=2, D=128, T=330, block_size=16, S=2),
                               dict(B=2, Hq=6, Hkv=2, D=64, T=256, block_size=32, S=4)], ids=cfg_id)
def test_small_blocks_are_fp32_arithmetic(c):
    """Selection on 16- and 32-token blocks by default: every result is the 64-bit value rounded to bf16 (8
    significant bits: half a step is at most 2^-8 of the value), plus what fp32 arithmetic leaves: sums
    of a few hundred terms and exponents of up to 2^3, each good to 2^-24, under 2e-5 of the largest
    value.  Probabilities in bf16 (2^-9 of the largest terms) miss that wherever terms cancel."""
    nsa = pkg()
    t = make_inputs(c, torch.bfloat16, seed=3)
    bs, idx = c["block_size"], t["block_idx"]
    o64, lse64, delta, dq64, dk64, dv64 = _selection_64(t, idx, bs)
    live = torch.isfinite(lse64)
    q, k, v, do = (dev(t[n], torch.bfloat16) for n in ("q", "ks", "vs", "do"))

    def close(got, want, what):
        bound = 2.0 ** -8 * want.abs() + 2e-5 * want.abs().max()
        assert ((got.double().cpu() - want).abs() <= bound).all(), what

    o, lse = nsa.selection_forward_triton(q, k, v, idx.cuda(), bs, return_lse=True)
    close(o, o64, "o")
    close(nsa.selection_attn_triton(q, k, v, idx.cuda(), bs), o64, "o through autograd")
    ones = torch.ones_like(lse)
    lse_in = torch.where(live, lse64, torch.full_like(lse64, O.LSE_EMPTY)).float().cuda()
    grads = nsa.ops._selection_backward(q, k, v, idx.cuda(), bs, do, o, lse_in, ones, delta.float().cuda())
    for got, want, what in zip(grads, (dq64, dk64, dv64), ("dq", "dk", "dv")):
        close(got, want, what)
    # the whole op, its gate open for the selection branch alone
    gate = torch.tensor([-1e4, 1e4, -1e4]).expand(*t["gate"].shape).bfloat16().cuda()
    ins = [dev(t[n], torch.bfloat16) for n in ("q", "kc", "vc", "ks", "vs", "kw", "vw")]
    close(nsa.nsa_fused_forward(*ins, gate, idx.cuda(), bs, 64), o64, "o of the whole op")
    ins = [x.requires_grad_(True) for x in ins]
    close(nsa.nsa_fused_forward(*ins, gate, idx.cuda(), bs, 64), o64, "o of the whole op, training")
    assert nsa.lib().nsa_device_status(None) == 0


@pytest.mark.parametrize("c", [dict(B=1, Hq=8, Hkv=2, D=64, T=1000), dict(B=2, Hq=16, Hkv=1, D=128, T=448),
                               dict(B=1, Hq=6, Hkv=2, D=64, T=333)], ids=str)
def test_branches_round_alike(c):
    """The three branches on the same keys give the same bits: a window over everything, summaries of one
    token each, and a list of every block (query-outer kernel) are one attention in one order."""
    nsa = pkg()
    B, Hq, Hkv, D, T = (c[n] for n in ("B", "Hq", "Hkv", "D", "T"))
    g = torch.Generator().manual_seed(8)
    q, k, v = (torch.randn(B, h, T, D, generator=g).bfloat16().cuda() for h in (Hq, Hkv, Hkv))
    o, lse = nsa.range_attn_forward(q, k, v, nsa.MODE_COMPRESS, 0, 1)
    idx = torch.arange((T + 63) // 64, dtype=torch.int32, device="cuda").expand(B, Hkv, T, -1).contiguous()
    nsa.set_option("sel_fwd_variant", 1)
    for o2, lse2 in (nsa.range_attn_forward(q, k, v, nsa.MODE_WINDOW, T, 0),
                     nsa.selection_forward_triton(q, k, v, idx, 64, return_lse=True)):
        assert torch.equal(o, o2) and torch.equal(lse, lse2)
    assert nsa.lib().nsa_device_status(None) == 0


def _attends(kind, T, W, bs, idx, key):
    """[B, Hkv, T] bool (or [T] for the window and compression): does the row of query t attend `key`?"""
    t = torch.arange(T)
    if kind == "window":
        return (t >= key) & (t - key < W)
    if kind == "compression":
        return t >= (key + 1) * bs - 1
    return (idx == key // bs).any(-1) & (t >= key)


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")], ids=str)
@pytest.mark.parametrize("Hq,Hkv,D,bs", [(8, 2, 64, 64), (16, 1, 128, 64), (6, 2, 64, 16)])
def test_forward_keeps_non_finite_keys_to_their_rows(Hq, Hkv, D, bs, bad):
    """tcgen05 forward: a key that is infinite or NaN reaches the rows that attend it and no other; all other
    rows keep their bits."""
    nsa = pkg()
    nsa.set_impl("tc")
    B, T, W, S = 1, 500, 70, 3
    c = dict(B=B, Hq=Hq, Hkv=Hkv, D=D, T=T, block_size=bs, S=S)
    t = make_inputs(c, torch.bfloat16, seed=12)
    q, k, v = (dev(t[n], torch.bfloat16) for n in ("q", "ks", "vs"))
    idx = t["block_idx"]
    n_cmp = T // bs

    def runs(k):
        yield "window", nsa.range_attn_forward(q, k, v, nsa.MODE_WINDOW, W, 0)
        yield "compression", nsa.range_attn_forward(q, k[:, :, :n_cmp], v[:, :, :n_cmp], nsa.MODE_COMPRESS, 0, bs)
        for variant in (1, 2):
            nsa.set_option("sel_fwd_variant", variant)
            yield "selection", nsa.selection_forward_triton(q, k, v, idx.cuda(), bs, return_lse=True)

    clean = list(runs(k))
    for key in (3, 66, 127, 300):
        k2 = k.clone()
        k2[:, :, key, 5] = bad
        for (kind, (o, lse)), (_, (o2, lse2)) in zip(clean, runs(k2)):
            if kind == "compression" and key >= n_cmp:
                continue
            hit = _attends(kind, T, W, bs, idx, key)
            hit = (hit if hit.dim() == 3 else hit.expand(B, Hkv, T)).repeat_interleave(Hq // Hkv, 1).cuda()
            assert hit.any() and not hit.all()
            assert torch.equal(o[~hit], o2[~hit]) and torch.equal(lse[~hit], lse2[~hit]), (kind, key)
    assert nsa.lib().nsa_device_status(None) == 0


def test_forward_mode_derivatives_are_refused():
    """There is no forward-mode derivative of the op: a tangent raises instead of being dropped, also where
    no input requires a gradient."""
    import torch.autograd.forward_ad as fwd
    nsa = pkg()
    c = dict(B=1, Hq=4, Hkv=2, D=64, T=192, block_size=64, S=2)
    t = make_inputs(c, torch.bfloat16, seed=1)
    ins = [dev(t[n], torch.bfloat16) for n in ("q", "kc", "vc", "ks", "vs", "kw", "vw", "gate")]
    idx = t["block_idx"].cuda()
    want = nsa.nsa_fused_forward(*ins, idx, 64, 64)
    assert not want.requires_grad
    with fwd.dual_level():
        for at in (0, 3, 7):
            dual = list(ins)
            dual[at] = fwd.make_dual(ins[at], torch.ones_like(ins[at]))
            for call in (lambda: nsa.nsa_fused_forward(*dual, idx, 64, 64), lambda: nsa.nsa_attention(*dual, 64, 2, 64)):
                with pytest.raises(NotImplementedError):
                    call()
                with torch.no_grad(), pytest.raises(NotImplementedError):
                    call()
        assert torch.equal(nsa.nsa_fused_forward(*ins, idx, 64, 64), want)


@pytest.mark.parametrize("dtype,D,by", [(torch.bfloat16, 64, 1), (torch.bfloat16, 128, 4), (torch.float32, 64, 1),
                                        (torch.float32, 32, 3), (torch.bfloat16, 16, 3)], ids=str)
def test_pooled_tensors_and_parameters_may_start_anywhere(dtype, D, by):
    """kc, vc and the compressor's parameters as contiguous views at any element offset (a slice of a flat
    buffer): the results are those of aligned tensors."""
    nsa = pkg()
    bs = 64
    c = dict(B=2, Hq=4, Hkv=2, D=D, T=330, block_size=bs, S=2)
    t = make_inputs(c, dtype, seed=6)
    ins = [dev(t[n], dtype) for n in ("q", "kc", "vc", "ks", "vs", "kw", "vw", "gate")]
    do, idx = dev(t["do"], dtype), t["block_idx"].cuda()
    g = torch.Generator().manual_seed(3)
    comp = {}
    for p in ("k", "v"):
        comp[p + "_intra"] = 0.1 * torch.randn(bs, D, generator=g).cuda()
        comp[p + "_logits"] = 0.3 * torch.randn(bs, generator=g).cuda()
        comp[p + "_proj"] = (torch.randn(D, D, generator=g) * D ** -0.5).cuda()
    moved = [x if i not in (1, 2) else _shifted(x, by) for i, x in enumerate(ins)]
    moved_comp = {n: _shifted(x, by) for n, x in comp.items()}

    def op(xs, cp, learned):
        xs = [x.detach().requires_grad_(True) for x in xs]
        cp = {n: x.detach().requires_grad_(True) for n, x in cp.items()}
        leaves = xs + (list(cp.values()) if learned else [])
        with torch.no_grad():
            bare = (nsa.nsa_attention(*xs, bs, 2, 70, compressor=cp) if learned else
                    nsa.nsa_fused_forward(*xs, idx, bs, 70))
        out = (nsa.nsa_attention(*xs, bs, 2, 70, compressor=cp) if learned else
               nsa.nsa_fused_forward(*xs, idx, bs, 70))
        assert torch.equal(bare, out)
        return [out.detach(), *torch.autograd.grad(out, leaves, do if xs[1].data_ptr() % 16 == 0 else _shifted(do, by))]

    for learned in (False, True):
        want, got = op(ins, comp, learned), op(moved, moved_comp, learned)
        assert torch.equal(want[0], got[0]), learned
        for i, (a, b) in enumerate(zip(got[1:], want[1:])):
            # sums that meet by atomics differ in their order alone: a bf16 step, or 1e-5 for fp32 (d k_intra
            # is zero but for rounding)
            bound = (2.0 ** -7 if b.dtype == torch.bfloat16 else 1e-5) * max(b.float().abs().max().item(), 1e-1)
            assert (a.float() - b.float()).abs().max().item() <= bound, (learned, i)

    # the pooling by itself, forward and backward; the scalar kernels add the window in another order
    for x, m in zip(ins[1:3], moved[1:3]):
        check(nsa.block_mean_pool(m, bs), nsa.block_mean_pool(x, bs).float().cpu(), dtype, "mean pool")
        both = []
        for y, cp in ((x, comp), (m, moved_comp)):
            y = y.detach().requires_grad_(True)
            ps = [cp["k_" + n].detach().requires_grad_(True) for n in ("intra", "logits", "proj")]
            s = nsa.block_compress(y, *ps, bs)
            both.append([s.detach(), *torch.autograd.grad(s, [y, *ps], torch.ones_like(s))])
        for a, b in zip(*both):
            check(b, a.float().cpu(), b.dtype, "learned pool")
    assert nsa.lib().nsa_device_status(None) == 0


def test_unaligned_rows_are_refused_by_the_c_call():
    """The C entry point cannot copy: it refuses kc off a 16-byte boundary, before any of its rows is read."""
    from tests.test_refused_calls import _inputs
    from tests.test_streams import _forward_call
    ins = _inputs(1, 8, 2, 512, 64)
    launch, _ = _forward_call([ins[0], _shifted(ins[1]), *ins[2:]])
    assert launch(torch.cuda.current_stream().cuda_stream) == -1
    launch, out = _forward_call(ins)
    assert launch(torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert torch.isfinite(out).all() and out.abs().sum() > 0


@pytest.mark.parametrize("where", ["k", "v", "q", "do"])
@pytest.mark.parametrize("dtype,D,bad", [(torch.float32, 64, float("nan")), (torch.float32, 16, float("inf")),
                                         (torch.float32, 128, float("-inf")), (torch.bfloat16, 32, float("inf"))], ids=str)
def test_cuda_core_tiles_keep_non_finite_values_to_their_rows(dtype, D, bad, where):
    """CUDA-core tiles of 64 rows x 64 keys, forward and backward: a value that is infinite or NaN reaches the rows
    that attend its key (k, v) or its own row (q, dO), and the gradients of the keys those rows
    attend; everything else is what it is without that value."""
    nsa = pkg()
    nsa.set_impl("simt")
    B, Hq, Hkv, T, bs, S, W = 22, 4, 2, 200, 16, 4, 40          # 22 x 14 tiles: two for every SM
    G = Hq // Hkv
    t = make_inputs(dict(B=B, Hq=Hq, Hkv=Hkv, D=D, T=T, block_size=bs, S=S), dtype, seed=9)
    q, k, v, do = (dev(t[n], dtype) for n in ("q", "ks", "vs", "do"))
    idx = t["block_idx"][:1].expand(B, -1, -1, -1).contiguous()
    tt, kk = torch.arange(T)[:, None], torch.arange(T)[None, :]
    keep = {"window": ((tt >= kk) & (tt - kk < W)).expand(Hkv, T, T),
            "compression": (tt >= (kk + 1) * 3 - 1).expand(Hkv, T, T),
            "selection": (idx[0, :, :, None, :] == (kk // bs)[None, :, :, None]).any(-1) & (tt >= kk)}

    def run(kind, q, k, v, do):
        if kind == "selection":
            o, lse = nsa.selection_forward_triton(q, k, v, idx.cuda(), bs, return_lse=True)
            return o, lse, nsa.ops._selection_backward(q, k, v, idx.cuda(), bs, do, o, lse)
        mode, w = (nsa.MODE_WINDOW, W) if kind == "window" else (nsa.MODE_COMPRESS, 3)
        o, lse = nsa.range_attn_forward(q, k, v, mode, w, w)
        return o, lse, nsa.range_attn_backward(q, k, v, o, lse, do, mode, w, w)

    for kind, m in keep.items():
        o, lse, (dq, dk, dv) = run(kind, q, k, v, do)
        for at in (2, 61, 130):
            x = {"q": q, "k": k, "v": v, "do": do}
            x[where] = x[where].clone()
            x[where][:, :, at, 3] = bad
            o2, lse2, (dq2, dk2, dv2) = run(kind, **x)
            rows = m[:, :, at] if where in "kv" else (torch.arange(T) == at).expand(Hkv, T)      # [Hkv, T]
            keys = (m & rows[:, :, None]).any(1)
            if where in "kv":
                keys[:, at] = True
            assert not rows.all() and not keys.all()
            r, u = ~rows.repeat_interleave(G, 0).cuda(), ~keys.cuda()
            if where != "do":
                assert torch.equal(o[:, r], o2[:, r]) and torch.equal(lse[:, r], lse2[:, r]), (kind, at)
            assert torch.equal(dq[:, r], dq2[:, r]), (kind, at)
            # the keys' sums meet by atomics, in any order: 1e-5 of the largest, and a bf16 step
            step = 2.0 ** -7 if dtype == torch.bfloat16 else 0.0
            for a, b in ((dk, dk2), (dv, dv2)):
                a, b = a[:, u].float(), b[:, u].float()
                assert ((a - b).abs() <= step * a.abs() + 1e-5 * a.abs().max()).all(), (kind, at)


@pytest.mark.parametrize("B,T", [(1, 128), (28, 128), (14, 250), (8, 448), (6, 640)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=str)
def test_repeated_blocks_count_alike_both_ways(dtype, B, T):
    """A list that names a block more than once: on the CUDA cores every slot counts, whichever of the row
    and tile kernels serves a direction (8 to 40 blocks for 4 slots: tiles up to 16 forward and 32
    backward, where there are tiles enough, here 300 and more but for the first)."""
    nsa = pkg()
    nsa.set_impl("simt")
    Hq, Hkv, D, bs, S = 6, 2, 32, 16, 4
    t = make_inputs(dict(B=B, Hq=Hq, Hkv=Hkv, D=D, T=T, block_size=bs, S=S), dtype, seed=2)
    idx = t["block_idx"].clone()
    idx[:, :, ::3, 2] = idx[:, :, ::3, 0]
    idx[:, 1, 5::7, 1:] = idx[:, 1, 5::7, :1]
    q, k, v, do = (t[n].double() for n in ("q", "ks", "vs", "do"))
    tt, kk = torch.arange(T)[:, None], torch.arange(T)[None, :]
    times = ((idx[:, :, :, None, :] == (kk // bs)[None, None, :, :, None]).sum(-1) * (tt >= kk)).repeat_interleave(Hq // Hkv, 1)
    kx, vx = (x.repeat_interleave(Hq // Hkv, 1) for x in (k, v))
    s = (q @ kx.transpose(-1, -2) * D ** -0.5).masked_fill(times == 0, float("-inf"))
    lse = (torch.logsumexp(s + times.double().clamp(min=1).log(), -1))
    live = torch.isfinite(lse)
    p = torch.where(times > 0, times * (s - torch.where(live, lse, torch.zeros_like(lse))[..., None]).exp(), torch.zeros_like(s))
    o = p @ vx
    ds = p * (do @ vx.transpose(-1, -2) - (do * o).sum(-1, keepdim=True)) * D ** -0.5
    fold = lambda x: x.view(B, Hkv, -1, T, D).sum(2)
    want = (ds @ kx, fold(ds.transpose(-1, -2) @ q), fold(p.transpose(-1, -2) @ do))
    dq_, dk_, dv_ = (dev(t[n], dtype) for n in ("q", "ks", "vs"))
    got_o, got_lse = nsa.selection_forward_triton(dq_, dk_, dv_, idx.cuda(), bs, return_lse=True)
    check(got_o, o.float(), dtype, "repeats o")
    assert (got_lse.cpu()[live].double() - lse[live]).abs().max().item() <= 1e-4
    grads = nsa.ops._selection_backward(dq_, dk_, dv_, idx.cuda(), bs, dev(t["do"], dtype), got_o, got_lse)
    for g, w, n in zip(grads, want, ("dq", "dk", "dv")):
        check(g, w.float(), dtype, f"repeats {n}", abs32=4e-3)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("c", TILES, ids=cfg_id)
def test_cuda_core_selection_tiles_fill_the_gpu(c, dtype):
    """The selection tiles serve calls with tiles enough for the SMs: the shapes that end inside a tile, on a batch
    that has two tiles per SM, against the oracle."""
    G = c["Hq"] // c["Hkv"]
    per_batch = (c["T"] * G + 63) // 64 * c["Hkv"]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _branch(dict(c, B=(2 * sms + per_batch - 1) // per_batch), dtype, "simt", None, "full tiles")


def test_more_units_than_a_grid_dimension_holds():
    """B x Hkv above 65535 on the CUDA cores, forward and backward: the last units are those of a
    call with 320 units (tiles enough to take the same kernels)."""
    nsa = pkg()
    B, H, T, D, bs, S = 8193, 8, 20, 16, 16, 1
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v, do = (torch.randn(B, H, T, D, generator=g, device="cuda") for _ in range(4))
    idx = torch.where(torch.arange(T, device="cuda") >= 15, 0, -1).to(torch.int32)[:, None].expand(B, H, T, S).contiguous()

    def run(sl):
        a, b, c, d = (x[sl].contiguous() for x in (q, k, v, do))
        i = idx[sl].contiguous()
        o, lse = nsa.range_attn_forward(a, b, c, nsa.MODE_WINDOW, 7, 0)
        out = [o, lse, *nsa.range_attn_backward(a, b, c, o, lse, d, nsa.MODE_WINDOW, 7, 0)]
        o, lse = nsa.selection_forward_triton(a, b, c, i, bs, return_lse=True)
        return out + [o, lse, *nsa.ops._selection_backward(a, b, c, i, bs, d, o, lse)]

    assert B * H > 65535
    for a, b in zip(run(slice(None)), run(slice(B - 40, B))):
        assert torch.equal(a[B - 40:], b)
    assert nsa.lib().nsa_device_status(None) == 0


def test_attention_rows_have_to_be_dense():
    """The attention calls ask for stride(-1) == 1, the whole op too: q of the drop-in call, K and V of the
    selection and window branches.  The pooled pair may be any view."""
    nsa = pkg()
    t = make_inputs(dict(B=1, Hq=4, Hkv=2, D=64, T=192, block_size=64, S=2), torch.bfloat16, seed=1)
    ins = [dev(t[n], torch.bfloat16) for n in ("q", "kc", "vc", "ks", "vs", "kw", "vw", "gate")]
    idx = t["block_idx"].cuda()
    want = nsa.nsa_fused_forward(*ins, idx, 64, 64)
    for i in range(7):
        xs = list(ins)
        xs[i] = ins[i].transpose(-1, -2).contiguous().transpose(-1, -2)
        calls = [lambda: nsa.nsa_fused_forward(*xs, idx, 64, 64), lambda: nsa.nsa_attention(*xs, 64, 2, 64, block_idx=idx)]
        for call, refused in zip(calls, (i in (0, 3, 4, 5, 6), i >= 3)):
            if refused:
                with pytest.raises(AssertionError):
                    call()
            else:
                assert torch.equal(call(), want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=str)
def test_branches_of_different_shapes(dtype):
    """One kv head for the pooled pair, two for the selected one, and a window pair that is longer than q:
    nsa_fused_forward takes them, forward and backward; with all K / V alike in value it is the plain call."""
    nsa = pkg()
    B, Hq, T, D, bs, W = 1, 4, 192, 64, 64, 100
    t = make_inputs(dict(B=B, Hq=Hq, Hkv=2, D=D, T=T, block_size=bs, S=2), dtype, seed=4)
    q, kc, vc, ks, vs, kw, vw, gate, do = (dev(t[n], dtype) for n in ("q", "kc", "vc", "ks", "vs", "kw", "vw", "gate", "do"))
    idx = t["block_idx"].cuda()
    kc, vc = kc[:, :1].contiguous(), vc[:, :1].contiguous()
    same = [x.requires_grad_(True) for x in (q, kc.expand(-1, 2, -1, -1).contiguous(), vc.expand(-1, 2, -1, -1).contiguous(),
                                             ks, vs, kw, vw, gate)]
    want = nsa.nsa_fused_forward(*same, idx, bs, W)
    dwant = torch.autograd.grad(want, same, do)
    longer = [torch.cat([x.detach(), torch.full_like(x[:, :, :64], 3.0)], 2) for x in (kw, vw)]
    mixed = [x.detach().requires_grad_(True) for x in (q, kc, vc, ks, vs, *longer, gate)]
    got = nsa.nsa_fused_forward(*mixed, idx, bs, W)
    dgot = list(torch.autograd.grad(got, mixed, do))
    check(got, want.detach().float().cpu(), dtype, "mixed shapes out")
    assert all((d[:, :, T:] == 0).all() for d in dgot[5:7])
    dgot[5:7] = [d[:, :, :T] for d in dgot[5:7]]
    for i, (a, b) in enumerate(zip(dgot, dwant)):
        b = b.float().sum(1, keepdim=True) if i in (1, 2) else b.float()
        # (dq: three roundings instead of one; d kc, d vc: two heads summed after rounding)
        assert (a.float() - b).norm() <= (2.0 ** -6 if dtype == torch.bfloat16 else 1e-5) * b.norm(), i
    out, lists = nsa.nsa_attention(*[x.detach() for x in mixed], bs, 2, W, block_idx=idx, return_block_idx=True)
    assert torch.equal(out, got) and torch.equal(lists, idx.int())
    assert nsa.lib().nsa_device_status(None) == 0
