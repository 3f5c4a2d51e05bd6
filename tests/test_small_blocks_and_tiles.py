"""Edges of the selection kernels on 16- and 32-token blocks (several list blocks per 64-key tile),
of the tiled CUDA-core kernels and of the pooling kernels, against the oracle.  Tolerances are
those of tests/util.py:check (fp32: the reference's gates; bf16: rounding of the inputs)."""
import pytest
import torch

from oracle import nsa_oracle as O
from tests.util import cfg_id, check, dev, make_inputs, pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _reset():
    yield
    pkg().set_impl("auto")
    pkg().set_option("sel_fwd_variant", 0)


def _branch(c, dtype, impl, idx, tag):
    nsa = pkg()
    t = make_inputs(c, dtype, seed=5)
    bs, T = c["block_size"], c["T"]
    idx = t["block_idx"] if idx is None else idx
    keep = O.selection_keep_fn(idx, T, bs)
    o_ref, lse_ref = O.stream_attn_forward(t["q"], t["ks"], t["vs"], keep)
    grads_ref = O.stream_attn_backward(t["q"], t["ks"], t["vs"], o_ref, lse_ref, t["do"], keep)
    nsa.set_impl(impl)
    q, k, v, do = (dev(t[n], dtype) for n in ("q", "ks", "vs", "do"))
    o, lse = nsa.selection_forward_triton(q, k, v, idx.cuda(), bs, return_lse=True)
    check(o, o_ref, dtype, tag + " o")
    empty = lse_ref == O.LSE_EMPTY
    assert (lse.cpu()[empty] == O.LSE_EMPTY).all() and (o.float().cpu()[empty] == 0).all(), tag
    for g, r, n in zip(nsa.ops._selection_backward(q, k, v, idx.cuda(), bs, do, o, lse), grads_ref, ("dq", "dk", "dv")):
        check(g, r, dtype, f"{tag} {n}", abs32=4e-3)
    assert nsa.lib().nsa_device_status(None) == 0


# T around the edges of a 64-key tile and of a row tile; 1 to 16 blocks per list; 2, 3, 4 and 16 heads
# per kv head (64, 32, 32 and 8 queries per query-outer tile)
SMALL = [dict(B=1, Hq=8, Hkv=2, D=64, T=200, block_size=16, S=3),
         dict(B=2, Hq=16, Hkv=4, D=128, T=1000, block_size=16, S=8),
         dict(B=1, Hq=6, Hkv=2, D=64, T=575, block_size=32, S=5),
         dict(B=1, Hq=16, Hkv=1, D=128, T=449, block_size=32, S=16),
         dict(B=1, Hq=4, Hkv=2, D=64, T=17, block_size=16, S=1)]


@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("c", SMALL, ids=cfg_id)
def test_small_blocks_on_tensor_cores(c, variant):
    nsa = pkg()
    assert nsa.tc_supported(c["B"], c["Hq"], c["Hkv"], c["T"], c["D"], torch.bfloat16, c["block_size"])
    nsa.set_option("sel_fwd_variant", variant)
    _branch(c, torch.bfloat16, "tc", None, f"variant{variant}")
    recent = O.make_block_idx_recent(c["B"], c["Hkv"], c["T"], c["block_size"], c["S"])
    _branch(c, torch.bfloat16, "tc", recent, f"variant{variant} recent")


# row tiles of 64 rows: one head per kv head (64 queries a tile), 3 heads (a tile ends inside a
# query), more heads than rows; both sides of the tile rule's lines (4 and 8 blocks per slot)
TILES = [dict(B=1, Hq=2, Hkv=2, D=64, T=130, block_size=16, S=3),
         dict(B=1, Hq=6, Hkv=2, D=32, T=333, block_size=48, S=2),
         dict(B=1, Hq=80, Hkv=1, D=16, T=70, block_size=16, S=2),
         dict(B=1, Hq=4, Hkv=1, D=128, T=320, block_size=16, S=5),
         dict(B=1, Hq=4, Hkv=1, D=128, T=640, block_size=16, S=5),
         dict(B=1, Hq=4, Hkv=1, D=64, T=656, block_size=16, S=5)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("c", TILES, ids=cfg_id)
def test_cuda_core_tiles(c, dtype):
    nsa = pkg()
    _branch(c, dtype, "simt", None, "tile")
    t = make_inputs(c, dtype, seed=6)
    T = c["T"]
    q, k, v, do = (dev(t[n], dtype) for n in ("q", "kw", "vw", "do"))
    # (not W = 1: the softmax over one key is constant, so dq and dk are exactly zero and what either
    # side computes is the rounding of dP - delta, without a relative error to speak of)
    for W in (2, 63, 100, T + 5):
        keep = O.window_keep_fn(T, W)
        o_ref, lse_ref = O.stream_attn_forward(t["q"], t["kw"], t["vw"], keep)
        grads_ref = O.stream_attn_backward(t["q"], t["kw"], t["vw"], o_ref, lse_ref, t["do"], keep)
        o, lse = nsa.range_attn_forward(q, k, v, nsa.MODE_WINDOW, W, 0)
        check(o, o_ref, dtype, f"window {W} o")
        for g, r, n in zip(nsa.range_attn_backward(q, k, v, o, lse, do, nsa.MODE_WINDOW, W, 0), grads_ref, ("dq", "dk", "dv")):
            check(g, r, dtype, f"window {W} {n}", abs32=4e-3)


# few row tiles with long chains: clusters of 4 and 2 CTAs share one (the first tiles leave some of them without a
# key tile), at D = 64 and 128; lengths that end inside a tile
@pytest.mark.parametrize("c", [dict(B=1, Hq=8, Hkv=2, D=64, T=530, block_size=64, S=6),
                               dict(B=2, Hq=6, Hkv=2, D=64, T=1001, block_size=32, S=12),
                               dict(B=1, Hq=4, Hkv=1, D=128, T=530, block_size=64, S=6),
                               dict(B=1, Hq=4, Hkv=1, D=128, T=1090, block_size=64, S=5),
                               dict(B=1, Hq=12, Hkv=4, D=16, T=700, block_size=48, S=5)], ids=cfg_id)
def test_cuda_core_tiles_shared_by_clusters(c):
    nsa = pkg()
    _branch(c, torch.float32, "simt", None, "cluster")
    t = make_inputs(c, torch.float32, seed=6)
    q, k, v, do = (dev(t[n], torch.float32) for n in ("q", "kw", "vw", "do"))
    for W in (300, c["T"]):
        keep = O.window_keep_fn(c["T"], W)
        o_ref, lse_ref = O.stream_attn_forward(t["q"], t["kw"], t["vw"], keep)
        grads_ref = O.stream_attn_backward(t["q"], t["kw"], t["vw"], o_ref, lse_ref, t["do"], keep)
        o, lse = nsa.range_attn_forward(q, k, v, nsa.MODE_WINDOW, W, 0)
        check(o, o_ref, torch.float32, f"cluster window {W} o")
        assert (lse.cpu() - lse_ref).abs().max().item() <= 1e-4
        grads = nsa.range_attn_backward(q, k, v, o, lse, do, nsa.MODE_WINDOW, W, 0)
        for g, r, n in zip(grads, grads_ref, ("dq", "dk", "dv")):
            check(g, r, torch.float32, f"cluster window {W} {n}", abs32=4e-3)
        again = nsa.range_attn_backward(q, k, v, o, lse, do, nsa.MODE_WINDOW, W, 0)
        assert torch.equal(grads[0], again[0])           # dq adds up in rank order


# one summary row and many (2 and 8 rows per CTA, several groups per persistent CTA), windows longer
# than one pass of a CTA, a tail after the last window
@pytest.mark.parametrize("geom", [(1, 1, 64, 64, 64), (2, 3, 2500, 64, 64), (1, 2, 700, 128, 200), (1, 4, 333, 32, 48),
                                  (3, 8, 2048, 16, 16)], ids=str)
def test_learned_pooling_backward(geom):
    nsa = pkg()
    B, H, T, D, n = geom
    g = torch.Generator().manual_seed(2)
    x = torch.randn(B, H, T, D, generator=g).bfloat16()
    intra, logits = 0.1 * torch.randn(n, D, generator=g), 0.3 * torch.randn(n, generator=g)
    proj = torch.randn(D, D, generator=g) * D ** -0.5
    go = torch.randn(B, H, T // n, D, generator=g).bfloat16()
    ref = [t.float().clone().requires_grad_(True) for t in (x, intra, logits, proj)]
    blocks = ref[0][:, :, :T // n * n].reshape(B, H, T // n, n, D)
    pooled = ((blocks + ref[1]) * torch.softmax(ref[2], 0)[:, None]).sum(3)
    y_ref = pooled @ ref[3].T
    y_ref.backward(go.float())
    got = [t.cuda().requires_grad_(True) for t in (x, intra, logits, proj)]
    y = nsa.block_compress(*got, n)
    y.backward(go.cuda())
    check(y, y_ref.detach(), torch.bfloat16, "pooled")
    check(got[0].grad, ref[0].grad, torch.bfloat16, "pool dx")
    # fp32 sums over B*H*(T/n) rows in another order: relative to the largest entry
    for a, b, name in zip(got[1:], ref[1:], ("d_intra", "d_logits", "d_proj")):
        bound = 1e-4 * max(1.0, b.grad.abs().max().item())
        assert (a.grad.cpu() - b.grad).abs().max().item() <= bound, name


# eight tokens a thread (many rows) and one (few); lengths that end inside a group of eight
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=str)
@pytest.mark.parametrize("B,T,Hq,Hkv,D", [(2, 4141, 12, 4, 64), (3, 8, 5, 1, 32), (1, 4103, 16, 4, 128), (2, 9, 8, 2, 64)])
def test_projection_rows_to_heads_and_back(B, T, Hq, Hkv, D, dtype):
    ops = pkg().ops
    W = ops.fused_projection_width(Hq, Hkv, D)
    n = (Hq + 6 * Hkv) * D
    y = torch.randn(B, T, W, device="cuda").to(dtype)
    q, kv, gate = ops.split_heads(y, Hq, Hkv, D)
    assert torch.equal(q, y[..., :Hq * D].view(B, T, Hq, D).transpose(1, 2))
    assert torch.equal(kv, y[..., Hq * D:n].reshape(B, T, 6, Hkv, D).permute(2, 0, 3, 1, 4))
    assert torch.equal(gate, y[..., n:n + 3 * Hq].reshape(B, T, Hq, 3).transpose(1, 2))
    back = torch.full_like(y, float("nan"))
    ops._split_heads_launch(back, q, kv, gate, Hq, Hkv, D, True)
    assert torch.equal(back[..., :n + 3 * Hq], y[..., :n + 3 * Hq])
    assert (back[..., n + 3 * Hq:] == 0).all()
