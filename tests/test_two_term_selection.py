"""Selection on 16- and 32-token blocks by default: the tcgen05 kernels with P and dS in bf16 terms (three of them: the 24
bits of fp32) against the CUDA-core kernels (fp32 throughout) and against 64-bit arithmetic, over the forms of a call
that both accept; at small sizes too, which go to the CUDA cores otherwise."""
import pytest
import torch

from tests.test_call_forms import _selection_64, _shifted
from tests.util import cfg_id, dev, make_inputs, pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _reset():
    pkg().set_option("small_blocks_tc", 1)
    yield
    pkg().set_option("small_blocks_tc", 0)
    pkg().set_impl("auto")


def _both(q, k, v, do, idx, bs):
    """[o, dq, dk, dv, lse] by default and on the CUDA cores, both backward from the latter's o and LSE."""
    nsa = pkg()
    out = []
    for impl in ("simt", "auto"):
        nsa.set_impl(impl)
        o, lse = nsa.selection_forward_triton(q, k, v, idx, bs, return_lse=True)
        o_in, lse_in = (out[0][0], out[0][4]) if out else (o, lse)
        out.append([o, *nsa.ops._selection_backward(q, k, v, idx, bs, do, o_in, lse_in), lse])
    assert nsa.lib().nsa_device_status(None) == 0
    return out[1], out[0]


def _close(got, want, what):
    """Two bf16 roundings of the same value, each half a step (2^-9), and fp32 sums of up to a few thousand terms as large as the
    largest entry, 2^-24 off each (and 2^-21 in their exponentials): 4e-6 of it."""
    for a, b, n in zip(got, want, ("o", "dq", "dk", "dv")):
        a, b = a.double(), b.double()
        fin = torch.isfinite(b)
        assert torch.equal(torch.isfinite(a), fin), (what, n)
        a, b = a[fin], b[fin]
        assert ((a - b).abs() <= 2.0 ** -7 * b.abs() + 4e-6 * b.abs().max()).all(), (what, n)
    a, b = got[4], want[4]
    fin = torch.isfinite(b)
    assert torch.equal(torch.isfinite(a), fin) and ((a - b)[fin].abs() <= 1e-5 * b[fin].abs().clamp(min=1)).all(), (what, "lse")


# one key tile and less; tiles and row tiles that end ragged; 2, 3, 4, 16 and 64 heads a group; few key tiles with many
# rows (clusters); work items that are split (a block that every query lists, more than 128 row tiles); clusters of two, four and
# eight on more CTAs than SMs, and key tiles with too few rows for them
SHAPES = [dict(B=1, Hq=4, Hkv=2, D=64, T=17, block_size=16, S=1),
          dict(B=1, Hq=8, Hkv=2, D=128, T=64, block_size=16, S=3),
          dict(B=2, Hq=6, Hkv=2, D=64, T=129, block_size=32, S=2),
          dict(B=2, Hq=12, Hkv=4, D=128, T=447, block_size=16, S=8),
          dict(B=1, Hq=16, Hkv=1, D=128, T=833, block_size=32, S=5),
          dict(B=1, Hq=64, Hkv=1, D=64, T=321, block_size=16, S=40),
          dict(B=1, Hq=16, Hkv=1, D=64, T=1100, block_size=16, S=4),
          dict(B=1, Hq=16, Hkv=1, D=128, T=1100, block_size=16, S=4),
          dict(B=2, Hq=16, Hkv=4, D=128, T=1030, block_size=16, S=3),
          dict(B=1, Hq=8, Hkv=2, D=64, T=1543, block_size=16, S=3),
          dict(B=1, Hq=4, Hkv=1, D=64, T=1600, block_size=32, S=3),
          dict(B=8, Hq=16, Hkv=4, D=64, T=250, block_size=16, S=3)]


@pytest.mark.parametrize("c", SHAPES, ids=cfg_id)
def test_against_the_cuda_cores_and_64_bits(c):
    t = make_inputs(c, torch.bfloat16, seed=4)
    bs, idx = c["block_size"], t["block_idx"].clone()
    if c["T"] > 1000:
        idx[..., -1] = torch.where((idx == 0).any(-1), idx[..., -1], torch.zeros_like(idx[..., -1]))
    ins = [dev(t[n], torch.bfloat16) for n in ("q", "ks", "vs", "do")]
    got, want = _both(*ins, idx.cuda(), bs)
    _close(got, want, "auto against simt")
    if c["T"] > 500:
        return
    o64, _, _, dq64, dk64, dv64 = _selection_64(t, idx, bs)
    for a, b, r, n in zip(got, want, (o64, dq64, dk64, dv64), ("o", "dq", "dk", "dv")):
        e = [((x.double().cpu() - r).norm() / r.norm().clamp(min=1e-300)).item() for x in (a, b)]
        # a bf16 result is off by its rounding whoever computes it; 2 % for which way the ties of few values fall
        assert e[0] <= 1.02 * e[1] + 1e-6, (n, e)


@pytest.mark.parametrize("where", ["k", "v", "q", "do"])
@pytest.mark.parametrize("D,Hkv,bad", [(64, 2, float("inf")), (128, 1, float("nan")), (64, 1, float("-inf"))], ids=str)
def test_non_finite_values_stay_with_their_rows(D, Hkv, bad, where):
    """A value that is infinite or NaN reaches what attends it, as it does in the CUDA-core kernels, and no more."""
    c = dict(B=1, Hq=8, Hkv=Hkv, D=D, T=200, block_size=16, S=3)
    t = make_inputs(c, torch.bfloat16, seed=9)
    x = {n: dev(t[m], torch.bfloat16) for n, m in (("q", "q"), ("k", "ks"), ("v", "vs"), ("do", "do"))}
    idx = t["block_idx"].cuda()
    for at in (2, 61, 130):
        y = dict(x)
        y[where] = x[where].clone()
        y[where][:, :, at, 3] = bad
        _close(*_both(**y, idx=idx, bs=16), (where, at))


@pytest.mark.parametrize("bs,S", [(16, 4), (32, 3)])
@pytest.mark.parametrize("D", [64, 128])
def test_repeated_blocks_count_as_often_as_listed(D, bs, S):
    c = dict(B=2, Hq=6, Hkv=2, D=D, T=333, block_size=bs, S=S)
    t = make_inputs(c, torch.bfloat16, seed=2)
    idx = t["block_idx"].clone()
    idx[:, :, ::3, 2] = idx[:, :, ::3, 0]
    idx[:, 1, 5::7, 1:] = idx[:, 1, 5::7, :1]
    ins = [dev(t[n], torch.bfloat16) for n in ("q", "ks", "vs", "do")]
    _close(*_both(*ins, idx.cuda(), bs), "repeats")


def test_views_off_a_16_byte_boundary():
    """What the tensor cores load by TMA starts on a 16-byte boundary: q, v and dO that do not leave the call to the
    CUDA cores, whose row kernels read them by elements; K (and V in backward), which they read as
    16-byte vectors, are refused."""
    nsa = pkg()
    c = dict(B=1, Hq=8, Hkv=2, D=64, T=200, block_size=16, S=3)
    t = make_inputs(c, torch.bfloat16, seed=1)
    q, k, v, do = (dev(t[n], torch.bfloat16) for n in ("q", "ks", "vs", "do"))
    idx = t["block_idx"].cuda()
    nsa.set_impl("simt")
    o, lse = nsa.selection_forward_triton(q, k, v, idx, 16, return_lse=True)
    grads = nsa.ops._selection_backward(q, k, v, idx, 16, do, o, lse)
    nsa.set_impl("auto")
    for x in ((_shifted(q), k, v), (q, k, _shifted(v))):
        for a, b in zip(nsa.selection_forward_triton(*x, idx, 16, return_lse=True), (o, lse)):
            assert torch.equal(a, b)
    for x in ((_shifted(q), k, v, do), (q, k, v, _shifted(do))):
        got = nsa.ops._selection_backward(*x[:3], idx, 16, x[3], o, lse)
        assert torch.equal(got[0], grads[0])
        for a, b in zip(got[1:], grads[1:]):                     # sums that meet by atomics, rounded to bf16
            assert ((a.float() - b.float()).abs() <= 2.0 ** -7 * b.float().abs() + 1e-5 * b.float().abs().max()).all()
    with pytest.raises(nsa._lib.NsaError):
        nsa.selection_forward_triton(q, _shifted(k), v, idx, 16)
    for x in ((q, _shifted(k), v), (q, k, _shifted(v))):
        with pytest.raises(nsa._lib.NsaError):
            nsa.ops._selection_backward(*x, idx, 16, do, o, lse)
    # the whole op, forward
    ins = [dev(t[n], torch.bfloat16) for n in ("q", "kc", "vc", "ks", "vs", "kw", "vw", "gate")]
    want = nsa.nsa_fused_forward(*ins, idx, 16, 64)
    ins[4] = _shifted(ins[4])
    got = nsa.nsa_fused_forward(*ins, idx, 16, 64)
    assert ((got.float() - want.float()).abs() <= 2.0 ** -6 * want.float().abs().clamp(min=1)).all()
    assert nsa.lib().nsa_device_status(None) == 0


@pytest.mark.parametrize("D,bs,S", [(64, 16, 4), (128, 16, 8), (64, 32, 4), (128, 32, 4)])
def test_sums_that_cancel_keep_the_bits_of_fp32(D, bs, S):
    """Scores close to one another and values that are +64 and -64 in turn: what is left of the sum is 2^-9 of its terms, so
    that 16 bits of P show (12 % over the rounding of the result, where fp32 stays within 1 %)."""
    T = 300
    g = torch.Generator().manual_seed(3)
    q, do = (torch.randn(1, 8, T, D, generator=g).bfloat16() for _ in range(2))
    k, v = (torch.randn(1, 2, T, D, generator=g).bfloat16() for _ in range(2))
    q = q / 512
    v[..., 0] = torch.where(torch.arange(T) % 2 == 0, 64., -64.)
    c = dict(B=1, Hq=8, Hkv=2, D=D, T=T, block_size=bs, S=S)
    idx = make_inputs(c, torch.bfloat16, seed=1)["block_idx"]
    got, want = _both(*(x.cuda() for x in (q, k, v, do)), idx.cuda(), bs)
    o64 = _selection_64(dict(q=q, ks=k, vs=v, do=do), idx, bs)[0][..., 0]
    err = [((x[0][..., 0].double().cpu() - o64).norm() / o64.norm()).item() for x in (got, want)]
    assert err[0] <= 1.03 * err[1], err


def test_small_calls_give_the_bits_of_the_cuda_cores():
    """The layer's default sizes, and one size past the line."""
    nsa = pkg()
    nsa.set_option("small_blocks_tc", 0)
    for T, same in ((256, True), (500, False)):
        t = make_inputs(dict(B=1, Hq=8, Hkv=2, D=64, T=T, block_size=16, S=4), torch.bfloat16, seed=3)
        ins = [dev(t[n], torch.bfloat16) for n in ("q", "ks", "vs", "do")]
        got, want = _both(*ins, t["block_idx"].cuda(), 16)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) or not same
        _close(got, want, T)


# past the plan that one cluster builds (2048 tokens, 64 units); S that divides 32 and S that does not; row tiles of a ragged end
@pytest.mark.parametrize("B,Hq,Hkv,D,T,bs,S", [(1, 4, 2, 64, 2100, 16, 4), (1, 8, 2, 128, 2100, 32, 5), (1, 4, 1, 64, 2049, 16, 5),
                                               (33, 4, 2, 64, 130, 16, 4), (33, 6, 2, 64, 130, 32, 3), (17, 8, 4, 128, 130, 16, 8)])
def test_repeats_are_seen_by_every_plan(B, Hq, Hkv, D, T, bs, S):
    """Lists without repeats, with one in the last unit alone, with many, and without again, in one piece of memory."""
    nsa = pkg()
    t = make_inputs(dict(B=B, Hq=Hq, Hkv=Hkv, D=D, T=T, block_size=bs, S=S), torch.bfloat16, seed=8)
    q, k, v, do = (dev(t[n], torch.bfloat16) for n in ("q", "ks", "vs", "do"))
    plain = t["block_idx"].clone()
    plain = torch.where((plain[..., :, None] == plain[..., None, :]).tril(-1).any(-1), torch.full_like(plain, -1), plain)
    one, many = plain.clone(), plain.clone()
    one[-1, -1, T - 3, 1:3] = one[-1, -1, T - 3, :1]
    many[:, :, ::3, -1] = many[:, :, ::3, 0]
    many[:, -1, 5::7, 1:] = many[:, -1, 5::7, :1]
    assert not torch.equal(one, plain) and not torch.equal(many, plain)
    L, lib = nsa._lib, nsa.lib()
    dims = L.dims(B, Hq, Hkv, T, D, L.DTYPE_BF16)
    n = lib.nsa_selection_bwd_workspace_bytes(dims, S, bs, 0)
    ws = torch.full((n,), 0xa5, dtype=torch.uint8, device="cuda")
    for idx in (plain, one, many, plain, many):
        i = idx.int().cuda()
        nsa.set_impl("simt")
        o, lse = nsa.selection_forward_triton(q, k, v, i, bs, return_lse=True)
        want = [o, *nsa.ops._selection_backward(q, k, v, i, bs, do, o, lse), lse]
        nsa.set_impl("auto")
        got_o, got_lse = nsa.selection_forward_triton(q, k, v, i, bs, return_lse=True)
        grads = [torch.empty_like(x) for x in (q, k, v)]
        L.check(lib.nsa_selection_bwd(*map(L.ptr, (q, k, v, i, o, lse, do, *grads)), dims, S, bs, None, None, L.ptr(ws), n, 0,
                                      L.stream()))
        _close([got_o, *grads, got_lse], want, "plan")
    assert lib.nsa_device_status(None) == 0


@pytest.mark.parametrize("where", ["k", "v", "q", "do"])
@pytest.mark.parametrize("D,T,bs,S", [(64, 1100, 16, 4), (128, 1100, 16, 4), (128, 833, 32, 5)], ids=str)
def test_non_finite_values_in_shared_and_split_tiles(D, T, bs, S, where):
    """Key tiles whose rows a cluster shares out, and one that every query lists: more row tiles than a work item has.  Repeated
    blocks among the lists."""
    t = make_inputs(dict(B=1, Hq=16, Hkv=1, D=D, T=T, block_size=bs, S=S), torch.bfloat16, seed=4)
    idx = t["block_idx"].clone()
    idx[..., -1] = 0
    idx[:, :, ::9, 1] = idx[:, :, ::9, 0]
    x = {n: dev(t[m], torch.bfloat16) for n, m in (("q", "q"), ("k", "ks"), ("v", "vs"), ("do", "do"))}
    for at, bad in ((3, float("nan")), (T - 40, float("inf"))):
        y = dict(x)
        y[where] = x[where].clone()
        y[where][:, :, at, 3] = bad
        _close(*_both(**y, idx=idx.cuda(), bs=bs), (where, at))


def test_a_value_that_is_not_finite_does_not_cost_a_hundred_passes():
    """Every query attends a NaN: the rows and tiles that are done again in scalar code take the backward from 1 to about 27 ms,
    the forward from 0.5 to 2 (by elements they took 151 and 9)."""
    nsa = pkg()
    B, Hq, Hkv, T, D, bs, S = 1, 4, 1, 8192, 128, 16, 8
    g = torch.Generator("cuda").manual_seed(3)
    mk = lambda h: torch.randn(B, h, T, D, generator=g, device="cuda").bfloat16()
    q, do, k, v = mk(Hq), mk(Hq), mk(Hkv), mk(Hkv)
    idx = torch.rand(B, Hkv, T, T // bs, generator=g, device="cuda").topk(S, -1).indices.int()
    idx[..., 0] = 0
    v[:, :, 3, 5] = float("nan")

    def once(f):
        f()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        b.synchronize()
        return a.elapsed_time(b)
    o, lse = nsa.selection_forward_triton(q, k, v, idx, bs, return_lse=True)
    assert once(lambda: nsa.selection_forward_triton(q, k, v, idx, bs)) < 5
    assert once(lambda: nsa.ops._selection_backward(q, k, v, idx, bs, do, o, lse)) < 70
    assert nsa.lib().nsa_device_status(None) == 0
