"""The autograd nodes in C++ (csrc/torch_op.cpp) against the Python nodes and the separate modules they stand for."""
import importlib

import pytest
import torch
import torch.autograd.forward_ad as fwd

from tests.util import dev, make_inputs, pkg

pytestmark = pytest.mark.gpu
COMP = ("k_intra", "k_logits", "k_proj", "v_intra", "v_logits", "v_proj")


def _op_inputs(dtype, D, bs, T=200, n=None):
    t = make_inputs(dict(B=2, Hq=8, Hkv=2, D=D, T=T, block_size=bs, S=3), dtype, seed=5)
    ins = [dev(t[n], dtype) for n in ("q", "kc", "vc", "ks", "vs", "kw", "vw", "gate")]
    g = torch.Generator().manual_seed(1)
    n = n or bs
    comp = {}
    for p in ("k", "v"):
        comp[p + "_intra"] = 0.1 * torch.randn(n, D, generator=g).cuda()
        comp[p + "_logits"] = 0.3 * torch.randn(n, generator=g).cuda()
        comp[p + "_proj"] = (torch.randn(D, D, generator=g) * D ** -0.5).cuda()
    return ins, comp, t["block_idx"].cuda(), dev(t["do"], dtype)


def _close(a, b, i):
    step = 2.0 ** -7 if b.dtype == torch.bfloat16 else 1e-5      # sums that meet by atomics differ in their order
    assert a.dtype == b.dtype and a.shape == b.shape, i
    assert (a.float() - b.float()).abs().max() <= step * max(b.float().abs().max().item(), 0.1), i


@pytest.mark.parametrize("learned", [True, False])
@pytest.mark.parametrize("dtype,D,bs", [(torch.bfloat16, 64, 64), (torch.bfloat16, 128, 16), (torch.float32, 32, 32)], ids=str)
def test_op_is_what_the_python_node_gives(dtype, D, bs, learned):
    nsa = pkg()
    ins, comp, idx, do = _op_inputs(dtype, D, bs)

    def run(given, needs):
        xs = [x.detach().requires_grad_(i in needs) for i, x in enumerate(ins)]
        cp = {n: x.detach().requires_grad_(8 in needs) for n, x in comp.items()} if learned else None
        leaves = [x for x in [*xs, *(cp or {}).values()] if x.requires_grad]
        out, lists = nsa.nsa_attention(*xs, bs, 3, 70, compressor=cp, block_idx=idx if given else None, return_block_idx=True)
        res = [out.detach(), lists]
        if leaves:
            assert out.grad_fn is not None and not lists.requires_grad
            res += torch.autograd.grad(out, leaves, do, retain_graph=True)
            for a, b in zip(res[2:], torch.autograd.grad(out, leaves, do)):
                _close(a, b, "again")
            with pytest.raises(RuntimeError):
                torch.autograd.grad(out, leaves, do)
        return res

    for given in (False, True):
        for needs in ((), range(9), (0, 3, 7), (8,)):
            if not learned and 8 in needs and len(needs) == 1:
                continue
            got = run(given, needs)
            with fwd.dual_level():
                want = run(given, needs)
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
            assert len(got) == len(want)
            for i, (a, b) in enumerate(zip(got[2:], want[2:])):
                _close(a, b, (given, i))
    assert nsa.lib().nsa_device_status(None) == 0


def test_forms_that_the_node_leaves_alone():
    """Strided, shifted and mixed-type tensors, transforms and dispatch modes go the way they went; saved-tensor hooks
    see what the node keeps."""
    nsa = pkg()
    op = nsa._lib.torch_op().op
    ins, comp, idx, do = _op_inputs(torch.bfloat16, 64, 64)
    tail = (64, 3, 70, 0, 0, 64, 64, 0, 0)
    want = op(*ins, None, None, *tail)[0]
    assert torch.equal(want, nsa.nsa_attention(*ins, 64, 3, 70))
    for i in range(8):
        for other in (ins[i].transpose(0, 1).contiguous().transpose(0, 1), torch.cat([ins[i].flatten(), ins[i].flatten()[:1]])[1:].view_as(ins[i]),
                      ins[i].float(), ins[i].cpu(), ins[i][:1], torch.empty_like(ins[i], device="meta")):
            assert op(*[other if k == i else x for k, x in enumerate(ins)], None, None, *tail) is None
    assert op(*ins, idx.long(), None, *tail) is None and op(*ins, idx[:, :, :-1], None, *tail) is None
    assert op(*ins, None, tuple(comp[n] for n in COMP[:5]) + (comp["v_proj"].half(),), *tail) is None
    assert op(*ins, None, None, 64, 3, 70, 0, 0, 32, 16, 0, 0) is None and op(*ins, None, None, 8, *tail[1:]) is None

    class Mode(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    with Mode():
        assert op(*ins, None, None, *tail) is None
        assert torch.equal(nsa.nsa_attention(*ins, 64, 3, 70), want)

    def under_grad(x):
        assert op(x, *ins[1:], None, None, *tail) is None
        return x.float().sum()
    torch.func.grad(under_grad)(ins[0])
    seen = []
    xs = [x.detach().requires_grad_(True) for x in ins]
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t.shape), t.clone())[1], lambda t: t + 0):
        out = nsa.nsa_attention(*xs, 64, 3, 70, compressor=comp)
    got = torch.autograd.grad(out, xs, do)
    assert len(seen) == 16
    for i, (a, b) in enumerate(zip(got, torch.autograd.grad(nsa.nsa_attention(*xs, 64, 3, 70, compressor=comp), xs, do))):
        _close(a, b, i)
    xs[0].data.mul_(1)                          # data: no version
    out = nsa.nsa_attention(*xs, 64, 3, 70)
    with torch.no_grad():
        xs[3].add_(1)
    with pytest.raises(RuntimeError, match="inplace"):
        torch.autograd.grad(out, xs, do)


def test_failed_calls_raise_the_package_error():
    nsa = pkg()
    ins, comp, idx, _ = _op_inputs(torch.bfloat16, 64, 64)
    for kw in (dict(n_init_blocks=-1), dict(compressor=comp, cmp_len=64, cmp_stride=65)):
        with pytest.raises(nsa.NsaError):
            nsa.nsa_attention(*ins, 64, 3, 70, **kw)
        with pytest.raises(nsa.NsaError):
            nsa.nsa_attention(*[x.requires_grad_(True) for x in ins], 64, 3, 70, **kw)


@pytest.mark.parametrize("x_dtype", [torch.float32, torch.bfloat16], ids=str)
@pytest.mark.parametrize("B,T,Hq,Hkv,dh,bs", [(2, 200, 6, 2, 64, 64), (1, 129, 5, 1, 32, 16), (1, 64, 8, 2, 128, 32)], ids=str)
def test_layer_is_what_its_modules_give(B, T, Hq, Hkv, dh, bs, x_dtype):
    """Under bf16 autocast; a hook on out_proj sends the call through the modules.  The outputs are the same bits; the
    gradients of x, the weights and the bias leave their products in fp32 and not in bf16."""
    mod = importlib.import_module("openbox-llm_b200.module")
    torch.manual_seed(3)
    layer = mod.NSAAttentionB200(Hq * dh, Hq, Hkv, block_size=bs, n_selected_blocks=2, window=40).cuda()
    for n, p in layer.named_parameters():
        p.data.normal_(0, 0.02) if n != "gate.bias" else p.data.normal_(0, 1)
    x = torch.randn(B, T, Hq * dh, device="cuda").to(x_dtype)
    do = torch.randn(B, T, Hq * dh, device="cuda").bfloat16()
    lists = torch.zeros(B, Hkv, T, 1, dtype=torch.int32, device="cuda")

    def run(frozen=(), **kw):
        leaves = []
        for n, p in layer.named_parameters():
            p.requires_grad_(n not in frozen)
            if p.requires_grad:
                leaves.append(p)
        xs = x.detach().requires_grad_("x" not in frozen)
        if "x" not in frozen:
            leaves.append(xs)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = layer(xs, **kw)
            with torch.no_grad():
                assert torch.equal(layer(xs, **kw), y)
        return [y.detach(), *torch.autograd.grad(y, leaves, do)]

    for frozen, kw in (((), {}), (("x", "q_proj.weight", "gate.bias"), dict(block_idx=lists)), (("out_proj.weight", "k_win.weight"), {})):
        got = run(frozen, **kw)
        hook = layer.out_proj.register_forward_hook(lambda *a: None)
        want = run(frozen, **kw)
        hook.remove()
        assert torch.equal(got[0], want[0])
        for i, (a, b) in enumerate(zip(got[1:], want[1:])):
            assert a.dtype == b.dtype and a.shape == b.shape
            # bf16 rounding of the entries and of what they are sums of; k_intra is zero but for rounding
            assert (a.float() - b.float()).norm() <= 2.0 ** -6 * b.float().norm() + 1e-3, i
    assert pkg().lib().nsa_device_status(None) == 0


@pytest.mark.parametrize("D", [64, 128])
def test_blend_in_the_merge(D):
    """A call that fills the GPU blends the branches where the selection's partials are merged, if the block-outer kernel
    served it, and by the gate kernel if the query-outer one did: the same output but for the partials' rounding to bf16
    (2^-9 of each term), bit for bit the same with and without a backward to come."""
    nsa = pkg()
    B, Hq, Hkv, T = 1, 16, 2, 12352
    g = torch.Generator("cuda").manual_seed(2)
    mk = lambda h, n=D: torch.randn(B, h, T, n, generator=g, device="cuda").bfloat16()
    ins = [mk(Hq), *[mk(Hkv) for _ in range(6)], mk(Hq, 3)]
    outs = []
    for variant in (1, 2, 0):
        nsa.set_option("sel_fwd_variant", variant)
        try:
            out, idx = nsa.nsa_attention(*ins, 64, 16, 512, return_block_idx=True)
            xs = [x.detach().requires_grad_(True) for x in ins]
            assert torch.equal(nsa.nsa_attention(*xs, 64, 16, 512), out)
            assert torch.equal(nsa.nsa_attention(*ins, 64, 16, 512, block_idx=idx), out)
        finally:
            nsa.set_option("sel_fwd_variant", 0)
        outs.append(out.float())
    assert torch.equal(outs[2], outs[0]) or torch.equal(outs[2], outs[1])
    assert not torch.equal(outs[0], outs[1])
    assert (outs[0] - outs[1]).abs().max() <= 2.0 ** -6 and (outs[0] - outs[1]).norm() <= 2.0 ** -8 * outs[0].norm()
    assert nsa.lib().nsa_device_status(None) == 0


def _layer(dh=64, Hq=8, Hkv=2):
    mod = importlib.import_module("openbox-llm_b200.module")
    torch.manual_seed(3)
    layer = mod.NSAAttentionB200(Hq * dh, Hq, Hkv, block_size=64, n_selected_blocks=2, window=40).cuda()
    for n, p in layer.named_parameters():
        p.data.normal_(0, 0.02)
    return layer, torch.randn(2, 200, Hq * dh, device="cuda")


def test_out_proj_is_called_where_it_is_more_than_a_linear(monkeypatch):
    """A forward set on the instance or the class, a replaced F.linear and an active TorchFunctionMode take part in the call as
    they do in a call of the modules; the default-device mode does not keep the node away."""
    layer, x = _layer()
    lin = torch.nn.Linear.forward

    def call():
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return layer(x)
    want = call()
    assert "LayerNode" in want.grad_fn.name()
    with torch.device("cuda"):
        assert "LayerNode" in call().grad_fn.name()
    layer.out_proj.forward = lambda t: lin(layer.out_proj, t) + 1
    assert torch.equal(call(), want + 1)
    del layer.out_proj.forward
    assert torch.equal(call(), want)
    with monkeypatch.context() as m:
        m.setattr(torch.nn.Linear, "forward", lambda self, t: lin(self, t) + 1)
        assert torch.equal(call(), want + 1)
    seen = []
    with monkeypatch.context() as m:
        real = torch.nn.functional.linear
        m.setattr(torch.nn.functional, "linear", lambda *a, **k: (seen.append(a[1].shape), real(*a, **k))[1])
        assert torch.equal(call(), want)
    assert len(seen) == 2

    class Mode(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))
    with Mode():
        assert torch.equal(call(), want)
    assert seen.count(torch.nn.functional.linear) == 2


def test_frozen_parameters_cost_nothing():
    """With only out_proj trainable, or some other part of the layer, what a forward keeps and what a backward launches is no
    more than what the modules keep and launch, and the gradients are theirs."""
    nsa = pkg()
    layer, x = _layer()
    x = torch.cat([x] * 8)                       # 2.5 MB of activations a tensor: the weights are smaller
    do = torch.randn_like(x).bfloat16()
    names = [n for n, _ in layer.named_parameters()]
    parts = {"out_proj": ["out_proj.weight"], "compressor": [n for n in names if n.startswith("comp_")], "x": ["x"],
             "bias": ["gate.bias"], "weights": ["q_proj.weight", "v_win.weight"], "out_proj and compressor": ["out_proj.weight", "comp_k.proj.weight"]}

    requested = lambda: torch.cuda.memory_stats()["requested_bytes.all.current"]     # without what the allocator rounds up

    def run(what, asked=None):
        leaves = []
        for n, p in layer.named_parameters():
            p.requires_grad_(n in what)
            if n in what and n in (asked or what):
                leaves.append(p)
        xs = x.detach().requires_grad_("x" in what)
        if "x" in (asked or what):
            leaves.append(xs)
        torch.cuda.synchronize()
        base = requested()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = layer(xs)
        held, before = requested() - base, nsa.lib().nsa_launch_count()
        g = torch.autograd.grad(y, leaves, do)
        return y.detach(), g, held, nsa.lib().nsa_launch_count() - before

    for name, what in parts.items():
        run(what)
        got = run(what)
        hook = layer.out_proj.register_forward_hook(lambda *a: None)
        run(what)
        want = run(what)
        hook.remove()
        assert torch.equal(got[0], want[0]), name
        for a, b in zip(got[1], want[1]):
            assert a.dtype == b.dtype and (a.float() - b.float()).norm() <= 2.0 ** -6 * b.float().norm() + 1e-3, name
        assert got[2] <= want[2] + 64 * 1024, (name, got[2], want[2])
        assert got[3] <= want[3], (name, got[3], want[3])
    # trainable, but not asked for
    assert run(names, ["out_proj.weight"])[3] == 0
    assert run(names, ["out_proj.weight", "comp_v.proj.weight"])[3] < run(names, ["q_proj.weight"])[3]


def test_gradients_are_not_differentiated_again():
    """create_graph: the same gradients, which may be used and changed, and an error where a second derivative would have to
    come through the kernels: in the layer and in the op, through its C++ and its Python node."""
    nsa = pkg()
    layer, x = _layer()
    ins, comp, idx, do = _op_inputs(torch.bfloat16, 64, 64)
    strided = ins[0].transpose(1, 2).contiguous().transpose(1, 2)        # goes to the Python node

    def the_layer(x):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return layer(x)
    for f, x0 in ((the_layer, x), (lambda q: nsa.nsa_attention(q, *ins[1:], 64, 3, 70, compressor=comp), ins[0]),
                  (lambda q: nsa.nsa_attention(q, *ins[1:], 64, 3, 70, compressor=comp), strided)):
        leaf = x0.detach().requires_grad_(True)
        want, = torch.autograd.grad(f(leaf).float().square().sum(), leaf)
        y = f(leaf).float().square().sum()
        g, = torch.autograd.grad(y, leaf, create_graph=True)
        _close(g.detach(), want, "first")
        for loss in (g.float().square().sum(), y + g.float().square().sum()):
            with pytest.raises(RuntimeError, match="differentiated again"):
                loss.backward(retain_graph=True)
        leaf.grad = None                        # (what the failed passes reached before they failed)
        f(leaf).float().square().sum().backward(create_graph=True)
        with torch.no_grad():
            leaf.grad.mul_(2.)
        _close(leaf.grad.detach(), 2 * want, "second")
