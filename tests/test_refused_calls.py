"""Calls the library refuses, and that a refusal leaves nothing behind."""
import ctypes
import importlib

import pytest
import torch

from tests.util import pkg


def _sizes(**changes):
    """Return code of nsa_attention_sizes for a small learned-pooling call (a host function: no GPU needed)."""
    L = importlib.import_module("openbox-llm_b200._lib")
    f = dict(block_size=64, n_sel=4, window=64, n_init=0, n_local=0, cmp_len=32, cmp_stride=16, learned=1,
             given_lists=0, need_grad=1, dq_accumulator=0, impl=0)
    dims = dict(B=1, Hq=4, Hkv=2, T=256, D=64, dtype=L.DTYPE_BF16)
    dims.update({k: v for k, v in changes.items() if k in dims})
    f.update({k: v for k, v in changes.items() if k not in dims})
    desc = L.NsaAttentionDesc(L.dims(**dims), *f.values())
    return L.lib().nsa_attention_sizes(desc, *[ctypes.c_size_t() for _ in range(3)])


def test_sizes_of_a_valid_call():
    assert _sizes() == 0
    assert _sizes(n_sel=0, given_lists=1) == 0


def test_scored_lists_need_a_slot():
    assert _sizes(n_sel=0) == -1


@pytest.mark.parametrize("bad", [dict(cmp_stride=12), dict(cmp_stride=24), dict(block_size=40), dict(n_init=-1),
                                 dict(n_local=1 << 18), dict(window=0), dict(T=1 << 20, dtype=1, n_sel=17)], ids=str)
def test_bad_arguments_are_refused_before_any_launch(bad):
    """What the scorer and the branches require is checked with the sizes: no kernel of a refused call runs."""
    assert _sizes(**bad) == -1


@pytest.mark.parametrize("name,dtype,at,says", [
    ("fwd_tokens", 1, {}, "token-major"), ("bwd_tokens", 1, {}, "token-major"), ("fwd_tokens", 0, dict(out=8), "16-byte"),
    ("bwd_tokens", 0, dict(tokens=8), "16-byte"), ("bwd_tokens", 0, dict(d_out=2), "16-byte"), ("fwd", 0, dict(out=8), "16-byte"),
    ("bwd", 0, dict(d_out=2), "16-byte")], ids=str)
def test_outputs_the_gates_cannot_take_are_refused_before_any_launch(name, dtype, at, says):
    """Tokens of another type than bf16, and a bf16 output, or its gradient, off a 16-byte boundary.  The addresses are no one's: the
    refusal has to come from the host, ahead of every launch."""
    L = importlib.import_module("openbox-llm_b200._lib")
    if torch.cuda.is_available():
        pytest.skip("for a machine without a GPU: what is not refused would be launched")
    lib, far = L.lib(), 1 << 20
    desc = L.NsaAttentionDesc(L.dims(1, 4, 2, 128, 64, dtype), 64, 1, 16, 0, 0, 64, 64, 0, 1, 1, 0, 0)
    n = [ctypes.c_size_t() for _ in range(3)]
    assert lib.nsa_attention_sizes(desc, *n) == 0
    t = L.OP_TENSORS(*[far] * 8, *(None,) * 6, *[far] * 11)
    t[15], t[16] = far + at.get("out", 0), far + at.get("d_out", 0)
    before = lib.nsa_launch_count()
    args = [desc, t, far, far, n[1 if "fwd" in name else 2].value]
    if name == "bwd_tokens":
        args.append(far + at.get("tokens", 0))
    assert getattr(lib, "nsa_attention_" + name)(*args, None) == -1 and says in lib.nsa_last_error().decode()
    assert lib.nsa_launch_count() == before


def _inputs(B, Hq, Hkv, T, D, seed=4):
    g = torch.Generator(device="cuda").manual_seed(seed)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    return [mk(B, Hq, T, D)] + [mk(B, Hkv, T, D) for _ in range(6)] + [mk(B, Hq, T, 3)]


def _off_by_one(t):
    """The same values in a contiguous view that starts one element into its buffer."""
    buf = t.new_empty(t.numel() + 1)
    view = buf[1:].view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.gpu
@pytest.mark.parametrize("grad", [False, True])
def test_a_call_that_fails_midway_joins_its_side_streams(grad):
    """ks at an odd address is refused by its tensor map (on the host) after the window kernel has gone to
    a side stream.  Under capture an unjoined side stream makes the capture fail; outside, the
    caller's stream waits for the side streams' work, and the next call is right."""
    nsa = pkg()
    L = importlib.import_module("openbox-llm_b200._lib")
    ins = [x.requires_grad_(grad) for x in _inputs(1, 16, 4, 512, 64)]
    want = nsa.nsa_attention(*ins, 64, 4, 128)
    bad = list(ins)
    bad[3] = _off_by_one(ins[3].detach()).requires_grad_(grad)

    def refused():
        with pytest.raises(L.NsaError):
            nsa.nsa_attention(*bad, 64, 4, 128)

    refused()
    assert torch.equal(nsa.nsa_attention(*ins, 64, 4, 128), want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        refused()
        out = nsa.nsa_attention(*ins, 64, 4, 128)
    graph.replay()
    assert torch.equal(out, want)
    assert nsa.lib().nsa_device_status(None) == 0
