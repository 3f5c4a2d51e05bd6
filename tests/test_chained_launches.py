"""Kernels that are placed before the one ahead of them has ended read nothing of it early."""
import pytest
import torch

from tests.test_refused_calls import _inputs
from tests.util import pkg

pytestmark = pytest.mark.gpu

SHAPES = [(1, 8, 2, 64, 64, 2), (2, 6, 2, 200, 64, 4), (1, 16, 4, 1024, 64, 8), (1, 4, 1, 2500, 128, 16)]


def _parts(ins, S, settle):
    """The branches by their own entry points, with `settle` between the calls."""
    nsa = pkg()
    q, kc, vc, ks, vs, kw, vw, gate = ins
    k_cmp, v_cmp = nsa.block_mean_pool(kc, 64), nsa.block_mean_pool(vc, 64)
    settle()
    o_cmp, lse = nsa.range_attn_forward(q, k_cmp, v_cmp, nsa.MODE_COMPRESS, 0, 64)
    settle()
    idx = nsa.topn_blocks(q, k_cmp, lse, 64, S)
    settle()
    o_sel = nsa.selection_attn_triton(q, ks, vs, idx, 64)
    settle()
    return nsa.gate_combine(o_cmp, o_sel, nsa.window_attn_triton(q, kw, vw, 128), gate), idx, o_sel


@pytest.mark.parametrize("B,Hq,Hkv,T,D,S", SHAPES)
def test_one_behind_the_other_and_each_alone(B, Hq, Hkv, T, D, S):
    """Different inputs one behind the other on one stream, whose workspaces take over each other's memory, give bit for bit
    what parts that each start on an idle GPU give; so does the whole call, also replayed from a graph."""
    nsa = pkg()
    ins = [_inputs(B, Hq, Hkv, T, D, seed=s) for s in range(4)]
    with torch.no_grad():
        want = [_parts(x, S, torch.cuda.synchronize) for x in ins]
        got = [_parts(ins[k % 4], S, lambda: None) for k in range(16)]
        whole = [nsa.nsa_attention(*ins[k % 4], 64, S, 128, return_block_idx=True) for k in range(16)]
        held = [x.clone() for x in ins[0]]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = nsa.nsa_attention(*held, 64, S, 128)
        for k in range(8):
            for a, b in zip(held, ins[k % 4]):
                a.copy_(b)
            graph.replay()
            assert torch.equal(out, want[k % 4][0])
    for k in range(16):
        for a, b in zip(got[k], want[k % 4]):
            assert torch.equal(a, b)
        assert torch.equal(whole[k][0], want[k % 4][0]) and torch.equal(whole[k][1], want[k % 4][1])
    assert nsa.lib().nsa_device_status(None) == 0


@pytest.mark.parametrize("B,Hq,Hkv,T,D,S", SHAPES)
def test_the_backward_of_selection_behind_one_another(B, Hq, Hkv, T, D, S):
    """Row statistics, plan, backward and dQ sum in a row, of different inputs, against passes that each start on an idle GPU: dq bit for
    bit, dk and dv up to the order of fp32 adds (2^-7 of the largest entry)."""
    nsa = pkg()
    ins = [_inputs(B, Hq, Hkv, T, D, seed=s) for s in range(4)]
    g = torch.Generator("cuda").manual_seed(9)
    idx = [torch.randint(-1, (T + 63) // 64, (B, Hkv, T, S), generator=g, device="cuda", dtype=torch.int32) for _ in ins]

    def grads(k):
        q, _, _, ks, vs = (x.detach().requires_grad_(True) for x in ins[k][:5])
        return torch.autograd.grad(nsa.selection_attn_triton(q, ks, vs, idx[k], 64), (q, ks, vs), ins[(k + 1) % 4][0].detach())

    want = []
    for k in range(4):
        torch.cuda.synchronize()
        want.append(grads(k))
    torch.cuda.synchronize()
    got = [grads(k % 4) for k in range(16)]
    for k in range(16):
        assert torch.equal(got[k][0], want[k % 4][0])
        for a, b in zip(got[k][1:], want[k % 4][1:]):
            assert (a.float() - b.float()).abs().max() <= 2.0 ** -7 * b.float().abs().max()
    assert nsa.lib().nsa_device_status(None) == 0


@pytest.mark.parametrize("B,Hq,Hkv,T,D,S", [(1, 16, 4, 1024, 64, 8), (2, 6, 2, 300, 64, 4), (3, 12, 4, 1100, 128, 16)])
def test_a_training_pass_from_a_graph(B, Hq, Hkv, T, D, S):
    """Forward and backward of the whole call, captured once and replayed on other inputs: the branches' kernels lie on side
    streams, and the dQ sum is chained to one of them and waits for all.  Against passes outside of a graph, dq and d_gate bit
    for bit, the rest up to the order of fp32 adds."""
    nsa = pkg()
    ins = [[x.detach() for x in _inputs(B, Hq, Hkv, T, D, seed=s)] for s in range(3)]

    def run(leaves):
        out = nsa.nsa_attention(*leaves, 64, S, 128)
        return [out.detach(), *torch.autograd.grad(out, leaves, leaves[0].detach())]

    want = []
    for x in ins:
        torch.cuda.synchronize()
        want.append(run([t.clone().requires_grad_(True) for t in x]))
    held = [t.clone().requires_grad_(True) for t in ins[0]]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        run(held)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run(held)
    for k in range(9):
        with torch.no_grad():
            for a, b in zip(held, ins[k % 3]):
                a.copy_(b)
        graph.replay()
        for n, (a, b) in enumerate(zip(got, want[k % 3])):
            if n in (0, 1, 8):
                assert torch.equal(a, b), n
            else:
                assert (a.float() - b.float()).abs().max() <= 2.0 ** -7 * b.float().abs().max(), n
    assert nsa.lib().nsa_device_status(None) == 0
