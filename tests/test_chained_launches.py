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
