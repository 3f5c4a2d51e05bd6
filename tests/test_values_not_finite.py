"""How far a value that is infinite or NaN reaches in the backward of the 64-token selection and of the window."""
import pytest
import torch

from tests.util import pkg

pytestmark = pytest.mark.gpu

BAD = [float("nan"), float("inf"), -float("inf")]


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda").bfloat16()


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("B,Hq,Hkv,D", [(1, 6, 2, 64), (2, 8, 2, 64), (1, 5, 1, 128), (1, 16, 2, 128), (60, 3, 1, 64)])
def test_selected_keys_that_no_query_reaches(B, Hq, Hkv, D, bad):
    """A list may name the block that holds its query, and of that the keys behind the query are not attended.  What stands there
    leaves dK and dV bit for bit as they are: rows that a tile does not have (groups of 3 and 5, a last tile that is not full)
    are zeros in Q and dO, and zeros times such a key are not zeros."""
    nsa = pkg()
    T, S = 256, 4
    g = torch.Generator("cuda").manual_seed(Hq)
    q, do, k, v = (_randn(g, B, h, T, D) for h in (Hq, Hq, Hkv, Hkv))
    t = torch.arange(T, device="cuda", dtype=torch.int32)
    own = torch.where(t % 64 < 40, t // 64, torch.full_like(t, -1))
    idx = torch.stack([own, torch.where(t >= 64, 0, -1).int(), torch.full_like(t, -1), torch.full_like(t, -1)], -1)
    idx = idx[None, None].expand(B, Hkv, T, S).contiguous()
    got = []
    for value in (0.0, bad):
        k2 = k.clone()
        k2[:, :, 64 + 50] = value
        k2[:, :, 192 + 63, 3] = value
        leaves = [x.clone().requires_grad_(True) for x in (q, k2, v)]
        o = nsa.selection_attn_triton(*leaves, idx, 64)
        got.append((o.detach(), *torch.autograd.grad(o, leaves, do)[1:]))
    for a, b in zip(*got):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b)
    assert nsa.lib().nsa_device_status(None) == 0
