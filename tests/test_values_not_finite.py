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


# tiles of 128 keys (csrc/tc_bwd_wide.cu: more tiles of 64 keys than SMs); rows per tile 126, 128, 125, 120 and 110
WINDOWS = [(40, 6, 2, 200, 64, 50), (40, 8, 2, 200, 128, 70), (20, 10, 2, 300, 64, 100), (20, 24, 2, 260, 128, 64), (10, 44, 2, 500, 64, 90)]


def _window(B, Hq, Hkv, T, D):
    assert B * Hkv * ((T + 63) // 64) > 148
    g = torch.Generator("cuda").manual_seed(Hq + T)
    q, do, k, v = (_randn(g, B, h, T, D) for h in (Hq, Hq, Hkv, Hkv))
    q[..., 0] = q[..., 0].abs() + 0.5
    return q, k, v, do


def _same_but(a, b, spare):
    """a and b bit for bit, but for the positions of dim 2 in `spare`, and finite there."""
    keep = torch.ones(a.shape[2], dtype=torch.bool, device=a.device)
    keep[list(spare)] = False
    return torch.equal(a[:, :, keep], b[:, :, keep]) and torch.isfinite(a[:, :, keep].float()).all().item()


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("B,Hq,Hkv,T,D,W", WINDOWS)
def test_window_v_that_is_not_finite_stays_with_the_rows_that_attend_it(B, Hq, Hkv, T, D, W, bad):
    nsa = pkg()
    q, k, v, do = _window(B, Hq, Hkv, T, D)
    o, lse = nsa.range_attn_forward(q, k, v, nsa.MODE_WINDOW, W, 0)
    want = nsa.range_attn_backward(q, k, v, o, lse, do, nsa.MODE_WINDOW, W, 0)
    at = 100
    v[:, :, at, 5] = bad
    dq, dk, dv = nsa.range_attn_backward(q, k, v, o, lse, do, nsa.MODE_WINDOW, W, 0)
    assert _same_but(dq, want[0], range(at, min(T, at + W)))
    assert not torch.isfinite(dq[:, :, at:at + W].float()).any(-1).any()
    assert _same_but(dk, want[1], [at]) and torch.equal(dv, want[2])
    assert nsa.lib().nsa_device_status(None) == 0


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("B,Hq,Hkv,T,D,W", WINDOWS)
def test_window_gradient_row_that_is_not_finite(B, Hq, Hkv, T, D, W, bad):
    """It reaches dK and dV of the key tiles that its query attends (0 x inf in the products over a tile), no other row's dQ."""
    nsa = pkg()
    q, k, v, do = _window(B, Hq, Hkv, T, D)
    o, lse = nsa.range_attn_forward(q, k, v, nsa.MODE_WINDOW, W, 0)
    want = nsa.range_attn_backward(q, k, v, o, lse, do, nsa.MODE_WINDOW, W, 0)
    t = 140
    do[:, 0, t, 7] = bad
    dq, dk, dv = nsa.range_attn_backward(q, k, v, o, lse, do, nsa.MODE_WINDOW, W, 0)
    assert torch.equal(dq[:, 1:], want[0][:, 1:]) and _same_but(dq[:, :1], want[0][:, :1], [t])
    assert torch.equal(dk[:, 1:], want[1][:, 1:]) and torch.equal(dv[:, 1:], want[2][:, 1:])
    reached = range((t - W + 1) // 128 * 128, min(T, t // 128 * 128 + 128))
    assert _same_but(dk[:, :1], want[1][:, :1], reached) and _same_but(dv[:, :1], want[2][:, :1], reached)
    assert nsa.lib().nsa_device_status(None) == 0


@pytest.mark.parametrize("B,Hq,Hkv,T,D,W", WINDOWS)
def test_window_key_without_weight_leaves_nothing(B, Hq, Hkv, T, D, W):
    """A key at minus infinity has p = 0 in every row: its dK and dV are 0, also beside rows that a tile does not have."""
    nsa = pkg()
    q, k, v, do = _window(B, Hq, Hkv, T, D)
    at, got = 77, []
    for value in (-1e30, -float("inf")):
        k[:, :, at, 0] = value
        o, lse = nsa.range_attn_forward(q, k, v, nsa.MODE_WINDOW, W, 0)
        got.append((o, lse, *nsa.range_attn_backward(q, k, v, o, lse, do, nsa.MODE_WINDOW, W, 0)))
    for a, b in zip(got[0][:2] + got[0][3:], got[1][:2] + got[1][3:]):
        assert torch.equal(a, b) and torch.isfinite(b.float()).all()
    assert (got[1][3][:, :, at] == 0).all() and (got[1][4][:, :, at] == 0).all()
    assert nsa.lib().nsa_device_status(None) == 0
