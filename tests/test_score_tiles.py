"""Block scoring with the heads added up in registers: tiles of 32, 64 and 128 summaries and their remainders."""
import pytest
import torch

from oracle import nsa_oracle as O
from tests.util import pkg

pytestmark = pytest.mark.gpu


# summaries: one, a tile of 32 and of 64 less, exactly and more than full, a second tile of every size, a third
@pytest.mark.parametrize("n_blk", [1, 31, 33, 64, 65, 96, 128, 129, 161, 200, 256, 300])
@pytest.mark.parametrize("Hq,Hkv,D", [(3, 1, 64), (8, 2, 64), (10, 2, 128), (16, 1, 128), (9, 1, 64), (8, 2, 128), (3, 1, 128)])
def test_importances_and_lists(n_blk, Hq, Hkv, D):
    """Importances of all rows against 64 bits, and the lists against the canonical order of the kernel's own importances, bit for bit.  A
    score of a few units is good to 2^-20 (64 to 128 products, each rounded to 2^-24, and the tensor cores' truncation), the
    exponential and its argument to 2^-21, an importance is the sum of up to 16 of them: 2^-17 of the largest."""
    nsa = pkg()
    bs, S, B = 16, 16, 2
    T, G = n_blk * bs + 5, Hq // Hkv
    g = torch.Generator(device="cuda").manual_seed(n_blk)
    q = torch.randn(B, Hq, T, D, generator=g, device="cuda").bfloat16()
    k = torch.randn(B, Hkv, n_blk, D, generator=g, device="cuda").bfloat16()
    _, lse = nsa.range_attn_forward(q, k, k, nsa.MODE_COMPRESS, 0, bs)
    idx, imp = nsa.topn_blocks(q, k, lse, bs, S, return_importance=True)
    t = torch.arange(T, device="cuda")
    valid = (t[:, None] + 1) // bs > torch.arange(n_blk, device="cuda")
    s = q.double() @ k.double().repeat_interleave(G, 1).transpose(-1, -2) * D ** -0.5
    want = (s - lse.double()[..., None]).exp().masked_fill(~valid, 0.0).view(B, Hkv, G, T, n_blk).sum(2)
    assert ((imp.double() - want).abs() <= 2.0 ** -17 * want.amax(-1, keepdim=True)).all()
    assert (idx.cpu() == O.canonical_topn(imp.cpu(), valid.cpu(), S)).all()
    # without the importances: the same lists
    assert torch.equal(nsa.topn_blocks(q, k, lse, bs, S), idx)
    assert nsa.lib().nsa_device_status(None) == 0


@pytest.mark.parametrize("n_init,n_local", [(1, 2), (0, 1), (3, 0), (7, 9)])
@pytest.mark.parametrize("n_blk,Hq,Hkv,D", [(1, 4, 1, 64), (33, 16, 1, 64), (64, 6, 2, 128), (127, 8, 2, 64), (129, 8, 2, 128), (160, 10, 2, 64), (300, 3, 1, 64),
                                            (300, 16, 1, 128)])
def test_forced_blocks_on_the_summaries_grid(n_blk, Hq, Hkv, D, n_init, n_local):
    """The first blocks and those up to the query's are listed whatever their importance (the last has no summary yet), the others
    in the canonical order, bit for bit; forced blocks at the ends of tiles and lanes, and in a tile with no summary."""
    nsa = pkg()
    bs, S, B = 16, 16, 2
    T = n_blk * bs + 5
    g = torch.Generator(device="cuda").manual_seed(n_blk)
    q = torch.randn(B, Hq, T, D, generator=g, device="cuda").bfloat16()
    k = torch.randn(B, Hkv, n_blk, D, generator=g, device="cuda").bfloat16()
    _, lse = nsa.range_attn_forward(q, k, k, nsa.MODE_COMPRESS, 0, bs)
    _, imp = nsa.topn_blocks(q, k, lse, bs, S, return_importance=True)
    idx = nsa.topn_blocks(q, k, lse, bs, S, n_init_blocks=n_init, n_local_blocks=n_local)
    t = torch.arange(T)
    valid = (t[:, None] + 1) // bs > torch.arange(n_blk)
    assert (idx.cpu() == O.forced_topn(imp.cpu(), valid, S, T, bs, n_init, n_local)).all()
    assert nsa.lib().nsa_device_status(None) == 0


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T", [544, 1040, 1056, 1072, 2064, 2080])
def test_blocks_whose_first_summary_ends_a_tile(T, D):
    """Summaries of 32 tokens every 16 under blocks of 64: a block is a candidate as soon as the summary before it, which reaches
    into it, is visible; that one may be the last of its tile."""
    nsa = pkg()
    g = torch.Generator(device="cuda").manual_seed(T)
    n = (T - 32) // 16 + 1
    q = torch.randn(1, 8, T, D, generator=g, device="cuda").bfloat16()
    k = torch.randn(1, 2, n, D, generator=g, device="cuda").bfloat16()
    _, lse = nsa.range_attn_forward(q, k, k, nsa.MODE_COMPRESS_STRIDED, 16, 32)
    idx, imp = nsa.topn_blocks(q, k, lse, 64, 16, return_importance=True, cmp_len=32, cmp_stride=16)
    t = torch.arange(T, device="cuda")
    sees = (t[:, None] - 31) // 16 >= torch.arange(n, device="cuda")
    s = q.double() @ k.double().repeat_interleave(4, 1).transpose(-1, -2) * D ** -0.5
    p = (s - lse.double()[..., None]).exp().masked_fill(~sees, 0.0).view(1, 2, 4, T, n).sum(2)
    want, valid = O.block_importance(p.float().cpu(), T, 32, 16, 64)
    assert (imp.cpu() - want * valid).abs().max() <= 2.0 ** -17 * want.max()
    assert (idx.cpu() == O.forced_topn(imp.cpu(), valid, 16, T, 64, 0, 0)).all()
