"""block_mean_pool takes any head size: those whose rows lie evenly over a warp's lanes by vectors, the others by elements."""
import ctypes

import pytest
import torch

from oracle import nsa_oracle as O
from tests.util import pkg


def test_which_sizes_go_by_vectors():
    ok = pkg().lib()["_ZN3nsa12pool_mean_okEii"]             # bool pool_mean_ok(int D, int dtype)
    ok.restype = ctypes.c_bool
    L = pkg()._lib
    for D in range(-8, 1100):
        assert ok(D, L.DTYPE_BF16) == (D in (8, 16, 32, 64, 128, 256)), D
        assert ok(D, L.DTYPE_F32) == (D in (4, 8, 16, 32, 64, 128)), D


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=str)
@pytest.mark.parametrize("D", [4, 8, 12, 20, 24, 40, 48, 64, 80, 96, 128, 256, 320, 512])
def test_against_the_oracle(D, dtype):
    nsa = pkg()
    for T, bs in ((70, 16), (37, 5)):                        # tokens behind the last block
        g = torch.Generator().manual_seed(D + T)
        x = torch.randn(2, 3, T, D, generator=g).to(dtype)
        n = T // bs
        do = torch.randn(2, 3, n, D, generator=g).to(dtype)
        xs = x.cuda().requires_grad_(True)
        out = nsa.block_mean_pool(xs, bs)
        out.backward(do.cuda())
        want = x[:, :, :n * bs].double().view(2, 3, n, bs, D).mean(3)
        assert torch.equal(O.ref_block_mean_pool(x.double(), bs), want)
        # fp32 sums of bs terms and, in bf16, half a step of the result
        step = 2.0 ** -8 if dtype == torch.bfloat16 else 0.
        assert ((out.double().cpu() - want).abs() <= step * want.abs() + 1e-6).all()
        dx = torch.zeros(2, 3, T, D, dtype=torch.float64)
        dx[:, :, :n * bs] = (do.double() / bs).repeat_interleave(bs, 2)
        assert ((xs.grad.double().cpu() - dx).abs() <= step * dx.abs() + 1e-6).all()
