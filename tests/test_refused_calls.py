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
