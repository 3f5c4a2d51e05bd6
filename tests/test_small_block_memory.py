"""Training on 16- and 32-token blocks: what it takes of memory, which sizes go where, and where its tensors may start."""
import ctypes

import pytest
import torch

from tests.util import cfg_id, dev, make_inputs, pkg


def _sizes(B, Hq, Hkv, T, D, bs, S, window=512, impl="auto"):
    L, lib = pkg()._lib, pkg().lib()
    d = L.NsaAttentionDesc(L.dims(B, Hq, Hkv, T, D, L.DTYPE_BF16), bs, S, window, 0, 0, bs, bs, 1, 0, 1, 0, L.IMPL[impl])
    n = [ctypes.c_size_t() for _ in range(3)]
    L.check(lib.nsa_attention_sizes(d, *n))
    return [x.value for x in n]


@pytest.mark.parametrize("T,D,bs,S", [(1024, 128, 16, 8), (2048, 64, 32, 4), (1000, 64, 16, 2)])
def test_backward_holds_the_partials_of_the_branches_and_no_second_set(T, D, bs, S):
    L, lib = pkg()._lib, pkg().lib()
    B, Hq, Hkv = 2, 16, 4
    dims = L.dims(B, Hq, Hkv, T, D, L.DTYPE_BF16)
    parts = (lib.nsa_range_attn_bwd_workspace_bytes(dims, T // bs, L.MODE_COMPRESS_STRIDED, bs, 0)
             + lib.nsa_range_attn_bwd_workspace_bytes(dims, T, L.MODE_WINDOW, 512, 0)
             + lib.nsa_selection_bwd_workspace_bytes(dims, S, bs, 0))
    n_q, n_c = B * Hq * T * D, B * Hkv * (T // bs) * D
    stats = 6 * B * Hq * T * 4 + 2 * n_c * 2 + 2 * (D * D + D + bs + 65) * 4
    assert parts <= _sizes(B, Hq, Hkv, T, D, bs, S)[2] <= parts + stats + 16 * 256 < parts + 3 * n_q * 2


def test_lines_of_the_tensor_core_kernels():
    """fp32 partials for calls of more than 12 M products up to 8 GB of them; on either side of that the accumulators of the
    CUDA cores."""
    L, lib = pkg()._lib, pkg().lib()
    ws = lambda T, S, D, impl, Hq=16, B=1, bs=16: lib.nsa_selection_bwd_workspace_bytes(
        L.dims(B, Hq, 4, T, D, L.DTYPE_BF16), S, bs, L.IMPL[impl])
    for S, on in ((1024, True), (1025, False)):              # a list of 32768 keys, and of more
        auto, simt = ws(64, S, 64, "auto", bs=32), ws(64, S, 64, "simt", bs=32)
        assert auto >= 16 * 64 * S * 64 * 4 if on else auto == simt
    most = int(8e9 / (16 * 8 * 128 * 4))                     # tokens
    for T, S, D, on in ((most, 8, 128, True), (most + 1, 8, 128, False), (4 * most, 4, 64, True), (4 * most + 4, 4, 64, False),
                        (184, 4, 64, True), (183, 4, 64, False), (2000, 1, 64, True)):
        assert on == (16 * T * S * 16 * D > 12e6 and 16 * T * S * D * 4 <= 8e9)
        auto, simt = ws(T, S, D, "auto"), ws(T, S, D, "simt")
        assert auto >= 16 * T * S * D * 4 if on else auto == simt, (T, S, D)


@pytest.mark.gpu
@pytest.mark.parametrize("c", [dict(B=2, Hq=16, Hkv=4, D=128, T=300, block_size=16, S=8),
                               dict(B=1, Hq=16, Hkv=1, D=64, T=833, block_size=32, S=5),      # clusters
                               dict(B=1, Hq=16, Hkv=1, D=128, T=833, block_size=32, S=5)], ids=cfg_id)
def test_gradients_may_start_anywhere(c):
    """Through the C interface: dks and dvs off every boundary; q, ks, vs, dO and dq off a 16-byte boundary are refused
    before anything is launched."""
    nsa = pkg()
    L, lib = nsa._lib, nsa.lib()
    t = make_inputs(c, torch.bfloat16, seed=3)
    ins = [dev(t[n], torch.bfloat16) for n in ("q", "kc", "vc", "ks", "vs", "kw", "vw", "gate")]
    do, bs, S = dev(t["do"], torch.bfloat16), c["block_size"], c["S"]
    idx = t["block_idx"].int().cuda()
    d = L.NsaAttentionDesc(L.dims(c["B"], c["Hq"], c["Hkv"], c["T"], c["D"], L.DTYPE_BF16), bs, S, 64, 0, 0, bs, bs, 0, 1, 1, 0, 0)
    n = [ctypes.c_size_t() for _ in range(3)]
    L.check(lib.nsa_attention_sizes(d, *n))
    saved, ws = (torch.empty(max(x.value, 1), dtype=torch.uint8, device="cuda") for x in (n[0], n[2]))
    out = torch.empty_like(ins[0])
    head = [x.data_ptr() for x in ins]
    fwd_ws = torch.empty(n[1].value + 1, dtype=torch.uint8, device="cuda")
    L.check(lib.nsa_attention_fwd(d, L.OP_TENSORS(*head, *(None,) * 6, idx.data_ptr(), out.data_ptr()), saved.data_ptr(),
                                  fwd_ws.data_ptr(), n[1].value, L.stream()))

    def backward(shift=(), src=head, d_out=do.data_ptr()):
        bufs = [x.new_full((x.numel() + 8,), float("nan")) for x in ins]
        grads = [b[(k in shift):][:x.numel()] for k, (b, x) in enumerate(zip(bufs, ins))]
        L.check(lib.nsa_attention_bwd(d, L.OP_TENSORS(*src, *(None,) * 6, idx.data_ptr(), None, d_out,
                                                      *[g.data_ptr() for g in grads]), saved.data_ptr(), ws.data_ptr(), n[2].value,
                                      L.stream()))
        return [g.clone() for g in grads]
    want = backward()
    for a, b in zip(backward(shift=(3, 4)), want):
        assert torch.isfinite(a).all()
        assert ((a.float() - b.float()).abs() <= 2.0 ** -7 * b.float().abs() + 1e-5 * b.float().abs().max()).all()
    before = lib.nsa_launch_count()
    for k in (0, 3, 4):
        with pytest.raises(nsa.NsaError, match="16-byte"):
            backward(src=[p + 2 * (j == k) for j, p in enumerate(head)])
    with pytest.raises(nsa.NsaError, match="16-byte"):
        backward(d_out=do.data_ptr() + 2)
    with pytest.raises(nsa.NsaError, match="16-byte"):
        backward(shift=(0,))
    assert lib.nsa_launch_count() == before
    assert lib.nsa_device_status(None) == 0
