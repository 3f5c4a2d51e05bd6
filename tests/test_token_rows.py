"""The whole op with its output and the gradient of it in token order, as the projection layer runs it."""
import ctypes

import pytest
import torch

from tests.util import cfg_id, dev, make_inputs, pkg


@pytest.mark.gpu
@pytest.mark.parametrize("variant", [0, 2])                 # 2: the block-outer selection, whose merge writes the blend
@pytest.mark.parametrize("c", [dict(B=2, Hq=6, Hkv=2, D=64, T=333, block_size=64, S=4),
                               dict(B=3, Hq=4, Hkv=2, D=16, T=77, block_size=16, S=2),
                               dict(B=1, Hq=16, Hkv=4, D=128, T=5121, block_size=64, S=4),
                               dict(B=1, Hq=64, Hkv=4, D=64, T=5121, block_size=64, S=4)], ids=cfg_id)   # (no overlap)
def test_token_rows(c, variant):
    """The same bits as in the order of the heads, in each route of the blend: the output; the gradient's rows that the
    backward writes; the gradients of its fixed-order sums, and the others to the rounding of bf16 under fp32 sums in any order."""
    nsa = pkg()
    L, lib = nsa._lib, nsa.lib()
    t = make_inputs(c, torch.bfloat16, seed=4)
    ins = [dev(t[n], torch.bfloat16) for n in ("q", "kc", "vc", "ks", "vs", "kw", "vw", "gate")]
    do, idx, bs, S = dev(t["do"], torch.bfloat16), t["block_idx"].int().cuda(), c["block_size"], c["S"]
    d = L.NsaAttentionDesc(L.dims(c["B"], c["Hq"], c["Hkv"], c["T"], c["D"], L.DTYPE_BF16), bs, S, 100, 0, 0, bs, bs, 0, 1, 1, 0, 0)
    head = [x.data_ptr() for x in ins]
    nsa.set_option("sel_fwd_variant", variant)
    try:
        n = [ctypes.c_size_t() for _ in range(3)]
        L.check(lib.nsa_attention_sizes(d, *n))

        def run(tokens):
            saved, fws, ws = (torch.empty(x.value + 1, dtype=torch.uint8, device="cuda") for x in n)
            out, rows = torch.empty_like(ins[0]), do
            if tokens:
                out, rows = out.transpose(1, 2).contiguous(), torch.full_like(do, float("nan"))
            fwd = lib.nsa_attention_fwd_tokens if tokens else lib.nsa_attention_fwd
            L.check(fwd(d, L.OP_TENSORS(*head, *(None,) * 6, idx.data_ptr(), out.data_ptr()), saved.data_ptr(), fws.data_ptr(),
                        n[1].value, L.stream()))
            grads = [torch.empty_like(x) for x in ins]
            args = [d, L.OP_TENSORS(*head, *(None,) * 6, idx.data_ptr(), None, rows.data_ptr(), *[g.data_ptr() for g in grads]),
                    saved.data_ptr(), ws.data_ptr(), n[2].value]
            if tokens:
                by_token = do.transpose(1, 2).contiguous()
                L.check(lib.nsa_attention_bwd_tokens(*args, by_token.data_ptr(), L.stream()))
                assert torch.equal(rows, do)
                out = out.transpose(1, 2)
            else:
                L.check(lib.nsa_attention_bwd(*args, L.stream()))
            torch.cuda.synchronize()
            return [out, *grads]
        a, b = run(True), run(False)
    finally:
        nsa.set_option("sel_fwd_variant", 0)
    for k, (x, y) in enumerate(zip(a, b)):
        if k in (0, 8) or c["D"] != 16 and k == 1:          # out, d_gate, dq
            assert torch.equal(x, y), k
        assert ((x.float() - y.float()).abs() <= 2.0 ** -7 * y.float().abs() + 1e-5 * y.float().abs().max()).all(), k
    assert lib.nsa_device_status(None) == 0


@pytest.mark.gpu
def test_token_rows_of_other_types_are_refused():
    """fp32 has the order of the heads only; what is refused launches nothing."""
    nsa = pkg()
    L, lib = nsa._lib, nsa.lib()
    x = [torch.zeros(1, h, 64, w, device="cuda") for h, w in ((2, 64), *[(1, 64)] * 6, (2, 3))]
    idx = torch.zeros(1, 1, 64, 1, dtype=torch.int32, device="cuda")
    d = L.NsaAttentionDesc(L.dims(1, 2, 1, 64, 64, L.DTYPE_F32), 64, 1, 16, 0, 0, 64, 64, 0, 1, 0, 0, 0)
    n = [ctypes.c_size_t() for _ in range(3)]
    L.check(lib.nsa_attention_sizes(d, *n))
    mem = [torch.empty(v.value + 1, dtype=torch.uint8, device="cuda") for v in n]
    out = torch.empty_like(x[0])
    t = L.OP_TENSORS(*[v.data_ptr() for v in x], *(None,) * 6, idx.data_ptr(), out.data_ptr())
    before = lib.nsa_launch_count()
    with pytest.raises(nsa.NsaError, match="token-major"):
        L.check(lib.nsa_attention_fwd_tokens(d, t, mem[0].data_ptr(), mem[1].data_ptr(), n[1].value, L.stream()))
    assert lib.nsa_launch_count() == before


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("c", [(3, 3001, 12, 4, 64), (2, 33, 3, 1, 8), (1, 7, 8, 2, 128), (1, 4097, 64, 4, 64)], ids=str)
def test_projection_rows(c, dtype):
    """Rows of the fused projection <-> heads, every element, on both sides of the line between one token and eight a thread;
    the padding behind the gates comes back as zeros."""
    B, T, Hq, Hkv, D = c
    L, lib = pkg()._lib, pkg().lib()
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    code = L.DTYPE_BF16 if dtype == "bf16" else L.DTYPE_F32
    W, n = lib.nsa_fused_projection_width(Hq, Hkv, D), (Hq + 6 * Hkv) * D
    y = torch.randn(B, T, W, device="cuda").to(dt)
    q, kv, gate = (torch.full(s, float("nan"), device="cuda", dtype=dt) for s in ((B, Hq, T, D), (6, B, Hkv, T, D), (B, Hq, T, 3)))
    L.check(lib.nsa_split_heads(y.data_ptr(), q.data_ptr(), kv.data_ptr(), gate.data_ptr(), B, T, Hq, Hkv, D, code, L.stream()))
    assert torch.equal(q, y[..., :Hq * D].view(B, T, Hq, D).transpose(1, 2))
    assert torch.equal(kv, y[..., Hq * D:n].view(B, T, 6, Hkv, D).permute(2, 0, 3, 1, 4))
    assert torch.equal(gate, y[..., n:n + 3 * Hq].view(B, T, Hq, 3).transpose(1, 2))
    back = torch.full_like(y, float("nan"))
    L.check(lib.nsa_merge_heads(q.data_ptr(), kv.data_ptr(), gate.data_ptr(), back.data_ptr(), B, T, Hq, Hkv, D, code, L.stream()))
    assert torch.equal(back[..., :n + 3 * Hq], y[..., :n + 3 * Hq]) and not back[..., n + 3 * Hq:].any()
