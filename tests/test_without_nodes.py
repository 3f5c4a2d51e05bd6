"""The package without its C++ autograd nodes, which have to be built against the torch that runs: the Python nodes
serve every call."""
import importlib
import subprocess
import warnings

import pytest
import torch

from tests.util import make_inputs, pkg


@pytest.fixture
def without(monkeypatch):
    L = pkg()._lib

    def go(path="/nonexistent/_nsa_torch.so"):
        monkeypatch.setattr(L, "_ext", None)
        monkeypatch.setattr(L, "EXT_PATH", path)
        return L
    return go


def test_one_warning_and_no_error(without, tmp_path):
    broken = tmp_path / "_nsa_torch.so"
    broken.write_bytes(b"not a library")
    for path, why in (("/nonexistent/_nsa_torch.so", "not been built"), (str(broken), "_nsa_torch.so")):
        L = without(path)
        with pytest.warns(RuntimeWarning, match=why):
            assert L.torch_op() is None
        with warnings.catch_warnings():
            warnings.simplefilter("error")
            assert L.torch_op() is None
            assert not pkg().ops.one_node_ok()


def test_other_torch(without, monkeypatch):
    L = without(pkg()._lib.EXT_PATH)
    importlib.import_module("openbox-llm_b200.build").build_library()
    assert L.torch_op().torch_version == torch.__version__
    L = without(L.EXT_PATH)
    monkeypatch.setattr(torch, "__version__", "0.1")
    with pytest.warns(RuntimeWarning, match="built against torch"):
        assert L.torch_op() is None


def test_library_builds_without_them(monkeypatch, tmp_path, capsys):
    b = importlib.import_module("openbox-llm_b200.build")
    monkeypatch.setattr(b, "EXT", str(tmp_path / "_nsa_torch.so"))
    monkeypatch.setattr(b, "_compile_ext", lambda: subprocess.CompletedProcess([], 1, "", "no compiler"))
    assert b.build_library() == b.LIB
    assert "no compiler" in capsys.readouterr().err


@pytest.mark.gpu
def test_the_python_nodes_serve_the_calls(without):
    t = make_inputs(dict(B=1, Hq=8, Hkv=2, D=64, T=200, block_size=64, S=3), torch.bfloat16, seed=5)
    nsa = pkg()
    layer = importlib.import_module("openbox-llm_b200.module").NSAAttentionB200(256, 4, 2, block_size=64, n_selected_blocks=2,
                                                                                window=40).cuda()
    x = torch.randn(1, 130, 256, device="cuda")

    def run():
        xs = [t[n].bfloat16().cuda().requires_grad_(True) for n in ("q", "kc", "vc", "ks", "vs", "kw", "vw", "gate")]
        out = nsa.nsa_attention(*xs, 64, 3, 70)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = layer(x)
        return out, y, torch.autograd.grad(out, xs, t["do"].bfloat16().cuda())
    want = run()
    without()
    with pytest.warns(RuntimeWarning):
        got = run()
    assert "LayerNode" in want[1].grad_fn.name() and "LayerNode" not in got[1].grad_fn.name()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    for a, b in zip(got[2], want[2]):
        assert (a.float() - b.float()).abs().max() <= 2.0 ** -7 * max(b.float().abs().max().item(), 0.1)
