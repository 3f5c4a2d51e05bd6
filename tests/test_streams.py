"""The whole-op call and its side streams: captures, callers' streams, threads."""
import ctypes
import importlib
import threading

import pytest
import torch

from tests.test_refused_calls import _inputs
from tests.util import pkg

pytestmark = pytest.mark.gpu


def _forward_call(ins, S=4, W=128, bs=64):
    """A forward through the C ABI on memory of its own: (launch(stream) -> return code, output)."""
    L = importlib.import_module("openbox-llm_b200._lib")
    q, k = ins[0], ins[1]
    B, Hq, T, D = q.shape
    desc = L.NsaAttentionDesc(L.dims(B, Hq, k.shape[1], T, D, L.DTYPE_BF16), bs, S, W, 0, 0, bs, bs, 0, 0, 0, 0, 0)
    n = [ctypes.c_size_t() for _ in range(3)]
    L.check(L.lib().nsa_attention_sizes(desc, *n))
    saved, ws = (torch.empty(x.value + 1, dtype=torch.uint8, device="cuda") for x in n[:2])
    idx = torch.empty(B, k.shape[1], T, S, dtype=torch.int32, device="cuda")
    out = torch.zeros_like(q)
    ptrs = L.OP_TENSORS(*[x.data_ptr() for x in ins], *(None,) * 6, idx.data_ptr(), out.data_ptr())
    keep = (saved, ws, idx)

    def launch(stream):
        return L.lib().nsa_attention_fwd(desc, ptrs, keep[0].data_ptr(), keep[1].data_ptr(), n[1], stream)

    return launch, out


def test_two_captures_open_in_one_thread():
    """A thread's side streams belong to one capture at a time: a call in another capture goes without them.  The
    thread is new, so its side streams are also made inside the first capture."""
    nsa = pkg()
    rt = ctypes.CDLL("libcudart.so.12")
    ins = [_inputs(1, 8, 2, 512, 64, seed=s) for s in (1, 2)]
    want = [nsa.nsa_attention(*x, 64, 4, 128) for x in ins]
    calls = [_forward_call(x) for x in ins]
    streams = [torch.cuda.Stream() for _ in ins]
    torch.cuda.synchronize()
    codes, graphs = [], [ctypes.c_void_p() for _ in ins]
    execs = [ctypes.c_void_p() for _ in ins]

    def body():
        torch.cuda.set_device(0)
        for s, (launch, _) in zip(streams, calls):
            codes.append(rt.cudaStreamBeginCapture(ctypes.c_void_p(s.cuda_stream), 1))   # thread-local mode
            codes.append(launch(s.cuda_stream))
        for s, g in zip(streams, graphs):
            codes.append(rt.cudaStreamEndCapture(ctypes.c_void_p(s.cuda_stream), ctypes.byref(g)))
        for g, e in zip(graphs, execs):
            codes.append(rt.cudaGraphInstantiateWithFlags(ctypes.byref(e), g, ctypes.c_ulonglong(0)))
        for s, e in zip(streams, execs):
            codes.append(rt.cudaGraphLaunch(e, ctypes.c_void_p(s.cuda_stream)))

    t = threading.Thread(target=body)
    t.start()
    t.join()
    assert codes == [0] * 10, codes
    torch.cuda.synchronize()
    for (_, out), w, g, e in zip(calls, want, graphs, execs):
        assert torch.equal(out, w)
        rt.cudaGraphExecDestroy(e)
        rt.cudaGraphDestroy(g)
    assert nsa.lib().nsa_device_status(None) == 0
