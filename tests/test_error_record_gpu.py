"""A launch that the runtime refuses is reported by the call that asked for it, and by nobody else: the runtime's own record of the
last error, which the next launch of whoever shares the thread looks at, is clear again."""
import ctypes

import pytest
import torch

from flash_cuda_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu
RELAXED, NON_BLOCKING = 2, 1

PROBLEMS = {
    "decode": ([(1, 1000)], dict(hq=8, hkv=8, hd=128, page_size=16)),
    "prefill": ([(256, 256)], dict(hq=8, hkv=8, hd=128)),
    "general": ([(40, 40)], dict(hq=2, hkv=2, hd=80)),
}


@pytest.mark.parametrize("name", sorted(PROBLEMS))
def test_refused_launch(name, cuda_device):
    """On a stream whose capture a synchronisation has broken off, every launch is refused on the host."""
    lib, cudart = capi.load(), ctypes.CDLL("libcudart.so.12")
    reqs, kw = PROBLEMS[name]
    p = W.make_problem("refused", reqs, seed=471, **kw).to(cuda_device)
    out, lse, ws = capi.fwd(p.q, p.k, p.v, check=True, **p.capi_kw())
    want = out.clone()
    params, keep = capi.make_params(p.q, p.k, p.v, out, lse, **p.capi_kw())
    params.flags = 3          # (the header is clean: the first thing that the call does is a launch)
    stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert cudart.cudaStreamCreateWithFlags(ctypes.byref(stream), NON_BLOCKING) == 0
    try:
        assert cudart.cudaStreamBeginCapture(stream, RELAXED) == 0
        assert lib.fa_b200_check_status(ws.data_ptr(), stream, None) == capi.FA_ERR_LAUNCH
        assert cudart.cudaPeekAtLastError() == 0
        assert lib.fa_b200_fwd(ctypes.byref(params), ws.data_ptr(), ws.numel(), stream) == capi.FA_ERR_LAUNCH
        assert b"kernel" in lib.fa_b200_last_cuda_error()
        assert cudart.cudaPeekAtLastError() == 0
    finally:
        cudart.cudaStreamEndCapture(stream, ctypes.byref(graph))
        cudart.cudaGetLastError()
        cudart.cudaStreamDestroy(stream)
    out, lse, _ = capi.fwd(p.q, p.k, p.v, check=True, **p.capi_kw())
    assert torch.equal(out, want)
    del keep
