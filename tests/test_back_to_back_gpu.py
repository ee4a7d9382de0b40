"""Kernels that start while their predecessor in the stream ends still see what it wrote: calls back to back, their inputs
rewritten in the stream between them, give the bits of calls that nothing runs beside."""
import pytest
import torch

from flash_cuda_b200 import ops, workloads as W

pytestmark = pytest.mark.gpu

PROBLEMS = {   # one kernel each, and the sequences of kernels that the routes launch
    "decode": ([(1, 1000)], dict(hq=8, hkv=8, hd=128, page_size=16)),
    "decode_list": ([(1, 300 + 40 * i) for i in range(60)], dict(hq=16, hkv=16, hd=64, page_size=32)),
    "prefill": ([(256, 256), (100, 100)], dict(hq=8, hkv=8, hd=128, causal=False)),
    "parts": ([(300, 9000)], dict(hq=8, hkv=2, hd=128, page_size=64)),
    "mixed": ([(1, 3000)] * 6 + [(200, 9000)], dict(hq=8, hkv=2, hd=128, page_size=64)),
    "widened": ([(1, 900), (200, 3000), (3, 65)], dict(hq=8, hkv=2, hd=128, page_size=16, kv_dtype="fp8")),
}


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("name", sorted(PROBLEMS))
def test_inputs_rewritten_between_calls(name, graph, cuda_device):
    reqs, kw = PROBLEMS[name]
    ps = [W.make_problem("stream", reqs, seed=430 + i, **kw).to(cuda_device) for i in range(3)]
    want = []
    for p in ps:
        out, lse = ops.call_fwd(p.q, p.k, p.v, **p.capi_kw())
        torch.cuda.synchronize()
        want.append((out.clone(), lse.clone()))
    cur = W.make_problem("stream", reqs, seed=430, **kw).to(cuda_device)
    call = cur.capi_kw()

    def step(p):
        cur.q.copy_(p.q); cur.k.copy_(p.k); cur.v.copy_(p.v)
        for n, v in p.capi_kw().items():
            if isinstance(v, torch.Tensor):
                call[n].copy_(v)
        first = ops.call_fwd(cur.q, cur.k, cur.v, **call)
        return first, ops.call_fwd(cur.q, cur.k, cur.v, **call)

    got = []
    if graph:
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            step(ps[0])
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            got = [step(ps[i % 3]) for i in range(6)]
        g.replay()
        g.replay()
    else:
        got = [step(ps[i % 3]) for i in range(6)]
    torch.cuda.synchronize()
    for i, results in enumerate(got):
        for out, lse in results:
            assert torch.equal(out, want[i % 3][0]) and torch.equal(lse, want[i % 3][1])
