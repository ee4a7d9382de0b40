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
    "depaged": ([(600, 600), (300, 500)], dict(hq=8, hkv=2, hd=128, page_size=8)),
    "splits": ([(1, 3000), (2, 700)], dict(hq=8, hkv=2, hd=128, page_size=64)),
    "all_e4m3": ([(300, 300), (100, 100)], dict(hq=4, hkv=2, hd=128, dtype="fp8")),
    "widened": ([(1, 900), (200, 3000), (3, 65)], dict(hq=8, hkv=2, hd=128, page_size=16, kv_dtype="fp8")),
}


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("name", sorted(PROBLEMS))
def test_inputs_rewritten_between_calls(name, graph, cuda_device):
    reqs, kw = PROBLEMS[name]
    extra = dict(num_splits=4) if name == "splits" else {}
    ps = [W.make_problem("stream", reqs, seed=430 + i, **kw).to(cuda_device) for i in range(3)]
    want = []
    for p in ps:
        out, lse = ops.call_fwd(p.q, p.k, p.v, **p.capi_kw(), **extra)
        torch.cuda.synchronize()
        want.append((out.clone(), lse.clone()))
    cur = W.make_problem("stream", reqs, seed=430, **kw).to(cuda_device)
    call = dict(cur.capi_kw(), **extra)

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


@pytest.mark.parametrize("graph", [False, True])
def test_work_list_made_and_used_at_once(graph, cuda_device):
    """Lengths and pages are rewritten, the list is made from them and the call that reads it follows: `get_scheduler_metadata` and
    `fwd` back to back, as a serving step without shared lists has them."""
    lens = [300 + 40 * i for i in range(60)]
    kw = dict(hq=16, hkv=16, hd=64, page_size=32)
    ps = [W.make_problem("list", [(1, n) for n in lens[9 * i:] + lens[:9 * i]], seed=440 + i, **kw).to(cuda_device) for i in range(3)]

    def listed(d, kw):
        return ops.get_scheduler_metadata(len(lens), 1, max(lens), 16, 16, 64, 64, d.q.dtype, kw["seqused_k"], kw["cu_seqlens_q"], None,
                                          None, None, None, 32, 0, True, -1, -1, False, 0, None, 0)

    want = []
    for p in ps:
        md = listed(p, p.capi_kw())
        torch.cuda.synchronize()
        out, lse = ops.call_fwd(p.q, p.k, p.v, scheduler_metadata=md, **p.capi_kw())
        torch.cuda.synchronize()
        want.append((out.clone(), lse.clone()))
    cur = W.make_problem("list", [(1, n) for n in lens], seed=440, **kw).to(cuda_device)
    call = cur.capi_kw()

    def step(p):
        cur.q.copy_(p.q); cur.k.copy_(p.k); cur.v.copy_(p.v)
        for n, v in p.capi_kw().items():
            if isinstance(v, torch.Tensor):
                call[n].copy_(v)
        return ops.call_fwd(cur.q, cur.k, cur.v, scheduler_metadata=listed(cur, call), **call)

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
    for i, (out, lse) in enumerate(got):
        assert torch.equal(out, want[i % 3][0]) and torch.equal(lse, want[i % 3][1])
