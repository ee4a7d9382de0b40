"""The op's scratch under stream capture.  A graph may run before, after and beside other graphs and calls of the stream it was
captured on, whatever ran there when it was captured."""
import pytest
import torch

from flash_cuda_b200 import ops, workloads as W

pytestmark = pytest.mark.gpu

PROBLEMS = {   # one that keeps tickets in its scratch, one that keeps arrival counters and pieces, key-range parts, a widened cache
    "list": ([(1, 300 + 40 * i) for i in range(60)], dict(hq=16, hkv=16, hd=64, page_size=32)),
    "pieces": ([(1, 9000), (1, 40)], dict(hq=8, hkv=2, hd=128, page_size=16)),
    "parts": ([(300, 9000)], dict(hq=8, hkv=2, hd=128, page_size=64)),
    "widened": ([(1, 900), (200, 3000), (3, 65)], dict(hq=8, hkv=2, hd=128, page_size=16, kv_dtype="fp8")),
}


def _problem(name, seed, dev):
    reqs, kw = PROBLEMS[name]
    p = W.make_problem("capture", reqs, seed=seed, **kw).to(dev)
    want = ops.call_fwd(p.q, p.k, p.v, **p.capi_kw())      # (on the current stream: kernels are loaded, the capture stream is new)
    torch.cuda.synchronize()
    return p, want


def _capture(p, stream, calls=2):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        got = [ops.call_fwd(p.q, p.k, p.v, **p.capi_kw()) for _ in range(calls)]
    return g, got


def _check(got, want):
    for out, lse in got:
        assert torch.equal(out, want[0]) and torch.equal(lse, want[1])


def _dirty(dev, stream):
    """Whatever memory is free for the taking holds no zeros."""
    with torch.cuda.stream(stream):
        for n in (1 << 20, 2 << 20, 9 << 20, 1 << 20):
            torch.full((n,), 0x5a, dtype=torch.uint8, device=dev)
    torch.cuda.synchronize()


@pytest.mark.parametrize("name", sorted(PROBLEMS))
def test_second_graph_of_a_stream_runs_first(name, cuda_device):
    stream = torch.cuda.Stream()
    _dirty(cuda_device, stream)
    (pa, wa), (pb, wb) = (_problem(name, s, cuda_device) for s in (461, 462))
    ga, a = _capture(pa, stream)
    gb, b = _capture(pb, stream)
    for g, got, want in ((gb, b, wb), (ga, a, wa), (gb, b, wb)):
        g.replay()
        torch.cuda.synchronize()
        _check(got, want)


@pytest.mark.parametrize("name", sorted(PROBLEMS))
def test_larger_call_between_capture_and_replay(name, cuda_device):
    stream = torch.cuda.Stream()
    p, want = _problem(name, 463, cuda_device)
    g, got = _capture(p, stream)
    big = W.make_problem("big", [(200, 9000)], hq=32, hkv=8, hd=128, page_size=64, seed=464).to(cuda_device)
    with torch.cuda.stream(stream):
        ops.call_fwd(big.q, big.k, big.v, **big.capi_kw())
    torch.cuda.synchronize()
    held = [torch.full((1 << 20,), 0x5a, dtype=torch.uint8, device=cuda_device) for _ in range(8)]
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        _check(got, want)
    assert all(bool((h == 0x5a).all()) for h in held)


@pytest.mark.parametrize("name", sorted(PROBLEMS))
def test_graphs_of_one_stream_run_beside_each_other(name, cuda_device):
    capture, streams = torch.cuda.Stream(), [torch.cuda.Stream() for _ in range(3)]
    problems = [_problem(name, 465 + i, cuda_device) for i in range(3)]
    graphs = [_capture(p, capture) for p, _ in problems]
    for _ in range(20):
        for (g, _), s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        with torch.cuda.stream(capture):
            ops.call_fwd(problems[0][0].q, problems[0][0].k, problems[0][0].v, **problems[0][0].capi_kw())
    torch.cuda.synchronize()
    for (_, got), (_, want) in zip(graphs, problems):
        _check(got, want)


def test_capture_of_two_streams(cuda_device):
    """One graph, two branches: each has its own scratch."""
    (pa, wa), (pb, wb) = (_problem("pieces", s, cuda_device) for s in (468, 469))
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=main):
        side.wait_stream(main)
        a = [ops.call_fwd(pa.q, pa.k, pa.v, **pa.capi_kw()) for _ in range(3)]
        with torch.cuda.stream(side):
            b = [ops.call_fwd(pb.q, pb.k, pb.v, **pb.capi_kw()) for _ in range(3)]
        main.wait_stream(side)
    for _ in range(20):
        g.replay()
    torch.cuda.synchronize()
    _check(a, wa)
    _check(b, wb)
