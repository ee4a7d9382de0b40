"""`call_fwd` skips the dispatcher for plain calls only: what it takes gives the op's bits, everything else goes through the op."""
import pytest
import torch
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

from flash_cuda_b200 import ops, workloads as W

pytestmark = pytest.mark.gpu

PROBLEMS = {
    "decode": ([(1, 700), (1, 90)], dict(hq=8, hkv=2, hd=128, page_size=16, sink=True, leftpad=[3, 0])),
    "prefill": ([(200, 200), (65, 65)], dict(hq=4, hkv=4, hd=64, dtype="fp16", window_left=100, softcap=20.0)),
    "e4m3": ([(130, 130)], dict(hq=4, hkv=2, hd=128, dtype="fp8")),
}


def _args(pd, **over):
    kw = dict(dict(cu_seqlens_k=None, seqused_k=None, page_table=None, leftpad_k=None, q_descale=None, k_descale=None, v_descale=None,
                   window_left=-1, window_right=-1, softcap=0.0, s_aux=None, num_splits=0, scheduler_metadata=None, out=None,
                   sm_margin=0), **pd.capi_kw())
    kw.update(over)
    names = ("out", "cu_seqlens_q", "cu_seqlens_k", "seqused_k", "max_seqlen_q", "max_seqlen_k", "page_table", "leftpad_k",
             "q_descale", "k_descale", "v_descale", "softmax_scale", "causal", "window_left", "window_right", "softcap",
             "scheduler_metadata", "num_splits", "sm_margin", "s_aux")
    return [kw.get("q", pd.q), kw.get("k", pd.k), kw.get("v", pd.v)] + [kw[n] for n in names]


@pytest.fixture(scope="module")
def problem(cuda_device):
    ops.load()
    return W.make_problem("direct", *PROBLEMS["decode"][:1], seed=421, **PROBLEMS["decode"][1]).to(cuda_device)


@pytest.mark.parametrize("name", sorted(PROBLEMS))
@pytest.mark.parametrize("form", ["plain", "out", "inference_mode", "no_grad"])
def test_same_bits_as_the_op(name, form, cuda_device, monkeypatch):
    ops.load()
    pd = W.make_problem("direct", PROBLEMS[name][0], seed=422, **PROBLEMS[name][1]).to(cuda_device)
    kw = pd.capi_kw()
    if form == "out":
        kw["out"] = torch.empty(pd.q.shape[0], pd.q.shape[1], pd.v.shape[-1], device=cuda_device,
                                dtype=torch.bfloat16 if name == "e4m3" else pd.q.dtype)
    q = pd.q.clone().requires_grad_() if form == "no_grad" and name != "e4m3" else pd.q
    with torch.inference_mode(form == "inference_mode"), torch.set_grad_enabled(form != "no_grad"):
        direct = ops._direct(*_args(pd, q=q, out=kw.get("out")))
        assert direct is not None
        direct = [x.clone() for x in direct]
        got = [x.clone() for x in ops.call_fwd(q, pd.k, pd.v, **kw)]
        monkeypatch.setattr(ops, "_direct", None)
        want = ops.call_fwd(q, pd.k, pd.v, **kw)
    for a, b, c in zip(direct, got, want):
        assert torch.equal(a, c) and torch.equal(b, c) and a.dtype == c.dtype and a.shape == c.shape and a.stride() == c.stride()
    if form == "out":
        assert want[0].data_ptr() == kw["out"].data_ptr()


class _Sub(torch.Tensor):
    pass


class _Dispatch(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class _Function(TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def test_what_it_declines(problem, cuda_device):
    p, declined = problem, lambda **over: ops._direct(*_args(p, **over)) is None
    assert not declined()
    assert declined(q=p.q.as_subclass(_Sub)) and declined(q=p.q.clone().requires_grad_()) and declined(k=p.k.cpu())
    assert declined(max_seqlen_q=1.0) and declined(softmax_scale=1) and declined(causal=1) and declined(num_splits=1 << 70)
    with _Dispatch():
        assert declined()
    with _Function():
        assert declined()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]):
        assert declined()
    with torch.autograd.forward_ad.dual_level():
        assert declined(q=torch.autograd.forward_ad.make_dual(p.q, torch.ones_like(p.q)))
    seen = []
    torch.vmap(lambda x: seen.append(declined(q=x)) or x)(p.q[None])
    torch.func.functionalize(lambda x: seen.append(declined(q=x)) or x)(p.q)
    torch.jit.trace(lambda x: (seen.append(declined(q=x)), x + 0)[1], (p.q,), check_trace=False)
    assert seen and all(seen)
    assert not declined()


def test_a_refusal_is_still_an_error(problem):
    with pytest.raises(RuntimeError, match="unsupported"):
        ops.call_fwd(problem.q[None], problem.k, problem.v, **problem.capi_kw())
    with pytest.raises(RuntimeError, match="seqused_k"):
        ops.call_fwd(problem.q, problem.k, problem.v, **dict(problem.capi_kw(), seqused_k=None))


def test_numbers_of_other_types_are_converted_as_before(problem):
    kw = problem.capi_kw()
    want = ops.call_fwd(problem.q, problem.k, problem.v, **kw)
    got = ops.call_fwd(problem.q, problem.k, problem.v, **dict(kw, max_seqlen_q=torch.tensor(kw["max_seqlen_q"]), causal=1))
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])
