"""Softcap on the tensor-core prefill route: blocks whose scores stay below the cap take tanh as a polynomial, others the
special-function unit's, decided block by block."""
import pytest
import torch

from flash_cuda_b200 import capi, workloads as W
from oracle.ref_attention import ref_attention

pytestmark = pytest.mark.gpu
CAP = 30.0
SHAPES = [(128, 128, "bf16"), (128, 128, "fp16"), (64, 64, "bf16"), (192, 128, "bf16"), (192, 192, "bf16"), (256, 256, "fp16")]
TANH = 4.9e-4        # relative error of the coarser of the two forms (tanh.approx.f32: 2^-11)


def _run(p, dev):
    d = p.to(dev)
    out, lse, _ = capi.fwd(d.q, d.k, d.v, check=True, route=capi.FA_ROUTE_PREFILL_TC, **d.capi_kw())
    return out.float().cpu(), lse.cpu()


def _check(p, dev, largest):
    """A logit is off by TANH of its size at most, so is the LSE; a weight by twice that and the rounding of P (2^-8 in
    bf16); an output is a mean of values under such weights, rounded to 16 bits."""
    out, lse = _run(p, dev)
    want, want_lse = ref_attention(p.q, p.k, p.v, **p.oracle_kw())
    d = TANH * min(CAP, largest)
    assert (lse - want_lse).abs().max().item() <= d + 1e-4
    assert (out - want).abs().max().item() <= (2 * d + 2 ** -8 + 2 ** -8) * p.v.float().abs().max().item()


@pytest.mark.parametrize("hd,hdv,dtype", SHAPES)
@pytest.mark.parametrize("size", [1.0, 6.0, 40.0], ids=["far_below_the_cap", "around_it", "far_above"])
def test_scores_of_every_size(size, hd, hdv, dtype, cuda_device):
    p = W.make_problem("cap", [(129, 1281), (300, 300), (1, 1025)], hq=4, hkv=2, hd=hd, hdv=hdv, dtype=dtype, softcap=CAP, seed=401)
    p.softmax_scale *= size
    _check(p, cuda_device, 6.0 * size)


@pytest.mark.parametrize("first", [0, 1, 3], ids=["from_the_start", "from_block_1", "from_block_3"])
@pytest.mark.parametrize("window", [-1, 300])
def test_scores_that_pass_the_cap_late(first, window, cuda_device):
    """Keys from block `first` on are forty times as large: the item begins in one form and ends in the other."""
    p = W.make_problem("cap", [(256, 1000)], hq=4, hkv=2, hd=128, softcap=CAP, window_left=window, seed=402)
    p.k[128 * first:] *= 40.0
    _check(p, cuda_device, 240.0)


def test_scores_that_are_all_far_below_their_reference(cuda_device):
    """Large negative logits beside small ones, in and out of the polynomial's range, and a zero scale."""
    p = W.make_problem("cap", [(256, 900)], hq=4, hkv=2, hd=128, softcap=CAP, seed=403)
    p.q[:, :, 0] = 16.0
    p.k[:, :, 0] = torch.where(torch.arange(900)[:, None] % 3 == 0, -15.0, 0.0).to(p.k.dtype)
    _check(p, cuda_device, 30.0)
    p.softmax_scale = 0.0
    _check(p, cuda_device, 0.0)


def test_a_nan_query_stays_in_its_row(cuda_device):
    """(The rows beside it may take the other form of tanh: twice its error, on logits below 6.)"""
    p = W.make_problem("cap", [(256, 900)], hq=4, hkv=2, hd=128, softcap=CAP, seed=404)
    out, lse = _run(p, cuda_device)
    p.q[100] = float("nan")
    out_n, lse_n = _run(p, cuda_device)
    keep, d = torch.arange(256) != 100, 2 * TANH * 6.0
    assert out_n[100].isnan().all()
    assert (lse_n - lse)[:, keep].abs().max().item() <= d + 1e-4
    assert (out_n - out)[keep].abs().max().item() <= (2 * d + 2 ** -8 + 2 ** -8) * p.v.float().abs().max().item()


@pytest.mark.parametrize("hd,hdv,dtype", SHAPES)
@pytest.mark.parametrize("sign", [1, -1])
def test_polynomial_is_as_exact_as_it_says(sign, hd, hdv, dtype, cuda_device):
    """Every row has one score s for all keys, 0 .. 0.6 of the cap (-4 .. 0: further down the bound by |s| leaves the fast form), except
    that the first block, which always takes the special-function unit's tanh, has 0.7 s (1.3 s for s < 0): its weight is
    128 e^(-0.3 |s|) in 8192.  So the LSE shows the error of tanh at s itself: 2.2e-6 of 18 at most, 1.3e-5 of the first block's
    (4.9e-4 x 1.3 |s| x its weight), and fp32 sums of 65 blocks and exp2, some 1.5e-5.  tanh.approx would be off by up to 8.8e-3."""
    keys, first = 8320, 128
    p = W.make_problem("cap", [(256, keys)], hq=2, hkv=1, hd=hd, hdv=hdv, dtype=dtype, softcap=CAP, causal=False, seed=405)
    p.softmax_scale = 1.0
    p.q.zero_()
    p.k.zero_()
    p.q[:, :, 0] = torch.linspace(0.0, 17.9 if sign > 0 else -4.0, 512).reshape(256, 2).to(p.q.dtype)
    p.k[:, :, 0] = 1.0
    p.k[:first, :, 0] = 0.7 if sign > 0 else 1.3
    d = p.to(cuda_device)
    _, lse, _ = capi.fwd(d.q, d.k, d.v, check=True, route=capi.FA_ROUTE_PREFILL_TC, num_splits=1, **d.capi_kw())
    s = p.q[:, :, 0].double().T
    y = torch.stack([CAP * torch.tanh(s * p.k[i, 0, 0].double() / CAP) for i in (0, keys - 1)])
    want = torch.logsumexp(y + torch.tensor([first, keys - first]).double().log()[:, None, None], dim=0)
    assert (lse.cpu().double() - want).abs().max().item() <= 2.2e-6 * 18 + 1.3e-5 + 1.5e-5


@pytest.mark.parametrize("hd,hdv,dtype", [(128, 128, "bf16"), (64, 64, "fp16"), (192, 192, "bf16")])
@pytest.mark.parametrize("cap", [1e-30, 1e-9, 1e-6, 1e-3, 1e4, 1e10, 1e20, 1e30])
def test_caps_out_of_proportion(cap, hd, hdv, dtype, cuda_device):
    """Caps for which the polynomial's coefficients, up to (scale / cap)^6, leave fp32's range.  The first tile's scores are all exactly 0,
    which lies in the polynomial's range under any cap."""
    p = W.make_problem("cap", [(200, 900)], hq=2, hkv=1, hd=hd, hdv=hdv, dtype=dtype, softcap=cap, causal=False, seed=406)
    p.q[:128] = 0.0
    _check(p, cuda_device, 6.0)
