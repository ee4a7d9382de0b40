"""Softcap on the tensor-core prefill route: blocks whose scores stay below the cap take tanh as a polynomial, others the
special-function unit's, decided block by block."""
import pytest
import torch

from flash_cuda_b200 import capi, workloads as W
from oracle.ref_attention import ref_attention

pytestmark = pytest.mark.gpu
CAP = 30.0
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


@pytest.mark.parametrize("hd,hdv,dtype", [(128, 128, "bf16"), (128, 128, "fp16"), (64, 64, "bf16"), (192, 128, "bf16")])
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
