"""Decode calls of more than 16 packed rows that take 32 rows at a time (long passes only: the host decides from the longest
sequence it is told of, so a loose bound stands in for long ones), against the CPU oracle with the benchmark's tolerances (2e-2,
LSE 5e-3 and 1e-2), and against the same call with a work list, which goes 16 rows at a time: an output differs by one rounding
to 16 bits of |values| < 4 and by the rounding of P against another maximum."""
import pytest
import torch

from flash_cuda_b200 import capi, workloads as W
from oracle.ref_attention import ref_attention

pytestmark = pytest.mark.gpu
LONG = 1 << 21       # bound on the keys per sequence


def _run(p, dev, **kw):
    d = p.to(dev)
    out, lse, _ = capi.fwd(d.q, d.k, d.v, check=True, **dict(d.capi_kw(), max_seqlen_k=LONG, **kw))
    return out.float().cpu(), lse.cpu()


def _check(p, dev, **kw):
    out, lse = _run(p, dev, **kw)
    want, want_lse = ref_attention(p.q, p.k, p.v, **p.oracle_kw())
    assert (out - want).abs().max().item() <= 2e-2, p.name
    fin = torch.isfinite(want_lse)
    assert torch.equal(torch.isfinite(lse), fin), p.name
    torch.testing.assert_close(lse[fin], want_lse[fin], atol=5e-3, rtol=1e-2)


HEADS = [(64, 64, "fp16"), (128, 128, "bf16"), (192, 128, "bf16")]


@pytest.mark.parametrize("hd,hdv,dtype", HEADS)
@pytest.mark.parametrize("q_len", [5, 8, 9, 12, 13, 16])       # x 4 heads: 20, 32, 36, 48, 52, 64 rows
@pytest.mark.parametrize("page", [0, 1, 16, 64])
def test_rows(page, q_len, hd, hdv, dtype, cuda_device):
    """Ragged keys around the borders of blocks (64) and stages (128), a sequence of one row, one without rows, one without keys."""
    reqs = [(q_len, k) for k in (q_len, 63, 64, 129, 400)] + [(1, 200), (0, 100), (q_len, 0), (5, 300)]
    p = W.make_problem("two", reqs, hq=8, hkv=2, hd=hd, hdv=hdv, dtype=dtype, page_size=page, seed=501)
    _check(p, cuda_device)
    _check(p, cuda_device, num_splits=1)         # work items instead of one line


@pytest.mark.parametrize("hd,hdv,dtype", HEADS)
@pytest.mark.parametrize("kw", [dict(window_left=100), dict(window_left=90, window_right=3, causal=False), dict(softcap=20.0, sink=True),
                                dict(leftpad=[60, 290, 0])], ids=["window", "two_sided", "cap_sink", "leftpad"])
def test_options(kw, hd, hdv, dtype, cuda_device):
    p = W.make_problem("two", [(11, 700), (3, 333), (7, 90)], hq=14, hkv=2, hd=hd, hdv=hdv, dtype=dtype, page_size=32, seed=502, **kw)
    _check(p, cuda_device)


@pytest.mark.parametrize("hd,hdv,dtype", HEADS)
def test_pieces_and_lists(hd, hdv, dtype, cuda_device):
    """One long sequence among short ones: cut into more pieces than are merged in one trip, and the same bits every time."""
    p = W.make_problem("two", [(6, 12000), (6, 50), (2, 900)], hq=16, hkv=2, hd=hd, hdv=hdv, dtype=dtype, page_size=64, seed=503)
    d = p.to(cuda_device)
    kw = dict(d.capi_kw(), max_seqlen_k=LONG)
    out, lse, _ = capi.fwd(d.q, d.k, d.v, check=True, **kw)
    again, again_lse, _ = capi.fwd(d.q, d.k, d.v, check=True, **kw)
    assert torch.equal(out, again) and torch.equal(lse, again_lse)
    _check(p, cuda_device)
    one, one_lse, _ = capi.fwd(d.q, d.k, d.v, check=True, **dict(kw, max_seqlen_k=12000, num_splits=1))
    assert (out.float() - one.float()).abs().max().item() <= 2 ** -6 + 2 ** -8
    torch.testing.assert_close(lse, one_lse, atol=1e-4, rtol=1e-5)
