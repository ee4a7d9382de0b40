"""Decode calls of more than 16 packed rows that take 32 rows at a time (long passes only: the host decides from the longest
sequence it is told of, so a loose bound stands in for long ones), against the CPU oracle with the benchmark's tolerances (2e-2,
LSE 5e-3 and 1e-2), and against the same call under a tight bound with one pass per sequence, which goes 16 rows at a time: an
output differs by one rounding to 16 bits of |values| < 4 and by the rounding of P against another maximum."""
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


def _list(d, kw, bound=LONG):
    return capi.get_scheduler_metadata(
        d.q.device, batch=d.cu_seqlens_q.numel() - 1, max_seqlen_q=kw["max_seqlen_q"], max_seqlen_k=bound, hq=d.q.shape[1], hkv=d.k.shape[-2],
        hd=d.q.shape[2], hdv=d.v.shape[-1], dtype=d.q.dtype, seqused_k=kw["seqused_k"], cu_seqlens_q=kw["cu_seqlens_q"],
        leftpad_k=kw.get("leftpad_k"), page_size=d.k.shape[1], causal=kw["causal"], window_left=kw["window_left"],
        window_right=kw["window_right"], has_softcap=False, num_splits=kw.get("num_splits", 0))


@pytest.mark.parametrize("hd,hdv,dtype", HEADS)
@pytest.mark.parametrize("window", [-1, 40])
@pytest.mark.parametrize("q_len", [5, 12, 16])
@pytest.mark.parametrize("copies", [1, 30])        # 6 sequences, or more entries than the records of a small line
def test_callers_list(copies, q_len, window, hd, hdv, dtype, cuda_device):
    """A list made by the caller has an entry for every 16 rows, which the pass of 32 joins: as a line that the kernel cuts, and as work
    items."""
    reqs = [(q_len, 400), (1, 200), (0, 100), (q_len, 0), (5, 129), (q_len, 64)] * copies
    p = W.make_problem("two", reqs, hq=4, hkv=1, hd=hd, hdv=hdv, dtype=dtype, page_size=16, seed=504, window_left=window)
    d = p.to(cuda_device)
    want, want_lse = ref_attention(p.q, p.k, p.v, **p.oracle_kw())
    fin = torch.isfinite(want_lse)
    for splits in (0, 1):
        kw = dict(d.capi_kw(), max_seqlen_k=LONG, num_splits=splits)
        out, lse, _ = capi.fwd(d.q, d.k, d.v, check=True, **kw, scheduler_metadata=_list(d, kw))
        assert (out.float().cpu() - want).abs().max().item() <= 2e-2
        assert torch.equal(torch.isfinite(lse.cpu()), fin)
        torch.testing.assert_close(lse.cpu()[fin], want_lse[fin], atol=5e-3, rtol=1e-2)


@pytest.mark.parametrize("splits", [0, 1])
@pytest.mark.parametrize("tile", [0, 1])
def test_callers_list_is_checked(tile, splits, cuda_device):
    """A key range outside the sequence is an error in the entry of either tile, also in the one that is passed over."""
    p = W.make_problem("two", [(6, 500)], hq=8, hkv=2, hd=128, hdv=128, dtype="bf16", page_size=16, seed=505)
    d = p.to(cuda_device)
    kw = dict(d.capi_kw(), max_seqlen_k=LONG, num_splits=splits)
    md = _list(d, kw)
    capi.fwd(d.q, d.k, d.v, check=True, **kw, scheduler_metadata=md)
    host = md.cpu()
    entry = next(e for e in range(2) if host[16 + 4 * e + 1] == tile)
    md[16 + 4 * entry + 3] = 1000
    with pytest.raises(capi.FaError):
        capi.fwd(d.q, d.k, d.v, check=True, **kw, scheduler_metadata=md)
