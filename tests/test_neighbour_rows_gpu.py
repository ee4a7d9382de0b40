"""Rows that no key of a sequence lies in.  The decode kernel fetches 64 keys at a time; what it fetches for a sequence whose keys
end there are its own rows only, whatever its neighbours in memory hold."""
import pytest
import torch

from flash_cuda_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu
FORMS = [(64, None), (128, None), (192, None), (128, "fp8")]


def _run(p, dev, **kw):
    d = p.to(dev)
    out, lse, _ = capi.fwd(d.q, d.k, d.v, check=True, route=capi.FA_ROUTE_DECODE, **dict(d.capi_kw(), **kw))
    return out, lse


@pytest.mark.parametrize("hd,kv_dtype", FORMS)
@pytest.mark.parametrize("num_splits", [0, 1, 3])
def test_next_sequence_of_a_packed_cache(num_splits, hd, kv_dtype, cuda_device):
    """Every second sequence is all NaN; the others are an odd number of 64-key blocks and give the bits they give without it."""
    lens = [64, 70, 192, 5, 320, 64, 960, 1, 4160, 33]
    p = W.make_problem("rows", [(1, n) for n in lens], hq=8, hkv=4, hd=hd, hdv=min(hd, 128), kv_dtype=kv_dtype, seed=451)
    want = _run(p, cuda_device, num_splits=num_splits)
    at = 0
    for i, n in enumerate(lens):
        if i % 2:
            p.k[at:at + n] = float("nan")
            p.v[at:at + n] = float("nan")
        at += n
    got = _run(p, cuda_device, num_splits=num_splits)
    for i in range(0, len(lens), 2):
        assert torch.equal(got[0][i], want[0][i]) and torch.equal(got[1][:, i], want[1][:, i])


@pytest.mark.parametrize("hd,kv_dtype", FORMS)
@pytest.mark.parametrize("page_size", [1, 2, 4, 8, 16, 32])
def test_first_page_of_the_pool(page_size, hd, kv_dtype, cuda_device):
    """Page 0 belongs to nobody and is all NaN, as are the table's unused entries' pages; sequences end with a page."""
    lens = [page_size * n for n in (1, 3, 31)] + [64, 128 - page_size, 192, 1000 // page_size * page_size, 4160]
    p = W.make_problem("rows", [(1, n) for n in lens], hq=8, hkv=4, hd=hd, hdv=min(hd, 128), kv_dtype=kv_dtype, page_size=page_size, seed=452)
    want = _run(p, cuda_device)
    p.k, p.v = (torch.cat([torch.full_like(x[:1].float(), float("nan")).to(x.dtype), x]) for x in (p.k, p.v))
    p.page_table += 1
    for i, n in enumerate(lens):
        p.page_table[i, (n + page_size - 1) // page_size:] = 0
    got = _run(p, cuda_device)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
