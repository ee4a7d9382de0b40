"""Balanced decode at the limits of its set-up and merge: lines of about as many entries as keep their records in shared
memory (160), pieces of about as many as one thread merges at once (8), row counts that do not divide, stages that end
inside a piece."""
import pytest

from flash_cuda_b200 import capi, workloads as W
from oracle.ref_attention import ref_attention

pytestmark = pytest.mark.gpu


def _check(p, dev, tol=2e-2):
    """Against the oracle (the benchmark's tolerances) and the uncut form (one rounding to 16 bits of values below 2)."""
    d = p.to(dev)
    out, lse, _ = capi.fwd(d.q, d.k, d.v, check=True, **d.capi_kw())
    whole, whole_lse, _ = capi.fwd(d.q, d.k, d.v, check=True, **dict(d.capi_kw(), num_splits=1))
    want, want_lse = ref_attention(p.q, p.k, p.v, **p.oracle_kw())
    assert (out.float().cpu() - want).abs().max().item() <= tol
    assert (lse.cpu() - want_lse).abs().max().item() <= 5e-3
    assert (out.float() - whole.float()).abs().max().item() <= 2 ** -7
    assert (lse - whole_lse).abs().max().item() <= 1e-4


@pytest.mark.parametrize("entries", [1, 31, 33, 80, 159, 160, 161, 200])
def test_entries_of_a_line(entries, cuda_device):
    reqs = [(1, 64 + 211 * i % 900) for i in range(entries - 1)] + [(1, 9000)]
    _check(W.make_problem("line", reqs, hq=4, hkv=1, hd=64, page_size=16, seed=411), cuda_device)


@pytest.mark.parametrize("keys", [1000, 1025, 1100, 2200, 9100])
@pytest.mark.parametrize("hd,kv_dtype", [(64, None), (128, None), (192, None), (128, "fp8")])
def test_pieces_of_one_sequence(keys, hd, kv_dtype, cuda_device):
    p = W.make_problem("pieces", [(1, keys)], hq=8, hkv=8, hd=hd, hdv=min(hd, 128), page_size=64, kv_dtype=kv_dtype, seed=412, sink=True)
    _check(p, cuda_device, 6e-2 if kv_dtype else 2e-2)


@pytest.mark.parametrize("rep,q_len", [(1, 1), (3, 5), (5, 3), (7, 2), (13, 4), (16, 1), (17, 3)])
@pytest.mark.parametrize("kv_dtype", [None, "fp8"])
def test_rows_of_a_tile(rep, q_len, kv_dtype, cuda_device):
    p = W.make_problem("rows", [(q_len, 3001), (1, 191), (q_len, 65)], hq=2 * rep, hkv=2, hd=128, page_size=32, kv_dtype=kv_dtype, seed=413)
    _check(p, cuda_device, 6e-2 if kv_dtype else 2e-2)
