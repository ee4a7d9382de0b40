"""Where the decode kernel rounds its weights.  P goes to the tensor cores in 16 bits, relative to the running maximum of 16 keys
of a warp (of 32 over an e4m3 cache): a weight that is such a maximum is exact, so longer groups cost accuracy, and nothing else
shows it."""
import math

import pytest
import torch

from flash_cuda_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu
WARPS, BLOCK = 4, 64


def _rounded(s, v, dtype, group):
    """Attention of one row in 64 bits, but for the rounding of the weights; `s` in log2 units.  Warp w of four takes keys
    [group w, group (w + 1)) of every run of 4 x `group` keys, with a running maximum that moves group by group."""
    m = torch.full((WARPS,), -math.inf, dtype=torch.float32)
    l, o = torch.zeros(WARPS, dtype=torch.float64), torch.zeros(WARPS, v.shape[1], dtype=torch.float64)
    for k0 in range(0, len(s), group):
        w = k0 // group % WARPS
        x = s[k0:k0 + group]
        top = torch.maximum(m[w], x.max())
        p = torch.exp2(x - top)
        corr = torch.exp2((m[w] - top).double())
        l[w] = l[w] * corr + p.double().sum()
        o[w] = o[w] * corr + p.to(dtype).double() @ v[k0:k0 + group]
        m[w] = top
    e = torch.exp2((m - m.max()).double())
    return (e[:, None] * o).sum(0) / (e * l).sum()


@pytest.mark.parametrize("keys", [64, 100, 192, 1000, 3001])
@pytest.mark.parametrize("hd,dtype", [(64, "bf16"), (128, "bf16"), (128, "fp16"), (192, "bf16")])
@pytest.mark.parametrize("page_size", [0, 1, 16, 64])
def test_weights_are_rounded_against_the_maximum_of_sixteen_keys(keys, hd, dtype, page_size, cuda_device):
    """fp32 output, one pass: beside the rounding of P there are fp32 sums and exp2, relative errors of some 2^-20 of a weight.  They
    move one weight in 2^12 (bf16; fp16: 2^9) across a rounding border; groups of 32 keys round about half of all weights otherwise."""
    p = W.make_problem("rounding", [(1, keys)], hq=8, hkv=2, hd=hd, hdv=min(hd, 128), dtype=dtype, page_size=page_size, seed=440)
    d = p.to(cuda_device)
    out = torch.empty(1, 8, min(hd, 128), dtype=torch.float32, device=cuda_device)
    capi.fwd(d.q, d.k, d.v, out=out, check=True, num_splits=1, route=capi.FA_ROUTE_DECODE, **d.capi_kw())
    rows = p.page_table[0].long() if page_size else slice(None)
    k, v = ((x[rows].flatten(0, 1) if page_size else x)[:keys].double() for x in (p.k, p.v))
    off = {16: 0.0, 32: 0.0}
    for h in range(8):
        s = ((p.q[0, h].double() @ k[:, h // 4].T) * p.softmax_scale * math.log2(math.e)).float()
        for group in off:
            off[group] += (out[0, h].cpu().double() - _rounded(s, v[:, h // 4], p.q.dtype, group)).norm().item() ** 2
    assert off[16] ** 0.5 <= off[32] ** 0.5 / 2
