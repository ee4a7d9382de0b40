"""What a call that is cut along the keys must leave as an uncut call does: rows that no sequence owns, results after an
earlier call that failed, precision, key pages outside the window, workspaces sized for the plain form, loose bounds."""
import ctypes as C

import pytest
import torch

from flash_cuda_b200 import capi, ops, workloads as W
from oracle.ref_attention import ref_attention

pytestmark = pytest.mark.gpu

PARTS = dict(reqs=[(200, 9000)], hq=8, hkv=2, hd=128, page_size=64)             # key-range parts of the prefill kernel
MIXED = dict(reqs=[(1, 3000)] * 6 + [(200, 9000)], hq=8, hkv=2, hd=128, page_size=64)
DECODE = dict(reqs=[(1, 5000), (1, 300), (1, 2500)], hq=8, hkv=2, hd=128, page_size=64)
WIDEN = dict(reqs=[(1, 900), (200, 9000), (3, 65)], hq=8, hkv=2, hd=128, page_size=64, kv_dtype="fp8")


def _problem(spec, dev, **kw):
    spec = dict(spec, **kw)
    return W.make_problem("cut", spec.pop("reqs"), seed=301, **spec).to(dev)


@pytest.mark.parametrize("spec,kw", [(PARTS, {}), (MIXED, {}), (WIDEN, {}), (DECODE, {}), (DECODE, dict(num_splits=4)),
                                     (PARTS, dict(route=capi.FA_ROUTE_GENERAL, num_splits=3))],
                         ids=["parts", "mixed", "widened", "decode", "decode_split", "general_split"])
def test_rows_past_the_last_sequence_stay_as_they_are(spec, kw, cuda_device):
    """A batch padded for a captured graph: total_q is larger than cu_seqlens_q[batch]."""
    p = _problem(spec, cuda_device)
    n, pad = p.q.shape[0], 37
    q = torch.cat([p.q, p.q[:1].expand(pad, -1, -1)])
    out = torch.full((n + pad, *p.q.shape[1:]), 7.0, device=cuda_device, dtype=p.q.dtype)
    lse = torch.full((p.q.shape[1], n + pad), 7.0, device=cuda_device)
    capi.fwd(q, p.k, p.v, out=out, lse=lse, check=True, **dict(p.capi_kw(), **kw))
    tight, tight_lse, _ = capi.fwd(p.q, p.k, p.v, check=True, **dict(p.capi_kw(), **kw))
    assert (out[n:] == 7.0).all() and (lse[:, n:] == 7.0).all()
    # (the padding is part of total_q and may move the cuts: one rounding to 16 bits of values below 2)
    assert (out[:n].float() - tight.float()).abs().max().item() <= 2 ** -7
    torch.testing.assert_close(lse[:, :n], tight_lse, atol=1e-4, rtol=1e-5)


@pytest.mark.parametrize("failed", [False, True])
def test_decode_does_not_depend_on_what_an_earlier_call_left(failed, cuda_device):
    """Counters between byte 256 and 4095 are not zero: the caller keeps the first 256 bytes only, or a call whose
    waits ran out left them (its status word says so) and the caller goes on with the buffer."""
    p = _problem(DECODE, cuda_device)
    want, want_lse, ws = capi.fwd(p.q, p.k, p.v, check=True, **p.capi_kw())
    ws.zero_()
    ws[256:4096] = 1
    flags = capi.FA_FLAG_WORKSPACE_CLEAN
    if failed:
        ws.view(torch.int32)[0] = 1
        flags |= capi.FA_FLAG_WORKSPACE_CLEAN_4K
    out, lse = torch.zeros_like(want), torch.zeros_like(want_lse)
    capi.fwd(p.q, p.k, p.v, out=out, lse=lse, workspace=ws, flags=flags, **p.capi_kw())
    assert (out.float() - want.float()).abs().max().item() <= 2 ** -7      # (another cut: one rounding to 16 bits)
    torch.testing.assert_close(lse, want_lse, atol=1e-4, rtol=1e-5)


@pytest.mark.parametrize("reqs", [[(90, 1500)], [(90, 1500), (1, 700), (4, 300)]], ids=["chunk", "mixed"])
def test_softcap_over_an_e4m3_cache_keeps_the_exact_tanh(reqs, cuda_device):
    """More rows than the decode kernel takes: the LSE is as far from 64 bits as 32-bit sums and tanhf (2 ulp of values
    up to the cap, 30 * 2^-22) make it; the approximate tanh alone is off by up to 2^-11 of the cap, 0.015."""
    p = W.make_problem("cap", reqs, hq=8, hkv=2, hd=128, page_size=64, kv_dtype="fp8", softcap=30.0, seed=302)
    p.softmax_scale *= 12.0              # logits of the size of the cap
    pd = p.to(cuda_device)
    _, lse, _ = capi.fwd(pd.q, pd.k, pd.v, check=True, **pd.capi_kw())
    q0 = 0
    for b, (ql, kl) in enumerate(reqs):
        k = p.k[p.page_table[b].long()].flatten(0, 1)[:kl].double()
        seen = torch.arange(kl)[None] <= torch.arange(kl - ql, kl)[:, None]
        for h in range(8):
            s = p.q[q0:q0 + ql, h].double() @ k[:, h // 4].t() * p.k_descale[b, h // 4].double() * p.softmax_scale
            z = (30.0 * torch.tanh(s / 30.0)).masked_fill(~seen, -float("inf")).logsumexp(1)
            assert (lse[h, q0:q0 + ql].cpu().double() - z).abs().max().item() <= 1e-4
        q0 += ql


@pytest.mark.parametrize("page_size", [16, 64])
def test_pages_that_no_row_sees_need_no_entry(page_size, cuda_device):
    """A serving program gives pages back that have left the window; their entries may then hold anything."""
    reqs, window, leftpad = [(90, 3000), (1, 700), (100, 1111)], 500, [0, 3, 900]
    p = _problem(dict(reqs=reqs, hq=8, hkv=2, hd=128, page_size=page_size, kv_dtype="fp8", window_left=window,
                      leftpad=leftpad), cuda_device)
    want, want_lse, _ = capi.fwd(p.q, p.k, p.v, check=True, **p.capi_kw())
    for b, (ql, kl) in enumerate(reqs):
        first = max(kl - ql - window, leftpad[b])              # the first key that a row sees
        p.page_table[b, :first // page_size] = -1
    out, lse, _ = capi.fwd(p.q, p.k, p.v, check=True, **p.capi_kw())
    assert torch.equal(out, want) and torch.equal(lse, want_lse)


@pytest.mark.parametrize("spec", [PARTS, MIXED, WIDEN, DECODE], ids=["parts", "mixed", "widened", "decode"])
def test_a_workspace_for_the_plain_form_is_enough(spec, cuda_device):
    """What only makes a call faster is left out where the workspace has no room for it."""
    p = _problem(spec, cuda_device)
    want, want_lse, _ = capi.fwd(p.q, p.k, p.v, check=True, **p.capi_kw())
    lib = capi.load()
    out, lse = torch.zeros_like(want), torch.zeros_like(want_lse)
    fp, keep = capi.make_params(p.q, p.k, p.v, out, lse, **p.capi_kw())
    # header, one work list of 16-byte entries per kernel, and the split partials that num_splits = 0 stands for
    splits = lib.fa_b200_num_splits(C.byref(fp))
    rows = p.q.shape[0] * p.q.shape[1]
    need = 256 + 2 * 4096 + (0 if splits == 1 else splits * rows * (p.v.shape[-1] + 1) * 4 + 512)
    assert lib.fa_b200_fwd_workspace_bytes(C.byref(fp)) > need
    ws = torch.full((need + (1 << 20),), 7, device=cuda_device, dtype=torch.uint8)
    rc = lib.fa_b200_fwd(C.byref(fp), ws.data_ptr(), need, torch.cuda.current_stream().cuda_stream)
    assert rc == capi.FA_OK, rc
    capi.check_status(ws)
    assert (ws[need:] == 7).all()
    tol = 2 ** -6 if spec is WIDEN else 2 ** -7       # one rounding of the result; over e4m3 also of P in another kernel
    assert (out.float() - want.float()).abs().max().item() <= tol
    torch.testing.assert_close(lse, want_lse, atol=1e-3, rtol=1e-4)
    del keep
    assert lib.fa_b200_fwd(C.byref(fp), ws.data_ptr(), 128, torch.cuda.current_stream().cuda_stream) == capi.FA_ERR_WORKSPACE


def test_the_op_runs_without_memory_for_its_scratch(cuda_device):
    """The memory limit of the allocator leaves no room for the partial results of a prefill in parts (16 MB here)."""
    p = _problem(dict(PARTS, reqs=[(500, 16000)], hq=32, hkv=8), cuda_device)
    out = torch.empty_like(p.q)
    want, _ = ops.call_fwd(p.q, p.k, p.v, num_splits=1, **p.capi_kw())
    fp, keep = capi.make_params(p.q, p.k, p.v, out, torch.empty(32, 500, device=cuda_device), **p.capi_kw())
    scratch = capi.load().fa_b200_fwd_workspace_bytes(C.byref(fp))
    assert scratch > 12 << 20
    stream = torch.cuda.Stream()         # (its workspace is not there yet)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(cuda_device).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (8 << 20)) / total)
    try:
        with torch.cuda.stream(stream):
            got, _ = ops.call_fwd(p.q, p.k, p.v, out=out, **p.capi_kw())
        torch.cuda.synchronize()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(got, want)
    del keep


@pytest.mark.parametrize("kw", [{}, dict(sink=True, window_left=300), dict(hd=192, hdv=128), dict(hd=256)],
                         ids=["plain", "sink_window", "hd192", "hd256"])
def test_few_keys_under_a_loose_bound_are_not_cut(kw, cuda_device):
    """max_seqlen_k may be any upper bound: 400 keys in a table for 131072 give the bits of the uncut call."""
    p = _problem(dict(PARTS, reqs=[(150, 300), (129, 400)]), cuda_device, **kw)
    args = dict(p.capi_kw(), max_seqlen_k=131072)
    pool = torch.zeros(2048 - p.k.shape[0], *p.k.shape[1:], device=cuda_device, dtype=p.k.dtype)     # (a pool of 131072 keys)
    k, v = torch.cat([p.k, pool]), torch.cat([p.v, pool[..., :p.v.shape[-1]]])
    out, lse, _ = capi.fwd(p.q, k, v, check=True, **args)
    whole, whole_lse, _ = capi.fwd(p.q, k, v, check=True, num_splits=1, **args)
    assert torch.equal(out, whole) and torch.equal(lse, whole_lse)


def test_few_rows_over_few_keys_of_an_e4m3_cache_stay_on_the_general_kernel(cuda_device):
    """At head_dim 64 a widened copy of the cache costs more than it saves there."""
    for ql, kl in ((1, 3000), (8, 1000), (50, 4096)):
        p = _problem(dict(reqs=[(ql, kl)], hq=8, hkv=2, hd=64, page_size=64, kv_dtype="fp8"), cuda_device)
        out, lse, _ = capi.fwd(p.q, p.k, p.v, check=True, **p.capi_kw())
        gen, gen_lse, _ = capi.fwd(p.q, p.k, p.v, check=True, route=capi.FA_ROUTE_GENERAL, **p.capi_kw())
        assert torch.equal(out, gen) and torch.equal(lse, gen_lse)


def test_a_sequence_that_does_not_fit_the_slabs_leaves_them_to_the_others(cuda_device):
    """The first of two sequences has more keys than 256 MB of slabs hold (65536 at 8 kv heads of 2 x 128 columns): it
    gets the general kernel's bits, the second one the tensor-core kernel's."""
    g = torch.Generator(device=cuda_device).manual_seed(303)
    lens, q_lens = [66000, 900], [17, 100]
    pages = [(n + 63) // 64 for n in lens]
    k, v = (torch.randn(sum(pages), 64, 8, 128, generator=g, device=cuda_device, dtype=torch.bfloat16).to(torch.float8_e4m3fn)
            for _ in range(2))
    table = torch.zeros(2, max(pages), dtype=torch.int32)
    table[0, :pages[0]] = torch.arange(pages[0], dtype=torch.int32)
    table[1, :pages[1]] = torch.arange(pages[0], sum(pages), dtype=torch.int32)
    q = torch.randn(117, 32, 128, generator=g, device=cuda_device, dtype=torch.bfloat16)
    kw = dict(cu_seqlens_q=torch.tensor([0, 17, 117], dtype=torch.int32, device=cuda_device), page_table=table.to(cuda_device),
              seqused_k=torch.tensor(lens, dtype=torch.int32, device=cuda_device), max_seqlen_q=100, max_seqlen_k=66000,
              softmax_scale=128 ** -0.5, causal=True)
    out, _, _ = capi.fwd(q, k, v, check=True, **kw)
    gen, _, _ = capi.fwd(q, k, v, check=True, route=capi.FA_ROUTE_GENERAL, num_splits=1, **kw)
    assert torch.equal(out[:17], gen[:17]) and not torch.equal(out[17:], gen[17:])
    assert (out[17:].float() - gen[17:].float()).abs().max().item() <= 2 ** -6
