"""The work whose speed this framework answers for, as calls of its public entry points.

Every case is one attention forward through `flash_cuda_b200.ops.call_fwd`, the torch op's keyword front end, on
inputs that a serving or training program has on the GPU already.  Lengths and leftpads are part of the case (drawn
from its `lens_seed`), so that the work of a case is known without its inputs; tensor values come from the seed.
Queries, keys and values are N(0, 1), the softmax scale is head_dim ** -0.5, pages are a random permutation of the
pool: the distributions of this repository's benchmark configurations.
"""
from __future__ import annotations

import math
import random

import torch

from flash_cuda_b200 import ops

_DT = {"bf16": torch.bfloat16, "fp16": torch.float16, "e4m3": torch.float8_e4m3fn}
_DEV = "cuda"


def _case(name, kind, **kw):
    base = dict(name=name, kind=kind, batch=1, q_lo=1, q_hi=1, k_lo=0, k_hi=0, chunks=0, chunk_lo=0, chunk_hi=0,
                hq=32, hkv=8, hd=128, hdv=128, dtype="bf16", kv="same", page=0, causal=True, window=-1, softcap=0.0,
                sink=False, leftpad=False, metadata=False, lens_seed=0)
    assert set(kw) <= set(base)
    base.update(kw)
    return base


def listed():
    return [
        # One user at a prompt of about a thousand tokens: the smallest decode step, all latency.  Pages of 16 keys.
        _case("decode_one", "decode", batch=1, k_lo=1000, k_hi=1000, page=16),
        # A server's ordinary decode step: a few sequences of very different age.
        _case("decode_ragged", "decode", batch=16, k_lo=1024, k_hi=16384, page=64, lens_seed=1),
        # The paged-decode benchmark configuration: batch 128, contexts uniform in [1024, 32768], pages of 64 keys,
        # leftpad; the scheduler metadata is computed once per step and shared by the layers, as serving programs do.
        _case("decode_batch", "decode", batch=128, k_lo=1024, k_hi=32768, page=64, leftpad=True, metadata=True,
              lens_seed=2),
        # Decode over an e4m3 cache with one descale per (batch, kv head).
        _case("decode_e4m3_cache", "decode", batch=48, k_lo=1024, k_hi=16384, page=64, kv="e4m3", leftpad=True,
              lens_seed=3),
        # Verification of four speculated tokens: head_dim 64, 64 / 8 heads, sink logits, fp16.
        _case("verify_sink_hd64", "decode", batch=24, q_lo=4, q_hi=4, k_lo=500, k_hi=8000, page=16, hq=64, hkv=8, hd=64,
              hdv=64, dtype="fp16", sink=True, lens_seed=4),
        # The smallest benchmark configuration: dense non-causal MHA, B=2 H=8 S=512 (an encoder, a short prompt).
        _case("dense_small", "prefill", batch=2, q_lo=512, q_hi=512, hq=8, hkv=8, causal=False),
        # The headline configuration: causal GQA prefill, B=4 S=4096.
        _case("causal_gqa", "prefill", batch=4, q_lo=4096, q_hi=4096),
        # The packed varlen configuration: 16 sequences of 128 .. 8192, window 4096, softcap 30, sinks.
        _case("varlen_window_cap_sink", "prefill", batch=16, q_lo=128, q_hi=8192, window=4096, softcap=30.0, sink=True,
              lens_seed=5),
        # The all-e4m3 variant of the causal configuration.
        _case("causal_e4m3", "prefill", batch=2, q_lo=4096, q_hi=4096, dtype="e4m3", kv="e4m3"),
        # Chunked prefill of one long prompt: 512 new tokens against everything before them, pages of 64 keys.
        _case("chunk_paged", "chunk", batch=1, q_lo=512, q_hi=512, k_lo=24500, k_hi=24500, page=64),
        # A continuous-batching step over an e4m3 cache: most sequences decode one token, one prefills a chunk.
        _case("mixed_e4m3_cache", "mixed", batch=33, k_lo=512, k_hi=8192, chunks=1, chunk_lo=1000, chunk_hi=1000, page=16,
              kv="e4m3", lens_seed=6),
        # A slice of the long-context configuration: head_dim 192 / 128, MHA, a chunk against a long paged context.
        _case("long_hd192", "chunk", batch=1, q_lo=2048, q_hi=2048, k_lo=32768, k_hi=32768, hq=16, hkv=16, hd=192,
              page=64),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def _cost(case):
    w = work(case)
    return max(w["bytes"] / 6.6e12, w["flops"] / 1.6e15)


def draw(rng):
    """One more case of the ranges above: the kind first, then its sizes and options."""
    limit = 0.9 * max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["decode", "decode", "verify", "prefill", "prefill", "varlen", "chunk", "mixed"])
        hq, hkv = rng.choice([(32, 8), (32, 8), (16, 16), (64, 8), (28, 4), (8, 1)])
        hd, hdv = rng.choice([(128, 128), (128, 128), (128, 128), (64, 64), (192, 128)])
        kw = dict(hq=hq, hkv=hkv, hd=hd, hdv=hdv, dtype=rng.choice(["bf16", "bf16", "fp16"]),
                  lens_seed=rng.randrange(1 << 30))
        if kind in ("decode", "verify", "mixed") or (kind == "chunk" and hd == 128):
            kw["kv"] = rng.choice(["same", "same", "e4m3"]) if hd == 128 else "same"
        page = rng.choice([16, 16, 32, 64, 128])
        if kind in ("decode", "verify"):
            lo = _log_int(rng, 64, 8192)
            kw.update(batch=_log_int(rng, 1, 128), k_lo=lo, k_hi=_log_int(rng, lo, 32768), page=page,
                      leftpad=rng.random() < 0.25, metadata=kw["kv"] == "same" and rng.random() < 0.3)
            if kind == "verify":
                n = rng.randint(2, max(2, 64 // (hq // hkv)))
                kw.update(q_lo=n, q_hi=n, sink=rng.random() < 0.5)
            kind = "decode"
        elif kind == "prefill":
            n = _log_int(rng, 128, 8192)
            kw.update(batch=_log_int(rng, 1, 8), q_lo=n, q_hi=n, causal=rng.random() < 0.75)
            if hd == 128 and rng.random() < 0.25:
                kw.update(dtype="e4m3", kv="e4m3")
        elif kind == "varlen":
            lo = _log_int(rng, 64, 1024)
            kw.update(batch=_log_int(rng, 2, 16), q_lo=lo, q_hi=_log_int(rng, lo, 8192), sink=rng.random() < 0.5,
                      window=rng.choice([-1, 1024, 4096]), softcap=rng.choice([0.0, 30.0]))
            kind = "prefill"
        elif kind == "chunk":
            n = _log_int(rng, 100, 2048)
            k = _log_int(rng, n, 65536)
            kw.update(batch=_log_int(rng, 1, 3), q_lo=n, q_hi=n, k_lo=k, k_hi=k, page=page)
        else:
            lo = _log_int(rng, 128, 4096)
            n = _log_int(rng, 100, 2048)
            kw.update(batch=_log_int(rng, 4, 64), k_lo=lo, k_hi=_log_int(rng, lo, 16384), chunks=rng.randint(1, 3),
                      chunk_lo=n, chunk_hi=n, page=page)
        case = _case("", kind, **kw)
        del case["name"]
        if 5e-7 <= _cost(case) <= limit:
            return case


def _lengths(case):
    """(query length, key length, leftpad) of every sequence."""
    rng = random.Random(case["lens_seed"])
    seqs = []
    for i in range(case["batch"]):
        if case["kind"] == "mixed" and i >= case["batch"] - case["chunks"]:
            ql = rng.randint(case["chunk_lo"], case["chunk_hi"])
            kl = ql + rng.randint(0, case["k_hi"])
        else:
            ql = rng.randint(case["q_lo"], case["q_hi"])
            kl = ql if case["kind"] == "prefill" else max(ql, rng.randint(case["k_lo"], case["k_hi"]))
        pad = min(rng.randint(0, 63), kl - ql) if case["leftpad"] else 0
        seqs.append((ql, kl, pad))
    return seqs


def _esz(name):
    return 1 if name == "e4m3" else 2


def work(case):
    hd, hdv, hq, hkv = case["hd"], case["hdv"], case["hq"], case["hkv"]
    kv = case["dtype"] if case["kv"] == "same" else case["kv"]
    nbytes = pairs = 0
    for ql, kl, pad in _lengths(case):
        nbytes += ql * hq * (hd * _esz(case["dtype"]) + hdv * 2 + 4)
        wl = case["window"]
        lo0 = pad if wl < 0 else max(pad, kl - ql - wl)
        nbytes += (kl - lo0) * hkv * (hd + hdv) * _esz(kv)
        if not case["causal"]:
            pairs += ql * (kl - pad)
        else:                                  # query i sees keys max(pad, p - window) .. p, p = kl - ql + i
            for p in (range(kl - ql, kl) if wl >= 0 else ()):
                pairs += max(0, p - max(pad, p - wl) + 1)
            if wl < 0:
                pairs += ql * (kl - ql - pad) + ql * (ql + 1) // 2
    return {"bytes": nbytes, "flops": 2 * (hd + hdv) * hq * pairs}


def _randn(shape, gen):
    return torch.randn(shape, generator=gen, device=_DEV, dtype=torch.bfloat16)


def _to_e4m3(x):
    """Per-kv-head quantisation of a (..., heads, dim) tensor: values and (heads,) descales, in slices of the pool."""
    d = (x.abs().flatten(0, -3).amax(dim=(0, -1)).float() / 448.0).clamp_min(1e-8)
    out = torch.empty(x.shape, device=_DEV, dtype=torch.float8_e4m3fn)
    step = max(1, (1 << 26) // max(1, x[0].numel()))
    for i in range(0, x.shape[0], step):
        out[i:i + step] = (x[i:i + step].float() / d.view(-1, 1)).to(torch.float8_e4m3fn)
    return out, d


def _ints(values):
    return torch.tensor(values, dtype=torch.int32, device=_DEV)


def _cumulative(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return _ints(cu)


def prepare(case, seed):
    seqs = _lengths(case)
    gen = torch.Generator(device=_DEV).manual_seed(seed)
    B, hq, hkv, hd, hdv, page = (case[n] for n in ("batch", "hq", "hkv", "hd", "hdv", "page"))
    q_lens, k_lens = [s[0] for s in seqs], [s[1] for s in seqs]
    kv = case["dtype"] if case["kv"] == "same" else case["kv"]
    kw = dict(cu_seqlens_q=_cumulative(q_lens), max_seqlen_q=max(q_lens), max_seqlen_k=max(k_lens),
              softmax_scale=hd ** -0.5, causal=case["causal"], softcap=case["softcap"])
    if case["window"] >= 0:
        kw.update(window_left=case["window"], window_right=0)
    if page:
        need = [(n + page - 1) // page for n in k_lens]
        pool = sum(need) + 5
        perm = torch.randperm(pool, generator=torch.Generator().manual_seed(seed)).to(torch.int32).tolist()
        width, at, table = max(need), 0, []
        for n in need:
            table.append(perm[at:at + n] + [0] * (width - n))
            at += n
        kw.update(page_table=_ints(table), seqused_k=_ints(k_lens))
        k_shape, v_shape = (pool, page, hkv, hd), (pool, page, hkv, hdv)
    else:
        kw["cu_seqlens_k"] = _cumulative(k_lens)
        k_shape, v_shape = (sum(k_lens), hkv, hd), (sum(k_lens), hkv, hdv)
    q = _randn((sum(q_lens), hq, hd), gen)
    k, v = _randn(k_shape, gen), _randn(v_shape, gen)
    if kv == "e4m3":
        k, kd = _to_e4m3(k)
        v, vd = _to_e4m3(v)
        if case["dtype"] == "e4m3":            # one descale per kv head for all sequences
            q, qd = _to_e4m3(q.unflatten(1, (hkv, hq // hkv)).flatten(2))
            q = q.unflatten(2, (hq // hkv, hd)).flatten(1, 2)
            kw["q_descale"] = qd.expand(B, hkv).contiguous()
        kw["k_descale"], kw["v_descale"] = kd.expand(B, hkv).contiguous(), vd.expand(B, hkv).contiguous()
    else:
        k, v = k.to(_DT[kv]), v.to(_DT[kv])
    if case["dtype"] != "e4m3":
        q = q.to(_DT[case["dtype"]])
    if case["sink"]:
        kw["s_aux"] = torch.randn(hq, generator=gen, device=_DEV)
    if case["leftpad"]:
        kw["leftpad_k"] = _ints([s[2] for s in seqs])
    if case["metadata"]:
        kw["scheduler_metadata"] = ops.get_scheduler_metadata(
            B, max(q_lens), max(k_lens), hq, hkv, hd, hdv, _DT[kv], kw["seqused_k"], kw["cu_seqlens_q"], None, None, None,
            kw.get("leftpad_k"), page, 0, case["causal"], -1, -1, False, 0, None, 0)
    return dict(q=q, k=k, v=v, kw=kw)


def run(state):
    return ops.call_fwd(state["q"], state["k"], state["v"], **state["kw"])


def tolerance(case):
    if case["dtype"] == "e4m3":
        return {"rel": 3e-2, "max": 0.9}     # probabilities and values are e4m3: 2^-4 per term, averaged over the keys
    if case["dtype"] == "fp16":
        return {"rel": 2e-3, "max": 3e-2}
    return {"rel": 1e-2, "max": 1.5e-1}


def exact(case, seed):
    """Attention in 64 bits on the inputs of `prepare`, one (sequence, kv head) at a time."""
    state = prepare(case, seed)
    seqs, kw = _lengths(case), state["kw"]
    hq, hkv, page = case["hq"], case["hkv"], case["page"]
    rep = hq // hkv
    total = sum(s[0] for s in seqs)
    out = torch.empty(total, hq, case["hdv"], device=_DEV, dtype=torch.float64)
    lse = torch.empty(hq, total, device=_DEV, dtype=torch.float64)
    q0 = k0 = 0
    for b, (ql, kl, pad) in enumerate(seqs):
        if page:
            rows = kw["page_table"][b, :(kl + page - 1) // page].long()
            kb, vb = (state[n][rows].flatten(0, 1)[:kl] for n in ("k", "v"))
        else:
            kb, vb = state["k"][k0:k0 + kl], state["v"][k0:k0 + kl]
        pos = torch.arange(kl - ql, kl, device=_DEV)
        keys = torch.arange(kl, device=_DEV)
        seen = (keys >= pad).expand(ql, kl)
        if case["causal"]:
            seen = seen & (keys <= pos[:, None])
        if case["window"] >= 0:
            seen = seen & (keys >= pos[:, None] - case["window"])
        for h in range(hkv):
            kh, vh = kb[:, h].float().double(), vb[:, h].float().double()
            if "v_descale" in kw:
                vh *= kw["v_descale"][b, h].double()
            for r in range(rep):
                head = h * rep + r
                s = state["q"][q0:q0 + ql, head].float().double() @ kh.t()
                s *= kw["softmax_scale"]
                for n in ("q_descale", "k_descale"):
                    if n in kw:
                        s *= kw[n][b, h].double()
                if case["softcap"] > 0:
                    s = torch.tanh(s / case["softcap"]) * case["softcap"]
                s.masked_fill_(~seen, -math.inf)
                z = torch.logsumexp(s, dim=1)
                if case["sink"]:
                    z = torch.logaddexp(z, kw["s_aux"][head].double())
                out[q0:q0 + ql, head] = s.sub_(z[:, None]).exp_() @ vh
                lse[head, q0:q0 + ql] = z
        q0 += ql
        k0 += kl
    return out, lse
