"""The torch-op boundary from Python: loads `fa_b200_torch.so`, which registers `fwd` and
`get_scheduler_metadata` with the reference's schemas (kernels/fa4_blackwell.cu:10187-10205), and mirrors
the reference harness' caller `call_fwd` (bench/scenarios.py:932-940).

There is no eager/PyTorch implementation behind these functions: if the extension cannot be loaded they raise.
"""
from __future__ import annotations

import importlib.util
import os
import warnings

import torch

from . import build as _build

NAMESPACE = "_vllm_fa3_C"
_loaded = False
_direct = None      # `fwd` of torch_direct.cpp, where it is built


def _load_direct(build_if_missing: bool):
    """`fwd` of torch_direct.cpp, or None with a warning: the op does all it does, some 4 us later per call."""
    try:
        if build_if_missing and not os.path.isfile(_build.DIRECT_SO):
            _build.build_direct()
        if not _build.direct_is_current():
            raise ImportError("it is missing, or was built from other sources, or for another Python or torch")
        spec = importlib.util.spec_from_file_location("fa_b200_direct", _build.DIRECT_SO)
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
        return module.fwd
    except (ImportError, OSError, RuntimeError) as e:
        warnings.warn(f"flash_cuda_b200: {_build.DIRECT_SO} is not used ({e}); call_fwd goes through the dispatcher")
        return None


def load(build_if_missing: bool = True):
    """Loads the op library (idempotent) and returns `torch.ops.<NAMESPACE>`."""
    global _loaded, _direct
    if not _loaded:
        if not (os.path.isfile(_build.TORCH_SO) and os.path.isfile(_build.CAPI_SO)):
            if not build_if_missing:
                raise RuntimeError("flash_cuda_b200 extension is not built; run `python -m flash_cuda_b200.build`")
            _build.build_all()
        torch.ops.load_library(_build.TORCH_SO)
        _direct = _load_direct(build_if_missing)
        _loaded = True
    ns = getattr(torch.ops, NAMESPACE)
    if getattr(ns, "fwd", None) is None:
        raise RuntimeError(f"torch.ops.{NAMESPACE}.fwd is not registered")
    return ns


def fwd(*args):
    """`torch.ops._vllm_fa3_C.fwd(*args)` with the 37 positional arguments of the schema.
    Returns [out, softmax_lse, empty, empty]."""
    return load().fwd(*args)


def get_scheduler_metadata(*args):
    return load().get_scheduler_metadata(*args)


def call_fwd(q, k, v, *, cu_seqlens_q, max_seqlen_q, max_seqlen_k, softmax_scale, causal, cu_seqlens_k=None,
             seqused_k=None, page_table=None, leftpad_k=None, q_descale=None, k_descale=None, v_descale=None,
             window_left=-1, window_right=-1, softcap=0.0, s_aux=None, num_splits=0, scheduler_metadata=None,
             out=None, sm_margin=0):
    """Keyword front end that places everything in the schema's positional order; returns (out, lse).

    Calls on plain CUDA tensors, with no mode, transform, trace or profiler active, skip the dispatcher (same
    implementation, same results); all others go through the op."""
    if not _loaded:
        load()
    if _direct is not None and not torch.compiler.is_compiling():
        res = _direct(q, k, v, out, cu_seqlens_q, cu_seqlens_k, seqused_k, max_seqlen_q, max_seqlen_k, page_table, leftpad_k,
                      q_descale, k_descale, v_descale, softmax_scale, causal, window_left, window_right, softcap,
                      scheduler_metadata, num_splits, sm_margin, s_aux)
        if res is not None:
            return res
    res = fwd(q, k, v, None, None, None, out, cu_seqlens_q, cu_seqlens_k, None, None, seqused_k,
              int(max_seqlen_q), int(max_seqlen_k), page_table, None, leftpad_k, None, None, None,
              q_descale, k_descale, v_descale, float(softmax_scale), bool(causal), int(window_left),
              int(window_right), float(softcap), True, scheduler_metadata, int(num_splits), None, int(sm_margin),
              s_aux, 1, 0, None)
    return res[0], res[1]
