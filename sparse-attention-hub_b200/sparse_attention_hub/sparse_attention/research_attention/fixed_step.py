"""Decode calls over bands and an exact top-k, through one native entry.

The stacks of sink and local-window maskers, alone or followed by an oracle top-k, need no mask
object between the maskers: the bands are numbers, and the top-k writes one bitmap that the
attention plan reads.  `fixed_step` hands such a call to `host/sah_step.cpp`, which launches the
kernels that the maskers and the attention step would (`sah_fixed_step_run`), for the same output (bit for bit,
but for bands alone over more than 32768 bfloat16 keys: they need no list and take the mma.sync kernel, where the
general path's list may take the tcgen05 one).  It returns None wherever the general path has to say or do something else: other
maskers or subclasses of these, sizes that select every key, tensors that are not plain CUDA tensors
of one dtype, rows whose selection is faster with a scratch buffer.
"""

from __future__ import annotations

import ctypes
import importlib.util
import warnings
from functools import lru_cache
from typing import List, Optional

import torch

from ... import _native
from ..utils import mask_attention_utils
from ..utils.mask import words_per_row
from .maskers.fixed.implementations.basic_fixed import LocalMasker, SinkMasker
from .maskers.fixed.implementations.oracle_top_k import OracleTopK

_MAX_BANDS = 6       # SAH_STEP_MAX_BANDS

#: the maskers that it serves, in some orders, and their `add_mask`, which it does the work of; their subclasses
#: are not among them
SERVED = {kind: kind.add_mask for kind in (SinkMasker, LocalMasker, OracleTopK)}
SERVED_ATTRIBUTES = 2  # of an instance: the configuration and the size; any other may stand in for a method

_module = None  # False: it cannot be loaded


def _step_module():
    """The native entry, or False (and a warning, once) where it is missing or made for another torch: the general
    path then serves its calls."""
    global _module
    if _module is None:
        path = _native.LIB_PATH.with_name("_sah_step.so")
        if not path.exists():
            path = _native.DEFAULT_LIB_DIR / "_sah_step.so"
        try:
            if not path.exists():
                raise ImportError(f"{path} is missing")
            spec = importlib.util.spec_from_file_location("_sah_step", path)
            module = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(module)
            if module.torch_version != torch.__version__.split("+")[0]:
                raise ImportError(f"{path} was made for torch {module.torch_version}")
        except ImportError as error:
            warnings.warn(f"decode calls take the slower general path: {error}; run "
                          "sparse-attention-hub_b200/build.py", RuntimeWarning, stacklevel=2)
            _module = False
            return _module
        lib = _native.load()
        module.bind(*(ctypes.cast(f, ctypes.c_void_p).value
                      for f in (lib.sah_fixed_step_plan, lib.sah_fixed_step_run, lib.sah_stream_capture)))
        _module = module
    return _module


@lru_cache(maxsize=1024)
def _select_fits(dtype: torch.dtype, rows: int, S: int) -> int:
    code = {torch.float32: _native.SAH_F32, torch.bfloat16: _native.SAH_BF16}.get(dtype)
    return 0 if code is None else _native.load().sah_topk_select_fits(code, rows, S, words_per_row(S))


def fixed_step(maskers: List, queries: torch.Tensor, keys: torch.Tensor, values: torch.Tensor,
               attention_mask: Optional[torch.Tensor], sinks: Optional[torch.Tensor],
               scaling: float) -> Optional[torch.Tensor]:
    """`[B, Sq, Hq, D]`, or None when the call is not one that the native entry serves."""
    if not maskers or type(queries) is not torch.Tensor or queries.dim() != 4 or not queries.is_cuda:
        return None
    if type(keys) is not torch.Tensor or keys.dim() != 4:
        return None
    Sq, S = queries.shape[2], keys.shape[2]
    # what sah_fixed_step_plan refuses for its key count, without the way there (57 -> 64 us of a call of four
    # positions over 40000 keys, 95 -> 102 us of one over 8 rows and a top-k, when the entry was tried first)
    if S >= 32768:
        if type(maskers[-1]) is OracleTopK:
            if not _select_fits(queries.dtype, queries.shape[0] * queries.shape[1] * Sq, S):
                return None
        elif Sq > 1 and S > 32768:
            return None
    bands, heavy = (), 0
    for masker in maskers:
        kind = type(masker)
        if heavy or len(bands) > 5 * (_MAX_BANDS - 2):
            return None
        if kind is SinkMasker:
            size = masker._calculate_effective_sink_size(S)
            if not 0 < size < S:
                return None
            bands += (0, 0, size, 0, 1)
        elif kind is LocalMasker:
            size = masker._calculate_effective_window_size(S)
            if not 0 < size < S - Sq:
                return None
            bands += (S - Sq - size + 1, 1, S - Sq + 1, 1, 1)
            if Sq > 1:
                bands += (S - Sq + 1, 1, S, 0, 0)
        elif kind is OracleTopK:
            heavy = masker._calculate_effective_heavy_size(S)
            if not 0 < heavy < S:
                return None
        else:
            return None
    module = _step_module()
    if module is False:
        return None
    device = queries.device
    stream = _native.stream_of(device)
    tickets, captured = mask_attention_utils.merge_tickets(device, stream)
    call = module.fixed_step
    done = call(queries, keys, values, attention_mask, sinks, float(scaling), bands, heavy, tickets,
                _native.sm_count(device), stream, captured)
    if done is None:
        return None
    if type(done) is tuple and len(done) == 1:  # nothing launched: the stream is being captured, with this identity
        tickets = mask_attention_utils.graph_tickets(device, stream, done[0])
        done = call(queries, keys, values, attention_mask, sinks, float(scaling), bands, heavy, tickets,
                    _native.sm_count(device), stream, True)
    if isinstance(done, int):
        tickets.zero_()  # a refused launch may leave tickets behind
        _native.check(done, "sah_fixed_step_run")
    out, scratch, ucols, umemb, ucount, groups, rows = done
    B, Hq, _, D = queries.shape
    mask_attention_utils._last_plan["step"] = (scratch, ucols, umemb, ucount, groups, rows, S, bands,
                                               (B, Hq, keys.shape[1], Sq, S, D, 0, _native.sm_count(device)))
    return out
