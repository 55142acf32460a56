"""Index selection on the GPU: score rows -> the ``indices`` / ``topk_length`` tensors of the attention
operators.

The reference has no producer for ``indices``; its callers fix the conventions (reference
tests/benchmark.py:119-147: int32 rows ``[s_q/2, 1, topk]`` for prefill with one row per PAIR of query
tokens, ``[b, s_q, topk]`` for decode with pool indices offset by ``request * pool_len``; -1 entries are
never attended; ``topk_length`` bounds the attended prefix).  ``select_topk_indices`` produces exactly
those tensors from score rows.  All compute is in libmxdsa.so (``mxdsa_topk_select``); there is no
fallback.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch


_module = None


def _ext():
    global _module
    if _module is None:
        from . import ext      # the package binds it after this module may have been imported
        _module = ext()
    return _module


def _score_rows(scores: torch.Tensor) -> torch.Tensor:
    """`scores` [n, s_kv] with the strides that the kernel is to read it by.  It takes a row stride of 0 for s_kv, so a
    row that is broadcast over n is copied out; the stride of a single row means nothing and is set to s_kv."""
    n, s_kv = scores.shape
    if scores.stride(1) != 1 or (n > 1 and scores.stride(0) == 0):
        scores = scores.contiguous()
    if n == 1:
        scores = scores.as_strided((1, s_kv), (s_kv, 1))
    return scores


def select_topk_indices(scores: torch.Tensor, topk: int, lengths: Optional[torch.Tensor] = None,
                        pair: bool = False, row_offset: Optional[torch.Tensor] = None
                        ) -> Tuple[torch.Tensor, torch.Tensor]:
    """scores f32 [n, s_kv] (CUDA, s_kv a multiple of 4) -> (indices i32 [rows, topk], topk_length i32 [rows]).

    rows = n, or n/2 with ``pair=True`` (score rows 2r and 2r+1 are the two tokens of pair r; a key's
    score is the larger of the two).  Row r selects the min(topk, candidates) best keys among
    ``j < lengths[r]``; NaN and -inf scores are no candidates; ties go to the smaller j.  The selected
    indices are ascending, ``row_offset[r]`` is added to each, and the row is padded with -1.
    """
    if not scores.is_cuda or scores.dtype != torch.float32 or scores.dim() != 2:
        raise RuntimeError("scores must be a CUDA float32 tensor of shape [n, s_kv]")
    n, s_kv = scores.shape
    group = 2 if pair else 1
    if n % group:
        raise RuntimeError("pair=True needs an even number of score rows")
    if s_kv <= 0 or s_kv % 4 or topk <= 0:
        raise RuntimeError("s_kv must be a positive multiple of 4 and topk positive")
    rows = n // group
    scores = _score_rows(scores)

    def opt(t, name):
        if t is None:
            return None
        if not t.is_cuda or t.dtype != torch.int32 or t.numel() != rows:
            raise RuntimeError(f"{name} must be a CUDA int32 tensor of {rows} elements")
        return t.contiguous()

    lengths, row_offset = opt(lengths, "lengths"), opt(row_offset, "row_offset")
    return _ext().topk_rows(scores, topk, lengths, group, row_offset)
