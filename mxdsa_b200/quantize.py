"""Fused quantise-and-pack on the GPU: one kernel per tensor instead of the chain of torch kernels
that the reference's helpers launch (reference tests/mxfp8_test_utils.py:30-104).

Same function names as those helpers and byte-identical packed tensors for the same input values;
the dequantised copy that the helpers also return is not produced here (``mxdsa_b200.packing``
keeps the torch versions, which do).  Inputs: CUDA tensors, bf16 or fp32, last dimension 512 and
contiguous.  All compute is in libmxdsa.so (``mxdsa_pack_q`` / ``mxdsa_pack_kv``); there is no
fallback.
"""
from __future__ import annotations

import torch

D = 512       # elements of a row
ROW = 528     # bytes of a packed row: the elements and a 16-byte slot of scales

_module = None


def _ext():
    global _module
    if _module is None:
        from . import ext      # the package binds it after this module may have been imported
        _module = ext()
    return _module


def pack_dual_q64(q: torch.Tensor, paired_storage: bool = False) -> torch.Tensor:
    """q [..., 64, 512] -> u8 [..., 64, 528]: 512 E4M3 bytes + 8 UE8M0 scale bytes stored twice; scale g is
    shared by dims [32g,32g+32) and [256+32g,256+32g+32) (reference pack_dual_q64)."""
    return _ext().pack_q_rows(q, bool(paired_storage))


def pack_dual_prefill_kv64(kv: torch.Tensor) -> torch.Tensor:
    """kv [s_kv, 1, 512] -> u8 [s_kv, 1, 528] view of one flat buffer: all data rows, then all 16-byte scale
    slots; scale g covers dims [64g,64g+64) (reference pack_dual_prefill_kv64)."""
    return _ext().pack_prefill_kv(kv)


def pack_dual_decode_kv_pages(kv: torch.Tensor) -> torch.Tensor:
    """kv [pages, page_size, 1, 512] -> u8 [pages, page_size, 1, 528]: per page, page_size*512 data bytes and
    then page_size 16-byte scale slots (reference pack_dual_decode_kv_pages)."""
    return _ext().pack_decode_kv_pages(kv)
