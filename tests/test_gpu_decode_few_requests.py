"""Decode of few requests on many parts against the oracle: a request is then divided into up to dozens of splits of
one or two 64-key blocks, most parts have no work, and the combine kernel counts requests and shares a head between
warps.  Sizes sit at the edges of the combine kernel's loops: 2 .. 9 splits around its eight rows in flight, 34 and 66
around its 32 weights per register, and both ways of counting (b <= parts and b > parts)."""
import numpy as np
import pytest
import torch

import cases
from helpers import check_against_oracle
from oracle import mxdsa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,s_q,main_len,topk,extra_len,extra_topk,min_splits",
                         [(1, 1, 128, 128, 0, 0, 2), (1, 1, 512, 448, 0, 0, 7), (1, 2, 576, 512, 0, 0, 8),
                          (2, 1, 640, 576, 0, 0, 9), (1, 1, 128, 128, 4096, 2048, 34), (1, 1, 128, 128, 4096, 4096, 33),
                          (30, 6, 128, 128, 512, 512, 2)])
def test_few_requests_many_splits(b, s_q, main_len, topk, extra_len, extra_topk, min_splits, monkeypatch):
    import mxdsa_b200
    spec = dict(seed=90 + b + topk + extra_topk, b=b, s_q=s_q, main_len=main_len, topk=topk, sink=True)
    if extra_topk:
        spec.update(extra_len=extra_len, extra_topk=extra_topk)
    monkeypatch.setitem(cases.DECODE_CASES, "few", spec)
    c = cases.build_decode("few")
    t = lambda x: None if x is None else torch.from_numpy(np.ascontiguousarray(x)).cuda()
    out, lse, meta, splits = mxdsa_b200.dual_mxfp8_sparse_decode_fwd(
        t(c["q"]), t(c["kv"]), t(c["indices"]), None, t(c["attn_sink"]), None, None, t(c["extra_kv"]),
        t(c["extra_indices"]), None, 512, 512, c["sm_scale"], c["w1"], c["w2"])
    mxdsa_b200.device_fault()
    n = np.diff(splits.cpu().numpy())
    assert n.max() >= min_splits, n
    parts = meta.shape[0]
    ro, rl = O.decode_ref(c["q"], c["kv"], c["indices"], None, c["attn_sink"], c["extra_kv"], c["extra_indices"], None,
                          c["sm_scale"], c["w1"], c["w2"], level=1, sched=O.sched_meta_ref(b, topk, extra_topk, parts))
    # partials are merged in fp32: the bounds of the whole path (tests/helpers.py) apply unchanged
    check_against_oracle(out.float().cpu().numpy(), ro)
    assert np.abs(lse.transpose(1, 2).cpu().numpy() - rl).max() <= 1e-3
