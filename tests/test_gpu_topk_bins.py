"""Selections whose threshold falls on the edge of a histogram bin (run with -m gpu): the search ends after the first or
second digit where a whole bin is taken, and must not end one key earlier or later.  Bit for bit against the oracle."""
import numpy as np
import pytest
import torch

from oracle import mxdsa_oracle as O

pytestmark = pytest.mark.gpu


def _check(scores, topk, pair):
    from mxdsa_b200.indexer import select_topk_indices
    idx, cnt = select_topk_indices(torch.from_numpy(scores).cuda(), topk, None, pair, None)
    ri, rc = O.topk_select_ref(scores, topk, None, pair, None)
    assert np.array_equal(cnt.cpu().numpy(), rc) and np.array_equal(idx.cpu().numpy(), ri)


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("s_kv,off", [(16384, -1), (16384, 0), (16384, 1), (1028, 0), (1028, 1)])
@pytest.mark.parametrize("digit", ["first", "second", "last"])
def test_threshold_on_the_edge_of_a_bin(digit, s_kv, off, pair):
    """A quarter of the keys lies above the edge: in bins of their own to 11, 22 or 32 bits, the rest just below."""
    rng = np.random.default_rng(s_kv + off)
    n = s_kv // 4
    bits = {"first": 1 << 21, "second": 1 << 10, "last": 1}[digit]
    edge = np.float32(1.0).view(np.uint32)                       # a bin begins here whatever the digit
    rows = []
    for _ in range(6):
        above = edge + rng.integers(0, 3, n).astype(np.uint32) * np.uint32(bits)
        below = edge - np.uint32(1) - rng.integers(0, 64, s_kv - n).astype(np.uint32)
        rows.append(rng.permutation(np.concatenate([above, below]).astype(np.uint32)).view(np.float32))
    scores = np.stack(rows)
    if pair:      # the other token's scores are lower: the larger of the two are the same keys
        scores = np.stack([scores, scores - np.float32(4.0)], axis=1).reshape(-1, s_kv)
    _check(scores, n + off, pair)


@pytest.mark.parametrize("topk", [5000, 10000, 10001])
def test_rows_of_several_sweeps(topk):
    """Lists longer than are staged: 10 000 keys share two values, the rest is lower."""
    rng = np.random.default_rng(topk)
    s = -np.abs(rng.standard_normal((5, 40000))).astype(np.float32) - 1
    for r in s:
        at = rng.permutation(40000)[:10000]
        r[at[:5000]], r[at[5000:]] = 2.0, 1.0
    _check(s, topk, False)
