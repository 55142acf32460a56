"""Score tensors of any layout reach the selection kernel with strides that it reads inside their storage.  The kernel
takes a row stride of 0 for "dense", so a broadcast row must not arrive as one."""
import pytest
import torch

from mxdsa_b200 import indexer

X = torch.arange(6 * 64, dtype=torch.float32).view(6, 64)


@pytest.mark.parametrize("scores", [
    X, X[:, :32], X[::2], X[1:2], X[1:2, 8:], X[0].clone().expand(5, 64), X[4:5].expand(4, 64), X[0].view(1, 64).as_strided((1, 64), (0, 1)),
    X.t()[:, :4], X.t().contiguous().t(), X[0].view(64, 1).t(), X[5].view(64, 1).t().expand(3, 64), X[:0]])
def test_strides_stay_inside_the_storage(scores):
    rows = indexer._score_rows(scores)
    assert torch.equal(rows, scores)
    n, s_kv = rows.shape
    stride = rows.stride(0) or s_kv        # what the kernel makes of it
    assert rows.stride(1) == 1 and stride >= s_kv
    assert n == 0 or rows.storage_offset() + (n - 1) * stride + s_kv <= rows.untyped_storage().nbytes() // 4
