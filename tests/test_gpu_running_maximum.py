"""Lists whose running maximum grows with every tile, for some heads only (run with -m gpu).

Every tile then rescales the accumulator between its own PV steps and those of the tile before it, which is work of
other warps than the softmax; heads of the other sign keep their first maximum.  The oracle evaluates the same tiles."""
import numpy as np
import pytest
import torch

from helpers import LSE_MAX_ABS, check_against_oracle
from oracle import mxdsa_oracle as O

pytestmark = pytest.mark.gpu
ONE = [0x7F7F7F7F] * 8
SCALE = 512 ** -0.5 * 20


def _rows(n, rng, u, step):
    """n keys along u, longer by `step` every 64: about 10 powers of two of probability for a head along u."""
    c = 0.05 + step * (np.arange(n) // 64)
    return (c[:, None] * u + 0.003 * rng.standard_normal((n, 512))).astype(np.float32)


def _queries(shape, rng, u):
    sign = np.where(np.arange(64) % 3 == 0, -1.0, 1.0)      # every group of 32 heads has both kinds
    return (sign[:, None] * u + 0.1 * rng.standard_normal(shape + (64, 512))).astype(np.float32)


def _t(x):
    return torch.from_numpy(np.array(x, order="C")).cuda()   # a copy: broadcast rows have no strides of their own


@pytest.mark.parametrize("s_q,topk", [(2, 64), (2, 65), (3, 128), (2, 192), (2, 448), (4, 512), (2, 640), (301, 577), (2, 1000)])
def test_prefill(s_q, topk):
    import mxdsa_b200 as M
    rng = np.random.default_rng(topk)
    u = rng.standard_normal(512)
    kv = O.pack_prefill_kv(_rows(topk, rng, u, 0.0155)[:, None])[0]
    few = _queries((min(s_q, 4),), rng, u)
    q = O.pack_q(few, paired_storage=True)[0][np.arange(s_q) % len(few)]
    pairs = (s_q + 1) // 2
    idx = np.broadcast_to(np.arange(topk, dtype=np.int32), (pairs, 1, topk))
    out, mxl, lse = M.dual_mxfp8_head64_sparse_prefill_fwd_ex(_t(q), _t(kv), _t(idx), SCALE, ONE, ONE)
    M.device_fault()
    n = len(few)
    ro, rm, rl = O.prefill_ref(q[:n], kv, idx[:(n + 1) // 2], SCALE, ONE, ONE, level=1)
    check_against_oracle(out[:n].float().cpu().numpy(), ro)
    assert np.abs(lse[:n].cpu().numpy() - rl).max() <= LSE_MAX_ABS and np.abs(mxl[:n].cpu().numpy() - rm).max() <= LSE_MAX_ABS
    if n == 4:                                              # the queries repeat: so do the results, bit for bit
        again = out.view(torch.int16)[: s_q // 4 * 4].view(-1, 4, 64, 512)
        assert (again == again[:1]).all()


@pytest.mark.parametrize("b,s_q,extra", [(1, 1, 0), (2, 2, 64), (3, 3, 448), (40, 2, 333)])
@pytest.mark.parametrize("whole", [False, True])
def test_decode(b, s_q, extra, whole):
    import mxdsa_b200 as M
    rng = np.random.default_rng(b + extra)
    u = rng.standard_normal(512)
    rows = _rows(576, rng, u, 0.0155).reshape(9, 64, 1, 512)
    pool = O.pack_decode_kv_pages(rows)[0]
    one = O.pack_q(_queries((1, s_q), rng, u), paired_storage=True)[0]
    q = np.repeat(one, b, axis=0)
    idx = np.broadcast_to(np.arange(128, dtype=np.int32), (b, s_q, 128))
    eidx = np.broadcast_to(np.arange(128, 128 + extra, dtype=np.int32), (b, s_q, extra)) if extra else None
    op = M.dual_mxfp8_sparse_decode_fwd_whole if whole else M.dual_mxfp8_sparse_decode_fwd
    out, lse, meta, splits = op(_t(q), _t(pool), _t(idx), None, None, None, None, _t(pool) if extra else None,
                                _t(eidx) if extra else None, None, 512, 512, SCALE, ONE, ONE)
    M.device_fault()
    sched = None if whole else O.sched_meta_ref(b, 128, extra, meta.shape[0], None, None)
    ro, rl = O.decode_ref(q, pool, idx, None, None, pool if extra else None, eidx, None, SCALE, ONE, ONE, level=1, sched=sched)[:2]
    check_against_oracle(out.float().cpu().numpy(), ro)
    assert np.abs(lse.transpose(1, 2).contiguous().cpu().numpy() - rl).max() <= LSE_MAX_ABS
