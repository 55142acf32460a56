"""Decode of one token to a request (run with -m gpu): both CTAs of a pair hold the token and store half of the columns each.  The
same token twice gives two rows that a CTA each stores whole: bit for bit the same by the same schedule."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("b,extra", [(1, 0), (1, 2048), (1, 4096), (3, 700), (8, 512), (9, 1000), (30, 2048), (64, 512), (100, 64), (40, 4096), (128, 1300)])
def test_one_token_is_half_of_two(b, extra, whole):
    import mxdsa_b200 as M
    from mxdsa_b200 import packing, quantize
    g = torch.Generator(device="cuda").manual_seed(10 * b + extra)
    q = quantize.pack_dual_q64(torch.randn(b, 64, 512, device="cuda", generator=g)).view(b, 1, 64, 528)
    kvf, w1, w2 = packing.make_rank1_kv((2 * b + 80, 64, 1), device="cuda", generator=g)
    kv = quantize.pack_dual_decode_kv_pages(kvf)
    at = torch.arange(b, device="cuda", dtype=torch.int32).view(b, 1, 1)
    idx = torch.rand(b, 128, device="cuda", generator=g).argsort(1).int().view(b, 1, 128) + at * 128
    ekv = eidx = elength = None
    if extra:
        ekv = kv[2 * b:].contiguous()
        eidx = torch.rand(b, 80 * 64, device="cuda", generator=g).argsort(1)[:, :extra].int().view(b, 1, extra).contiguous()
        elength = torch.randint(0, extra + 1, (b,), device="cuda", generator=g).int()
    sink = torch.randn(64, device="cuda", generator=g)
    op = M.dual_mxfp8_sparse_decode_fwd_whole if whole else M.dual_mxfp8_sparse_decode_fwd
    run = lambda n, *schedule: op(q.repeat(1, n, 1, 1), kv[: 2 * b].contiguous(), idx.repeat(1, n, 1), None, sink, *schedule, ekv,
                                  None if eidx is None else eidx.repeat(1, n, 1), elength, 512, 512, 512 ** -0.5, w1, w2)
    for _ in range(2):                 # and again, behind a call of the other kind
        two = run(2, None, None)
        # two tokens have half as many parts: the others have no work
        meta = torch.zeros_like(run(1, None, None)[2])
        meta[:, 0] = b
        meta[: two[2].size(0)] = two[2]
        one = run(1, meta, two[3])
    torch.cuda.synchronize()
    M.device_fault()
    for got, rows in ((one[0], two[0]), (one[1].transpose(1, 2), two[1].transpose(1, 2))):
        assert torch.equal(got, rows[:, :1]) and torch.equal(got, rows[:, 1:])
