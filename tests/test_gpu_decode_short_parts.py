"""Decode of short parts (up to 16 blocks of 64 keys on average) leaves through other stores than decode of longer ones (run
with -m gpu).  The rule counts what the index tensors hold, not what the lengths leave of it: the same work, its index rows
padded beyond the line and cut back by the lengths, takes the other route, and every bit must agree, divided requests and whole
ones, last work items and earlier ones, tokens and blocks that do not exist."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("s_q,keys", [(1, 896), (1, 65), (2, 896), (3, 500), (6, 896), (6, 1)])
def test_both_routes_agree(s_q, keys, whole):
    import mxdsa_b200 as M
    from mxdsa_b200 import packing, quantize
    parts = torch.cuda.get_device_properties(0).multi_processor_count // s_q
    b = max(1, 16 * parts // (2 + 14))       # 128 main keys and 896 extra ones a request: 16 blocks to a part, just short
    g = torch.Generator(device="cuda").manual_seed(s_q + keys)
    q = quantize.pack_dual_q64(torch.randn((b * s_q, 64, 512), device="cuda", dtype=torch.bfloat16, generator=g)).view(b, s_q, 64, 528)
    kvf, w1, w2 = packing.make_rank1_kv((64, 64, 1), device="cuda", generator=g)
    pool = quantize.pack_dual_decode_kv_pages(kvf)
    pick = lambda n: torch.rand((b * s_q, 4096), device="cuda", generator=g).topk(n, dim=1).indices.sort(dim=1).values.int().view(b, s_q, n)
    idx, eidx = pick(128), pick(keys)
    sink = torch.randn(64, device="cuda", generator=g)
    short, long = torch.full((b, s_q, 896), -1, device="cuda", dtype=torch.int32), torch.full((b, s_q, 1536), -1, device="cuda", dtype=torch.int32)
    short[:, :, :keys] = eidx
    long[:, :, :keys] = eidx
    elen = torch.randint(1, keys + 1, (b,), device="cuda", generator=g).int()
    length = torch.randint(1, 129, (b,), device="cuda", generator=g).int()
    op = M.dual_mxfp8_sparse_decode_fwd_whole if whole else M.dual_mxfp8_sparse_decode_fwd
    run = lambda rows: op(q, pool, idx, length, sink, None, None, pool, rows, elen, 512, 512, 512 ** -0.5, w1, w2)
    a, c = run(short), run(long)
    M.device_fault()
    assert torch.equal(a[2], c[2]) and torch.equal(a[3], c[3])       # the same schedule
    if not whole:
        assert (a[3][1:] - a[3][:-1]).max() > 1                      # of divided requests
    assert torch.equal(a[0].view(torch.int16), c[0].view(torch.int16)) and torch.equal(a[1], c[1])


@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("s_q", [1, 3])
def test_parts_that_find_no_sm_at_the_start(s_q, whole):
    """More parts than CTA pairs fit the chip at once: those that come late look at the schedule before they set anything up.
    Requests up to the first late part, up to it and beyond it, calls one behind the other, against the route for long parts."""
    import mxdsa_b200 as M
    from mxdsa_b200 import packing, quantize
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    parts, first_late = sms // s_q, sms // 2 // ((s_q + 1) // 2)
    assert first_late < parts
    g = torch.Generator(device="cuda").manual_seed(s_q)
    kvf, w1, w2 = packing.make_rank1_kv((16, 64, 1), device="cuda", generator=g)
    pool = quantize.pack_dual_decode_kv_pages(kvf)
    op = M.dual_mxfp8_sparse_decode_fwd_whole if whole else M.dual_mxfp8_sparse_decode_fwd
    short, long = [], []
    for b in (1, first_late - 1, first_late, first_late + 1, parts - 1):
        q = quantize.pack_dual_q64(torch.randn((b * s_q, 64, 512), device="cuda", dtype=torch.bfloat16, generator=g)).view(b, s_q, 64, 528)
        pick = lambda n: torch.rand((b * s_q, 1024), device="cuda", generator=g).topk(n, dim=1).indices.int().view(b, s_q, n)
        idx, eidx = pick(64), pick(65)
        elen = torch.randint(1, 66, (b,), device="cuda", generator=g).int()
        padded = torch.full((b, s_q, 64 * (16 * parts // b + 2)), -1, device="cuda", dtype=torch.int32)
        padded[:, :, :65] = eidx
        run = lambda rows: op(q, pool, idx, None, None, None, None, pool, rows, elen, 512, 512, 512 ** -0.5, w1, w2)
        short.append(run(eidx))
        long.append(run(padded))
    M.device_fault()
    for a, c in zip(short, long):
        assert torch.equal(a[2], c[2]) and torch.equal(a[0].view(torch.int16), c[0].view(torch.int16)) and torch.equal(a[1], c[1])
