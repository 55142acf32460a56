"""The work that users of this package have it do, as cases that can be prepared, run and timed.

A serving or training step around sparse attention makes four kinds of calls, and every kind is here over
its range of sizes:

  prefill   dual_mxfp8_head64_sparse_prefill_fwd and its extended form (odd token counts, any topk, float8 tensors)
  decode    dual_mxfp8_sparse_decode_fwd with a schedule computed once and reused, and the whole-request form
  select    indexer.select_topk_indices: score rows -> index rows, per pair of query tokens or per request
  pack      quantize.pack_*: activations -> the packed MXFP8 rows that the operators read

Values are N(0, 1) through the packers, KV group scales factor into token scale x dimension scale, index rows are
distinct, uniform and ascending as the selection writes them, as in this repository's benchmark and tests.
"""
import math

import torch

import mxdsa_b200 as M
from mxdsa_b200 import packing, quantize
from mxdsa_b200.indexer import select_topk_indices

HEADS, DIM, ROW = 64, 512, 528
SCALE = DIM ** -0.5
PAGE = 64


def listed():
    return [
        # a short prompt: the smallest prefill call of the tests and benchmark, latency counts
        dict(name="prefill_short", kind="prefill", s_q=256, s_kv=1024, topk=128, ext=False, sink=False, lengths=False,
             tail=0.0),
        # a chunk of chunked prefill over a filled cache at the usual list length
        dict(name="prefill_chunk", kind="prefill", s_q=4096, s_kv=16384, topk=2048, ext=False, sink=True, lengths=False,
             tail=0.0),
        # a ragged prompt: odd token count, odd list length, causal lengths, float8 tensors, attention sink
        dict(name="prefill_ragged", kind="prefill", s_q=1537, s_kv=5000, topk=700, ext=True, sink=True, lengths=True,
             tail=0.0),
        # the benchmark's headline: a long batch with long lists
        dict(name="prefill_long", kind="prefill", s_q=65536, s_kv=16384, topk=4096, ext=False, sink=False, lengths=False,
             tail=0.0),
        # one request, one token: the latency of a single user's step
        dict(name="decode_single", kind="decode", b=1, s_q=1, main_len=128, topk=128, extra_len=4096, extra_topk=2048,
             whole=False, fp8=False, sink=False, lengths=False),
        # a served batch with draft tokens and short extra lists
        dict(name="decode_batch", kind="decode", b=64, s_q=6, main_len=128, topk=128, extra_len=16384, extra_topk=512,
             whole=False, fp8=False, sink=False, lengths=False),
        # the benchmark's largest decode: gather-bound
        dict(name="decode_large", kind="decode", b=128, s_q=6, main_len=128, topk=128, extra_len=16384, extra_topk=4096,
             whole=False, fp8=False, sink=False, lengths=False),
        # requests of different lengths, two tokens each, float8 tensors, sink, no combine pass
        dict(name="decode_ragged", kind="decode", b=37, s_q=2, main_len=192, topk=128, extra_len=5056, extra_topk=1000,
             whole=True, fp8=True, sink=True, lengths=True),
        # index selection of a prefill chunk: one row per pair of query tokens
        dict(name="select_prefill", kind="select", rows=2048, pair=True, s_kv=16384, topk=2048, lengths=True, offset=False),
        # index selection of a decode step: few rows over a long context, pool offsets
        dict(name="select_decode", kind="select", rows=64, pair=False, s_kv=65536, topk=2048, lengths=True, offset=True),
        # the queries of a prefill chunk on their way in
        dict(name="pack_queries", kind="pack", what="q", rows=4096 * HEADS, dtype="bf16", paired=False),
        # the tokens that a decode step appends, one page each
        dict(name="pack_pages", kind="pack", what="pages", rows=64 * PAGE, dtype="bf16", paired=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["prefill", "prefill", "decode", "decode", "select", "pack"])
    if kind == "prefill":
        ext = rng.random() < 0.4
        topk = _log(rng, 64, 4096)
        s_q = _log(rng, 64, 65536)
        if not ext:
            topk = max(64, topk // 64 * 64)
            s_q = max(2, s_q // 2 * 2)
        s_kv = max(topk, _log(rng, 512, 32768))
        return dict(kind=kind, s_q=s_q, s_kv=s_kv, topk=topk, ext=ext, sink=rng.random() < 0.3,
                    lengths=rng.random() < 0.3, tail=rng.choice([0.0, 0.0, 0.1]))
    if kind == "decode":
        main_len = PAGE * rng.randint(2, 8)
        extra_topk = 0 if rng.random() < 0.15 else _log(rng, 64, 4096)
        extra_len = 0 if extra_topk == 0 else -(-max(extra_topk, _log(rng, 256, 16384)) // PAGE) * PAGE
        return dict(kind=kind, b=_log(rng, 1, 128), s_q=rng.choice([1, 1, 2, 3, 4, 5, 6]), main_len=main_len,
                    topk=rng.choice([64, 128, 128]), extra_len=extra_len, extra_topk=extra_topk,
                    whole=rng.random() < 0.3, fp8=rng.random() < 0.3, sink=rng.random() < 0.3,
                    lengths=rng.random() < 0.3)
    if kind == "select":
        pair = rng.random() < 0.5
        s_kv = max(1024, _log(rng, 1024, 131072) // 4 * 4)
        most = max(1, (1 << 28) // (s_kv * (2 if pair else 1)))
        return dict(kind=kind, rows=min(most, _log(rng, 1, 8192)), pair=pair, s_kv=s_kv,
                    topk=min(s_kv, _log(rng, 64, 4096)), lengths=rng.random() < 0.5, offset=not pair)
    what = rng.choice(["q", "q", "kv", "pages"])
    rows = _log(rng, 64, 1 << 20)
    if what != "kv":
        rows = max(1, rows // 64) * 64      # whole tokens of 64 heads, whole pages of 64 rows
    return dict(kind="pack", what=what, rows=rows, dtype=rng.choice(["bf16", "bf16", "f32"]),
                paired=what == "q" and rng.random() < 0.3)


# ---------------------------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _queries(tokens, g):
    """Packed queries of `tokens` tokens, u8 [tokens, 64, 528]."""
    q = torch.empty((tokens, HEADS, ROW), dtype=torch.uint8, device="cuda")
    for i in range(0, tokens, 4096):
        n = min(4096, tokens - i)
        x = torch.randn((n, HEADS, DIM), device="cuda", dtype=torch.bfloat16, generator=g)
        q[i:i + n] = quantize.pack_dual_q64(x)
    return q


def _distinct_rows(rows, pool, topk, g):
    """`rows` ascending rows of `topk` distinct uniform indices below `pool`."""
    idx = torch.empty((rows, topk), dtype=torch.int32, device="cuda")
    step = max(1, (1 << 26) // pool)
    for i in range(0, rows, step):
        n = min(step, rows - i)
        pick = torch.rand((n, pool), device="cuda", generator=g).topk(topk, dim=1, sorted=False).indices
        idx[i:i + n] = pick.sort(dim=1).values.int()
    return idx


def _sink(case, g):
    return torch.randn(HEADS, device="cuda", generator=g) * 2 if case["sink"] else None


def _prepare_prefill(case, g):
    s_q, s_kv, topk = case["s_q"], case["s_kv"], case["topk"]
    pairs = (s_q + 1) // 2
    q = _queries(s_q, g)
    kvf, w1, w2 = packing.make_rank1_kv((s_kv, 1), device="cuda", generator=g)
    kv = quantize.pack_dual_prefill_kv64(kvf)
    idx = _distinct_rows(pairs, s_kv, topk, g).view(pairs, 1, topk)
    if case["tail"]:
        idx[:, :, topk - int(topk * case["tail"]):] = -1
    lengths = None
    if case["lengths"]:      # a pair attends to what lies before it: short lists at the start, full ones later on
        lengths = torch.linspace(1, 2 * topk, pairs, device="cuda").clamp_(max=topk).int()
    if case["ext"]:
        q, kv = q.view(torch.float8_e4m3fn), kv.view(torch.float8_e4m3fn)
    return dict(q=q, kv=kv, idx=idx, w1=w1, w2=w2, sink=_sink(case, g), lengths=lengths)


def _pool(pages, wide, g):
    """`pages` packed pages: a rank-1 pool of at most 256 distinct pages, dealt out at random."""
    own = min(pages, wide.size(0))
    pick = torch.randint(0, own, (pages,), device="cuda", generator=g)
    return wide[pick].contiguous()


def _prepare_decode(case, g):
    b, s_q, topk, ek = case["b"], case["s_q"], case["topk"], case["extra_topk"]
    main_len, extra_len = case["main_len"], case["extra_len"]
    q = _queries(b * s_q, g).view(b, s_q, HEADS, ROW)
    kvf, w1, w2 = packing.make_rank1_kv((256, PAGE, 1), device="cuda", generator=g)
    wide = quantize.pack_dual_decode_kv_pages(kvf)
    kv = _pool(b * main_len // PAGE, wide, g)
    at = torch.arange(b, device="cuda", dtype=torch.int32).view(b, 1, 1)
    idx = _distinct_rows(b * s_q, main_len, topk, g).view(b, s_q, topk) + at * main_len
    ekv = eidx = length = elength = None
    if ek:
        ekv = _pool(b * extra_len // PAGE, wide, g)
        eidx = _distinct_rows(b * s_q, extra_len, ek, g).view(b, s_q, ek) + at * extra_len
    if case["lengths"]:
        length = torch.randint(1, topk + 1, (b,), device="cuda", generator=g).int()
        if ek:
            elength = torch.randint(0, ek + 1, (b,), device="cuda", generator=g).int()
    if case["fp8"]:
        q, kv = q.view(torch.float8_e4m3fn), kv.view(torch.float8_e4m3fn)
        ekv = ekv.view(torch.float8_e4m3fn) if ek else None
    op = M.dual_mxfp8_sparse_decode_fwd_whole if case["whole"] else M.dual_mxfp8_sparse_decode_fwd
    s = dict(op=op, q=q, kv=kv, idx=idx, length=length, sink=_sink(case, g), ekv=ekv, eidx=eidx, elength=elength, w1=w1,
             w2=w2)
    # the schedule depends on the lengths alone: a serving program computes it once and hands it to every layer
    s["meta"], s["splits"] = _decode(s, None, None)[2:]
    return s


def _decode(s, meta, splits):
    return s["op"](s["q"], s["kv"], s["idx"], s["length"], s["sink"], meta, splits, s["ekv"], s["eidx"], s["elength"],
                   DIM, DIM, SCALE, s["w1"], s["w2"])


def _prepare_select(case, g):
    rows, s_kv = case["rows"], case["s_kv"]
    scores = torch.randn((rows * (2 if case["pair"] else 1), s_kv), device="cuda", generator=g)
    lengths = offset = None
    if case["lengths"]:      # contexts between half full and full
        lengths = torch.randint(s_kv // 2, s_kv + 1, (rows,), device="cuda", generator=g).int()
    if case["offset"]:       # decode: a request's keys start at its place in the pool
        offset = torch.arange(rows, device="cuda", dtype=torch.int32) * s_kv
    return dict(scores=scores, topk=case["topk"], lengths=lengths, pair=case["pair"], offset=offset)


def _prepare_pack(case, g):
    rows = case["rows"]
    shape = {"q": (rows // HEADS, HEADS, DIM), "kv": (rows, 1, DIM), "pages": (rows // PAGE, PAGE, 1, DIM)}[case["what"]]
    x = torch.randn(shape, device="cuda", generator=g, dtype=torch.bfloat16 if case["dtype"] == "bf16" else torch.float32)
    return dict(x=x, what=case["what"], paired=case["paired"])


def prepare(case, seed):
    make = {"prefill": _prepare_prefill, "decode": _prepare_decode, "select": _prepare_select, "pack": _prepare_pack}
    s = make[case["kind"]](case, _generator(seed))
    s["kind"] = case["kind"]
    s["ext"] = case.get("ext", False)
    return s


# ---------------------------------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "prefill":
        op = M.dual_mxfp8_head64_sparse_prefill_fwd_ex if s["ext"] else M.dual_mxfp8_head64_sparse_prefill_fwd
        return op(s["q"], s["kv"], s["idx"], SCALE, s["w1"], s["w2"], s["sink"], s["lengths"])
    if kind == "decode":
        return _decode(s, s["meta"], s["splits"])[:2]
    if kind == "select":
        return select_topk_indices(s["scores"], s["topk"], s["lengths"], s["pair"], s["offset"])
    if s["what"] == "q":
        return quantize.pack_dual_q64(s["x"], s["paired"])
    return quantize.pack_dual_prefill_kv64(s["x"]) if s["what"] == "kv" else quantize.pack_dual_decode_kv_pages(s["x"])


# ---------------------------------------------------------------------------------------------- what a pass needs
def _seen(pool, topk, rows):
    """Expected number of distinct keys that `rows` independent rows of `topk` keys out of `pool` name."""
    return pool * (1.0 - (1.0 - min(1.0, topk / pool)) ** rows) if pool and topk else 0.0


def work(case):
    kind = case["kind"]
    if kind == "prefill":
        s_q, topk = case["s_q"], case["topk"]
        pairs = (s_q + 1) // 2
        keys = topk * (1.0 - case["tail"])
        if case["lengths"]:
            keys *= 0.75     # half the pairs attend to half a list on average
        data = s_q * HEADS * (ROW + 2 * DIM + 8) + pairs * keys * 4 + _seen(case["s_kv"], keys, pairs) * ROW
        return {"bytes": data, "flops": 2.0 * s_q * HEADS * keys * 2 * DIM}
    if kind == "decode":
        tokens, pairs = case["b"] * case["s_q"], (case["s_q"] + 1) // 2
        part = 0.5 if case["lengths"] else 1.0
        main, extra = case["topk"] * part, case["extra_topk"] * part
        kv = _seen(case["main_len"], main, pairs) + _seen(case["extra_len"], extra, pairs)
        data = tokens * HEADS * (ROW + 2 * DIM + 4) + case["b"] * (pairs * (main + extra) * 4 + kv * ROW)
        return {"bytes": data, "flops": 2.0 * tokens * HEADS * (main + extra) * 2 * DIM}
    if kind == "select":
        keys = case["s_kv"] * (0.75 if case["lengths"] else 1.0) * (2 if case["pair"] else 1)
        return {"bytes": case["rows"] * (keys * 4 + case["topk"] * 4 + 4), "flops": case["rows"] * keys}
    return {"bytes": case["rows"] * (DIM * (2 if case["dtype"] == "bf16" else 4) + ROW), "flops": case["rows"] * DIM * 2.0}


def tolerance(case):
    # selected indices and packed bytes are whole values
    if case["kind"] in ("select", "pack"):
        return "exact"
    # bf16 results; probabilities pass through E4M3 (steps of 1/16 to 1/8 of the value), so a sum in another order
    # can move single ones by a step, which weighs most where a row attends to few keys
    return {"rel": 1e-2, "max": 0.2}
