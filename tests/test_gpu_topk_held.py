"""Selection of rows that are held in registers (run with -m gpu): a sample points at an interval, keys are counted within it.
Bit for bit against the oracle where that can go wrong: rows that end at the edges of chunks, warps and groups of four; scores of
either sign, around zero, of few values and of very different size; samples that mislead; more rows than resident CTAs."""
import numpy as np
import pytest
import torch

from oracle import mxdsa_oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 3, 127, 128, 129, 1021, 2047, 2048, 2049, 4095, 4096, 6143, 6146, 8192, 8195, 14336, 14339, 16383, 16384]


def _check(scores, topk, lengths=None, pair=False, offset=None):
    from mxdsa_b200.indexer import select_topk_indices
    dev = "cuda:0"
    t = lambda a: None if a is None else torch.from_numpy(np.asarray(a, np.int32)).to(dev)
    idx, cnt = select_topk_indices(torch.from_numpy(scores).to(dev), topk, t(lengths), pair, t(offset))
    ri, rc = O.topk_select_ref(scores, topk, lengths, pair, offset)
    assert np.array_equal(cnt.cpu().numpy(), rc) and np.array_equal(idx.cpu().numpy(), ri)


def _scores(kind, n, s_kv, rng):
    x = rng.standard_normal((n, s_kv)).astype(np.float32)
    if kind == "negative":
        x = x - np.float32(50)
    elif kind == "zeros":              # most keys are zeros of either sign
        x[rng.random(x.shape) < 0.9] = 0.0
        x[rng.random(x.shape) < 0.5] *= np.float32(-1)
    elif kind == "few":                # five values
        x = np.round(x).clip(-2, 2)
    elif kind == "sizes":              # 1e-40 to 1e38, some infinite, some NaN
        x = (x * 10.0 ** rng.integers(-40, 39, x.shape)).astype(np.float32)
        x[rng.random(x.shape) < 0.01] = np.inf
        x[rng.random(x.shape) < 0.05] = np.nan
        x[rng.random(x.shape) < 0.05] = -np.nan
    elif kind == "misled":             # the best keys lie where no sample does, in adjacent pieces
        x[:, s_kv // 3: s_kv // 3 + 100] += np.float32(9)
        x[:, 1::8] = np.where(np.arange(s_kv)[1::8] % 256 < 128, x[:, 1::8] + np.float32(20), x[:, 1::8])
    elif kind == "close":              # differ in the last bits
        x = np.float32(3) + rng.integers(0, 40, x.shape).astype(np.float32) * np.float32(2.0 ** -22)
    return x


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("kind", ["normal", "negative", "zeros", "few", "sizes", "misled", "close"])
@pytest.mark.parametrize("s_kv,topk", [(16384, 2048), (16384, 33), (8196, 1), (2052, 130), (260, 64), (1536, 1200)])
def test_against_the_oracle(s_kv, topk, kind, pair):
    rng = np.random.default_rng(s_kv + topk)
    with np.errstate(over="ignore"):
        scores = _scores(kind, 6 if pair else 5, s_kv, rng)
    _check(scores, topk, pair=pair)


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("topk", [64, 1030, 4096])
def test_rows_that_end_anywhere(topk, pair):
    rng = np.random.default_rng(topk)
    n = len(LENGTHS)
    _check(rng.standard_normal((n * (2 if pair else 1), 16384)).astype(np.float32), topk, LENGTHS, pair,
           np.arange(n, dtype=np.int32) * 16384)


@pytest.mark.parametrize("pair", [False, True])
def test_more_rows_than_ctas(pair):
    rng = np.random.default_rng(7)
    rows = 700
    lengths = rng.integers(0, 2561, rows)
    _check(rng.standard_normal((rows * (2 if pair else 1), 2560)).astype(np.float32), 200, lengths, pair)


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("top", [0x3f7fffff, 0x3fffffff, 0x40000000, 0x7f7fffff, 0x7f800000])
def test_thresholds_just_below_zero(top, pair):
    """-0 and +0 are one score, which leaves a gap in the keys' integer images just below zero.  With a maximum of many low one
    bits the threshold's bin begins in the gap: negative subnormals by the hundred, zeros in the bin ahead of it."""
    rng = np.random.default_rng(top)
    best = np.uint32(top).view(np.float32)
    equal = np.full((2, 1024), -5, np.float32)
    equal[:, 10:60], equal[:, 200:300] = 0.0, np.float32(-1e-40)
    equal[:, 30:40] = np.float32(-0.0)
    mixed = np.zeros((2, 2048), np.float32)
    mixed[:, :100] = rng.random((2, 100))
    mixed[:, 548:] = -rng.integers(1, 5000, (2, 1500)).astype(np.uint32).view(np.float32)
    mixed = rng.permuted(mixed, axis=1)
    for x, topk in ((equal, 100), (mixed, 1000), (mixed, 700), (mixed, 140)):
        x = np.ascontiguousarray(np.repeat(x, 2, axis=0) if pair else x)
        x[:, 0] = best
        _check(x, topk, pair=pair)


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("largest,smallest", [(-1.0, -3.0), (-1e-45, -1e-42), (-1e-45, -1.0), (-1e-3, -3.4e38), (-3.4028235e38, -3.4028235e38),
                                              (-3.4028233e38, -3.4028235e38), (-0.0, -2.0)])
def test_no_score_is_positive(largest, smallest, pair):
    """Negative maxima near and far from the ends of the negative scores, with what must not pass for one of them: NaNs of either
    sign, -inf, and the keys behind the row's end."""
    rng = np.random.default_rng(11)
    ends = np.array([largest, smallest], np.float32).view(np.uint32).astype(np.int64)
    for s_kv, topk, lengths in ((2052, 300, [2052, 2051, 1025, 700]), (16384, 2048, [16384, 16381, 9000, 2049])):
        bits = rng.integers(min(ends), max(ends) + 1, (4, s_kv)).astype(np.uint32)      # even over the bit patterns
        x = bits.view(np.float32).copy()
        x[:, 5] = np.float32(largest)
        for at, what in ((0, np.uint32(0x7fc00000)), (1, np.uint32(0xffc00000)), (2, np.uint32(0xffffffff)), (3, np.uint32(0x7f800001)),
                         (4, np.uint32(0xff800000))):
            x[:, 8 + at:: 64] = what.view(np.float32)
        if pair:
            x = np.repeat(x, 2, axis=0)
            x[1::2] = np.roll(x[1::2], 64, axis=1)
        _check(np.ascontiguousarray(x), topk, lengths, pair)


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("scale", [1e-44, 1e-38, 1e-30, 1.0, 1e30, 1e38])
def test_intervals_across_zero(scale, pair):
    """Lists of which the sample points below zero while the maximum is positive: scores are counted by value, at scales where the
    distance across is subnormal, ordinary and beyond the largest float, also with many zeros, an infinite maximum, and one that
    leaves all others in one bin."""
    rng = np.random.default_rng(5)
    x = rng.standard_normal((4, 4100)).astype(np.float64) * scale
    x[1] = np.maximum(x[1], 0)
    x[2] = np.round(x[2] / scale * 2) / 2 * scale
    with np.errstate(over="ignore"):
        x = np.clip(x, -3.4028234e38, 3.4028234e38).astype(np.float32)
    x[:, 7::50] = np.nan
    x[:, 9::50] = -np.inf
    x[:, 11::50] = np.float32(-0.0)
    for best in (None, np.inf, np.float32(3.4028234e38)):
        if best is not None:
            x[:, 77] = best
        y = np.ascontiguousarray(np.repeat(x, 2, axis=0) if pair else x)
        if pair:
            y[1::2] = np.roll(y[1::2], 1000, axis=1)
        for topk in (1400, 1650, 2050, 2300, 3000, 3900):
            _check(y, topk, [4100, 4097, 3400, 2051], pair)


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("s_kv", [260, 512, 1028, 2052, 4096])
def test_either_side_of_the_line(s_kv, pair):
    """Rows of which most keys are taken go to the counting kernel: both sides of the line, scores that the interval reaches
    across zero for, negative ones, and lists as long as the row."""
    rank = lambda topk: int(topk / 8 + 4 * (topk / 8) ** 0.5 + 4)
    most = max(t for t in range(s_kv) if rank(t) <= (3 if pair else 4) * s_kv // 32)
    rng = np.random.default_rng(s_kv)
    scores = rng.standard_normal((8 if pair else 4, s_kv)).astype(np.float32)
    for topk in (most - 1, most, most + 1, most + 40, s_kv):
        for x in (scores, np.maximum(scores, 0), scores - 30):
            _check(x, topk, [s_kv, s_kv - 3, s_kv // 2, 1], pair)
