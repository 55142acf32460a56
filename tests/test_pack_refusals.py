"""What the fused packers refuse, with the message that names the rule, and what they take: the checks stand in the extension,
ahead of any device work."""
import pytest
import torch

from mxdsa_b200 import quantize as Z

Q, KV, PAGES = (2, 64, 512), (6, 1, 512), (2, 4, 1, 512)
OPS = [(Z.pack_dual_q64, Q, "q"), (Z.pack_dual_prefill_kv64, KV, "kv"), (Z.pack_dual_decode_kv_pages, PAGES, "kv")]
IDS = ["q", "prefill_kv", "decode_pages"]


@pytest.mark.parametrize("op,shape,name", OPS, ids=IDS)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_host_tensors(op, shape, name, dtype):
    with pytest.raises(RuntimeError, match=name + " must be on CUDA"):
        op(torch.zeros(shape, dtype=dtype))


@pytest.mark.parametrize("op,shape,needle", [
    (Z.pack_dual_prefill_kv64, (6, 512), r"\[s_kv, 1, 512\]"),
    (Z.pack_dual_prefill_kv64, (6, 2, 512), r"\[s_kv, 1, 512\]"),
    (Z.pack_dual_prefill_kv64, PAGES, r"\[s_kv, 1, 512\]"),
    (Z.pack_dual_decode_kv_pages, KV, r"\[pages, page_size, 1, 512\]"),
    (Z.pack_dual_decode_kv_pages, (2, 4, 2, 512), r"\[pages, page_size, 1, 512\]"),
    (Z.pack_dual_decode_kv_pages, (2, 2, 4, 1, 512), r"\[pages, page_size, 1, 512\]")])
def test_kv_shapes(op, shape, needle):      # looked at ahead of the device
    with pytest.raises(RuntimeError, match="kv must have shape " + needle):
        op(torch.zeros(shape))


@pytest.mark.parametrize("op", [o[0] for o in OPS], ids=IDS)
@pytest.mark.parametrize("thing", [[[1.0] * 512], "kv", 3])
def test_things_that_are_no_tensors(op, thing):
    with pytest.raises((TypeError, RuntimeError)):
        op(thing)


@pytest.mark.gpu
@pytest.mark.parametrize("op,shape,name", OPS, ids=IDS)
def test_dtypes_and_last_dimension(op, shape, name):
    for dtype in (torch.float16, torch.float64, torch.int32, torch.uint8, torch.float8_e4m3fn):
        with pytest.raises(RuntimeError, match=name + " must be bf16 or fp32"):
            op(torch.zeros(shape, device="cuda").to(dtype))
    for last in (511, 513, 256, 0):
        with pytest.raises(RuntimeError, match=name + " must have a last dimension of 512"):
            op(torch.zeros(shape[:-1] + (last,), device="cuda"))
    if name == "q":
        with pytest.raises(RuntimeError, match="q must have a last dimension of 512"):
            op(torch.zeros(512, device="cuda"))


@pytest.mark.gpu
@pytest.mark.parametrize("op,shape,name", OPS, ids=IDS)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_strides_and_no_rows_are_taken(op, shape, name, dtype):
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(shape, device="cuda", generator=g).to(dtype)
    want = op(x)
    assert want.shape == shape[:-1] + (528,) and want.dtype == torch.uint8 and want.is_contiguous() and not want.requires_grad
    spread = torch.randn(shape[:-1] + (1024,), device="cuda", generator=g).to(dtype)
    spread[..., ::2] = x
    assert torch.equal(op(spread[..., ::2]), want)                      # a stride of two elements
    wide = torch.randn((shape[0] * 2,) + shape[1:], device="cuda", generator=g).to(dtype)
    wide[::2] = x
    assert torch.equal(op(wide[::2]), want)                             # every other row, token or page
    assert torch.equal(op(x.clone().requires_grad_()), want)
    if name == "kv":                                                    # (no rows of q: refused by the library)
        assert op(x[:0]).shape == (0,) + shape[1:-1] + (528,)


def test_row_constants():
    from mxdsa_b200 import packing
    assert Z.D == packing.D_HEAD and Z.ROW == packing.D_HEAD + 16
