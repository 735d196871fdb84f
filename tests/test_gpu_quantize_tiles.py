"""The GPU quantizer and its inverse at the edges of their tiles (16 rows x 128 k), against the host library."""
import pytest
import torch

pytestmark = pytest.mark.gpu

NAMES = ["sym_int4", "asym_int4", "nf4", "fp4", "fp8_e4m3", "fp8_e5m2", "sym_int8"]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(1, 64), (16, 128), (17, 192), (31, 320), (80, 1088), (2500, 128)])
@pytest.mark.parametrize("name", NAMES)
def test_pack_and_expand(name, shape, dtype):
    from ipex_llm_b200.ops.cuda_ops import dequantize_device
    from ipex_llm_b200.ops.cuda_quant import quantize_to_device_layout
    from ipex_llm_b200.quant import qtypes as qt
    from ipex_llm_b200.quant.params import FP4Params, ggml_convert_fp32, ggml_convert_qtype
    N, K = shape
    if name.startswith("fp8"):
        K = (K + 127) // 128 * 128
    q = qt.qtype_from_name(name)
    g = torch.Generator().manual_seed(N * 7 + K)
    w = (torch.randn(N, K, generator=g) * 0.02).to(dtype)
    w[0, :64] = 0.0                                             # a block without a scale
    dev = w.cuda()
    packed = quantize_to_device_layout(dev, q)
    # rows that are neither aligned to 16 bytes nor packed one after another take the element-wise loads: same bytes
    wide = torch.zeros(N, K + 3, dtype=dtype, device="cuda")
    wide[:, 1:K + 1] = dev
    assert torch.equal(packed, quantize_to_device_layout(wide[:, 1:K + 1], q))
    # a used buffer is overwritten whole, padding included
    assert torch.equal(packed, quantize_to_device_layout(dev, q, out=torch.full_like(packed, 0xA5)))
    assert torch.equal(packed, FP4Params(dev, requires_grad=False, quantized=False, qtype=q).to("cuda").data)
    back = dequantize_device(packed, (N, K), q, torch.float32).cpu()
    host = ggml_convert_fp32(ggml_convert_qtype(w.float().contiguous(), q).view(torch.uint8), w.shape, w.numel(), q)
    if name.startswith("fp8"):
        # ties of the two roundings to fp8 may fall to either neighbour: half a unit of three (two) mantissa bits each
        step = w.float().abs() * (2.0 ** -3 if name == "fp8_e4m3" else 2.0 ** -2) + w.float().abs().amax() * 2.0 ** -14
        assert bool(((back - host).abs() <= step).all())
    else:
        assert torch.equal(back, host)
    for half in (torch.float16, torch.bfloat16):
        assert torch.equal(dequantize_device(packed, (N, K), q, half).cpu(), back.to(half))


def test_slices_between_other_bytes():
    """Packed bytes that begin anywhere in a larger buffer."""
    from ipex_llm_b200.ops.cuda_ops import dequantize_device
    from ipex_llm_b200.ops.cuda_quant import quantize_to_device_layout
    from ipex_llm_b200.quant import qtypes as qt
    w = torch.randn(40, 256, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).half()
    packed = quantize_to_device_layout(w, qt.SYM_INT4)
    buf = torch.full((packed.numel() + 8,), 0xA5, dtype=torch.uint8, device="cuda")
    part = buf[4:4 + packed.numel()]
    assert torch.equal(quantize_to_device_layout(w, qt.SYM_INT4, out=part), packed) and torch.equal(part, packed)
    assert bool((buf[:4] == 0xA5).all()) and bool((buf[-4:] == 0xA5).all())
    dense = dequantize_device(packed, (40, 256), qt.SYM_INT4, torch.float16)
    assert torch.equal(dequantize_device(part, (40, 256), qt.SYM_INT4, torch.float16), dense)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("name", ["sym_int4", "fp8_e4m3"])
def test_expand_into_rows_of_any_alignment(name, dtype):
    """Rows at multiples of 32, 16 and fewer bytes take stores of their own width, and leave the gaps between them alone."""
    from ipex_llm_b200.native import cuda_api as api
    from ipex_llm_b200.native.lib import cuda_lib, current_stream, ptr
    from ipex_llm_b200.ops.cuda_ops import QTYPE_TO_WF, dequantize_device
    from ipex_llm_b200.ops.cuda_quant import quantize_to_device_layout
    from ipex_llm_b200.quant import qtypes as qt
    N, K, q = 37, 384, qt.qtype_from_name(name)
    packed = quantize_to_device_layout(torch.randn(N, K, device="cuda").half(), q)
    dense = dequantize_device(packed, (N, K), q, dtype)
    for gap in (0, 32, 16 // dense.element_size(), 3):
        buf = torch.full((N, K + gap), 7.0, dtype=dtype, device="cuda")
        rc = cuda_lib().ipex_dequantize_tiles(ptr(packed), ptr(buf), N, K, K + gap, QTYPE_TO_WF[q], None, api.dtype_code(dtype),
                                              current_stream())
        assert rc == 0 and torch.equal(buf[:, :K], dense) and bool((buf[:, K:] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("name", ["sym_int4", "asym_int4", "nf4", "fp4", "sym_int8"])
def test_blocks_whose_scale_or_code_is_a_close_call(name, dtype):
    """Largest values of both signs in either order, zeros of either sign, elements on and between the values of a code book."""
    from ipex_llm_b200.ops.cuda_ops import dequantize_device
    from ipex_llm_b200.ops.cuda_quant import quantize_to_device_layout
    from ipex_llm_b200.quant import qtypes as qt
    from ipex_llm_b200.quant.params import ggml_convert_fp32, ggml_convert_qtype
    q = qt.qtype_from_name(name)
    w = torch.randn(24, 128, generator=torch.Generator().manual_seed(2)) * 0.1
    w[0, 5], w[0, 9], w[1, 5], w[1, 9] = 0.5, -0.5, -0.5, 0.5
    w[2, 0], w[2, 63], w[3, 0], w[3, 63] = -2.0, 2.0, 2.0, -2.0
    w[4], w[5], w[5, 1::2] = 0.0, 0.0, -0.0
    w[6] = torch.where(torch.arange(128) % 2 == 0, -1.0, 1.0)
    from ipex_llm_b200.ops.cuda_ops import _FP4, _NF4
    for row, book in ((7, _NF4), (8, [v / 6 for v in _FP4])):
        book = torch.tensor(sorted(book))
        w[row, :16], w[row, 16:31], w[row, 64], w[row, 65:81] = book, (book[1:] + book[:-1]) / 2, 1.0, book * (1 + 2.0 ** -9)
        w[row, 0] = 1.0
    w[9:] = (w[9:] * 30).round() / 8                          # many equal magnitudes
    w = w.to(dtype)
    packed = quantize_to_device_layout(w.cuda(), q)
    host = ggml_convert_fp32(ggml_convert_qtype(w.float().contiguous(), q).view(torch.uint8), w.shape, w.numel(), q)
    assert torch.equal(dequantize_device(packed, w.shape, q, torch.float32).cpu(), host)
    room = torch.empty(packed.numel() + 16, dtype=torch.uint8, device="cuda")
    assert torch.equal(quantize_to_device_layout(w.cuda(), q, out=room[16:]), packed)
