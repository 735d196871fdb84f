"""The product on pairs of SMs (more than 64 token rows) at the edges of its tiles, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (M, N, K): one token more than the narrow kernels take; a half-empty token tile; one row past a tile of 128 and of 256; fewer
# weight rows than one CTA's half; rows that end in the second CTA's half, and in the first; one k block; more units than
# the dequantizers hold in flight; many tiles per pair, so that accumulators and stages wrap
SHAPES = [(65, 16, 128), (129, 272, 256), (257, 400, 640), (191, 144, 1152), (515, 1040, 896), (1030, 5152, 384)]
U = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def _bound(x, w, ref, dtype, roundings, extra=0.0):
    """Rounding of every expanded weight (``roundings`` of half a unit each), 32-bit accumulation, rounding of the result."""
    mag = x.double().abs() @ w.double().abs().t()
    return mag * (roundings * U[dtype] + x.shape[1] * 2.0 ** -24) + (ref.abs() + extra) * U[dtype] + 1e-6


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("name", ["sym_int4", "asym_int4", "nf4", "fp8_e4m3", "fp8_e5m2", "sym_int8", "dense"])
def test_pair_gemm(name, shape, dtype):
    from ipex_llm_b200.ops import cuda_ops, cuda_quant, tcgen05_gemm
    from ipex_llm_b200.quant import qtypes as qt
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K + 8, device="cuda", generator=g).to(dtype)[:, :K]      # rows are not packed one after another
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(dtype)
    bias = torch.randn(N, device="cuda", generator=g).to(dtype)
    res = torch.randn(M, N, device="cuda", generator=g).to(dtype)
    if name == "dense":
        run = lambda **kw: tcgen05_gemm.gemm_dense(x, w, **kw)  # noqa: E731
        roundings = 0
    else:
        q = qt.qtype_from_name(name)
        packed = cuda_quant.quantize_to_device_layout(w, q)
        w = cuda_ops.dequantize_device(packed, (N, K), q, torch.float32)
        run = lambda **kw: tcgen05_gemm.gemm_lowbit(x, packed, q, N, K, **kw)  # noqa: E731
        # scale and product, the code book's value where there is one; a minimum beside a larger scale is bounded by its
        # block's largest weight, which the sum of magnitudes does not know: four more cover blocks of +-3 sigma
        roundings = {"nf4": 3, "asym_int4": 8}.get(name, 2)
    ref = x.double() @ w.double().t()
    out = run()
    full = run(bias=bias, residual=res)
    torch.cuda.synchronize()
    cuda_ops.check_error_flag(x.device)
    assert bool(((out.double() - ref).abs() <= _bound(x, w, ref, dtype, roundings)).all())
    ref2 = ref + bias.double() + res.double()
    assert bool(((full.double() - ref2).abs() <= _bound(x, w, ref2, dtype, roundings, 4.0)).all())
    assert torch.equal(out, run())


@pytest.mark.parametrize("act", [1, 2])
@pytest.mark.parametrize("shape", [(130, 288, 256), (700, 4128, 512)])
def test_pair_gemm_gated(shape, act):
    """Gate and up rows interleaved in tiles of sixteen: act(gate) * up."""
    from ipex_llm_b200.ops import cuda_ops, tcgen05_gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(act + N)
    x = torch.randn(M, K, device="cuda", generator=g).half()
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).half()
    out = tcgen05_gemm.gemm_dense(x, w, act=act)
    torch.cuda.synchronize()
    cuda_ops.check_error_flag(x.device)
    t = (x.double() @ w.double().t()).view(M, N // 32, 2, 16)
    gate = torch.nn.functional.silu(t[:, :, 0]) if act == 1 else \
        torch.nn.functional.gelu(t[:, :, 0], approximate="tanh")
    ref = (gate * t[:, :, 1]).reshape(M, N // 2)
    # 32-bit products of sums, an approximate exponential or tanh (2^-10 of the gate), rounding of the result
    assert bool(((out.double() - ref).abs() <= ref.abs() * U[torch.float16] + 2.0 ** -10 * t.abs().amax() ** 2 / 8).all())
