"""The product for few rows (a tile's k shared by a cluster) at the edges of its tiles, and the norm in front of it, against
float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

U = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}
# (M, N, K): one to 64 rows on both sides of every column count; fewer k tiles than CTAs in a cluster, a share that is not the
# same for all of them; fewer weight rows than a tile, tiles in a second round with a ragged last one
SHAPES = [(1, 16, 128), (5, 144, 384), (16, 272, 640), (17, 400, 1152), (32, 128, 512), (33, 5008, 256), (64, 1040, 896)]


def _weights(name, N, K, dtype, g):
    from ipex_llm_b200.ops import cuda_ops, cuda_quant
    from ipex_llm_b200.quant import qtypes as qt
    q = qt.qtype_from_name(name)
    packed = cuda_quant.quantize_to_device_layout((torch.randn(N, K, device="cuda", generator=g) * 0.05).to(dtype), q)
    return q, packed, cuda_ops.dequantize_device(packed, (N, K), q, torch.float32).double()


def _at_16_bytes(t):
    """The same bytes at an address that is a multiple of 16 but not of 32."""
    room = torch.empty(t.numel() + 16, dtype=t.dtype, device=t.device)
    room[16:].copy_(t)
    return room[16:]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("name", ["sym_int4", "asym_int4", "nf4", "fp8_e4m3", "fp8_e5m2", "sym_int8"])
def test_few_rows(name, shape, dtype):
    from ipex_llm_b200.ops import cuda_ops, tcgen05_gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    q, packed, w = _weights(name, N, K, dtype, g)
    wf = cuda_ops.QTYPE_TO_WF[q]
    xf = torch.randn(M, K, device="cuda", generator=g)
    bias = torch.randn(N, device="cuda", generator=g).to(dtype)
    res = torch.randn(M, N, device="cuda", generator=g).to(dtype)
    for pairs in (False, True):
        if pairs and 2 * M > tcgen05_gemm.FEW_MAX_ROWS:
            continue
        hi = xf.to(dtype)
        lo = (xf - hi.float()).to(dtype)
        x = torch.stack([hi, lo], 1).reshape(2 * M, K) if pairs else hi
        xd = hi.double() + lo.double() if pairs else hi.double()
        run = lambda **kw: tcgen05_gemm.gemm_few(x, packed, N, K, kw.pop("out"), wf, lut=cuda_ops.lut_for(q, x.device),  # noqa: E731
                                                 pairs=pairs, **kw)
        out, full = (torch.full((M, N), float("nan"), dtype=dtype, device="cuda") for _ in range(2))
        assert run(out=out) and run(out=full, bias=bias, residual=res)
        torch.cuda.synchronize()
        cuda_ops.check_error_flag(x.device)
        mag, ref = xd.abs() @ w.abs().t(), xd @ w.t()
        # roundings of a weight on its way (half a unit each): none where the codes are multiplied, the value of a code book,
        # and value, scale and product (a minimum beside them: bounded by its block's largest weight) where weights are expanded
        codes = pairs or M <= 32 or name.startswith("fp8")
        roundings = 8 if name == "asym_int4" else (1 if name == "nf4" else 0) if codes else 3
        bound = mag * (roundings * U[dtype] + K * 2.0 ** -23) + ref.abs() * U[dtype] + 1e-6
        assert bool(((out.double() - ref).abs() <= bound).all())
        ref2 = ref + bias.double() + res.double()
        assert bool(((full.double() - ref2).abs() <= bound + (ref2.abs() + 4.0) * U[dtype]).all())
        again = torch.empty_like(out)
        run(out=again)
        assert torch.equal(out, again)


@pytest.mark.parametrize("split", range(9))
@pytest.mark.parametrize("shape", [(1, 16, 64), (3, 144, 192), (8, 272, 832), (31, 160, 1088), (40, 400, 2112)])
@pytest.mark.parametrize("name", ["sym_int4", "asym_int4", "nf4", "sym_int8"])
def test_few_rows_shared_by_any_number(name, shape, split):
    """Every number of CTAs to a tile's k (0: chosen), k that ends in half a chunk of 128; minima up to 32 rows are not rounded."""
    from ipex_llm_b200.ops import cuda_ops, tcgen05_gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(K)
    q, packed, w = _weights(name, N, K, torch.float16, g)
    x = torch.randn(M, K, device="cuda", generator=g).half()
    out = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    assert tcgen05_gemm.gemm_few(x, packed, N, K, out, cuda_ops.QTYPE_TO_WF[q], lut=cuda_ops.lut_for(q, x.device), split=split)
    torch.cuda.synchronize()
    cuda_ops.check_error_flag(x.device)
    mag, ref = x.double().abs() @ w.abs().t(), x.double() @ w.t()
    roundings = 1 if name == "nf4" else 8 if name == "asym_int4" and M > 32 else 0
    # (the sums of a minimum's group cancel against those of its codes: up to the block's range times the tokens)
    spread = x.double().abs().sum(1, keepdim=True) * 0.5 * K ** 0.5 * 2.0 ** -23 if name == "asym_int4" else 0.0
    bound = mag * (roundings * U[torch.float16] + K * 2.0 ** -23) + spread + ref.abs() * U[torch.float16] + 1e-6
    assert bool(((out.double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("name,dtype", [("sym_int4", torch.float16), ("fp8_e4m3", torch.bfloat16), ("nf4", torch.float16),
                                        ("nf4", torch.bfloat16), ("asym_int4", torch.float16), ("sym_int8", torch.bfloat16)])
def test_one_to_eight_rows_by_either_way(name, dtype):
    """``gemv_lowbit`` on both sides of its rule, and with operands that only the GEMVs take."""
    from ipex_llm_b200.ops import cuda_ops
    g = torch.Generator(device="cuda").manual_seed(5)
    for N in (528, 8208):
        q, packed, w = _weights(name, N, 384, dtype, g)
        for M in (1, 2, 4, 5, 8):
            x = torch.randn(M, 384, device="cuda", generator=g).to(dtype)
            ref = x.double() @ w.t()
            top = x.double().abs().amax(1, keepdim=True) * w.abs().sum(1)
            bound = top * 2.0 ** -10 + ref.abs() * U[dtype] + 1e-6 if dtype == torch.float16 else top * U[dtype] + ref.abs() * U[dtype]
            for y in (cuda_ops.gemv_lowbit(x, packed, q, N, 384), cuda_ops.gemv_lowbit(x, _at_16_bytes(packed), q, N, 384)):
                assert bool(((y.double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("name", ["sym_int4", "nf4", "fp8_e4m3", "asym_int4"])
def test_linear_of_any_rows(name):
    """A packed linear layer on both sides of its one-call way: rows, a half chunk of k, odd outputs, shapes, rows apart."""
    from ipex_llm_b200.ops.linear import LowBitLinear
    from ipex_llm_b200.quant import qtypes as qt
    from ipex_llm_b200.quant.params import FP4Params
    g = torch.Generator(device="cuda").manual_seed(6)
    K = 384 if name == "fp8_e4m3" else 192
    for N in (16, 328):
        layer = LowBitLinear(K, N, qt.qtype_from_name(name), bias=False)
        w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).half()
        layer._parameters["weight"] = FP4Params(w, requires_grad=False, quantized=False, qtype=layer.qtype).to("cuda")
        dense = layer.weight.dequantize(torch.float32).double()
        for shape in ((1,), (3,), (8,), (9,), (64,), (65,), (2, 4), (0,), (1, 1, 5)):
            x = torch.randn(*shape, K + 8, device="cuda", generator=g).half()[..., :K].requires_grad_()
            with torch.no_grad():
                y = layer(x)
            assert y.shape == (*shape, N) and not y.requires_grad
            ref = x.detach().double() @ dense.t()
            top = x.detach().double().abs().sum(-1, keepdim=True) * float(dense.abs().max())
            assert bool(((y.double() - ref).abs() <= top * 2.0 ** -10 + 1e-3).all())


@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("shape", [(9, 288, 256), (24, 4128, 512)])
def test_few_rows_gated(shape, pairs):
    from ipex_llm_b200.ops import cuda_ops, tcgen05_gemm
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(N)
    q, packed, w = _weights("sym_int4", N, K, torch.float16, g)
    x = torch.randn(2 * M if pairs else M, K, device="cuda", generator=g).half()
    xd = x.double().view(M, 2, K).sum(1) if pairs else x.double()
    out = torch.empty(M, N // 2, dtype=torch.float16, device="cuda")
    assert tcgen05_gemm.gemm_few(x, packed, N, K, out, cuda_ops.QTYPE_TO_WF[q], act=1, pairs=pairs)
    torch.cuda.synchronize()
    cuda_ops.check_error_flag(x.device)
    t = (xd @ w.t()).view(M, N // 32, 2, 16)
    ref = (torch.nn.functional.silu(t[:, :, 0]) * t[:, :, 1]).reshape(M, N // 2)
    # an approximate exponential (2^-10 of the gate) and the rounding of the result
    assert bool(((out.double() - ref).abs() <= ref.abs() * U[torch.float16] + 2.0 ** -10 * t.abs().amax() ** 2 / 8).all())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H", [8, 264, 2048, 4096, 13824, 16384])
def test_rms_norm_rows(H, dtype):
    from ipex_llm_b200.ops import cuda_ops
    g = torch.Generator(device="cuda").manual_seed(H)
    x = torch.randn(5, H, device="cuda", generator=g).to(dtype)
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).to(dtype)
    ref = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-5) * w.double()
    pair = cuda_ops.rms_norm_pairs(x, w, 1e-5).view(5, 2, H).double()
    # the remainder has the type's relative precision, down to its smallest step
    assert bool(((pair.sum(1) - ref).abs() <= ref.abs() * (U[dtype] ** 2 * 2 + 2.0 ** -20) + 2.0 ** -24).all())
    one = cuda_ops.rms_norm(x, w, 1e-5).double()
    assert bool(((one - ref).abs() <= ref.abs() * (2.5 * U[dtype]) + 1e-7).all())    # value and product are rounded


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_norm_pairs_of_any_rows(dtype):
    """Rows that are not packed one after another, and a weight of another type."""
    from ipex_llm_b200.ops import cuda_ops
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(5, 512, device="cuda", generator=g).to(dtype)[:, :256]
    w = 1 + 0.1 * torch.randn(256, device="cuda", generator=g)
    for weight in (w.to(dtype), w):
        pair = cuda_ops.rms_norm_pairs(x, weight, 1e-5)
        assert torch.equal(pair, cuda_ops.rms_norm_pairs(x.contiguous(), weight.to(dtype), 1e-5))
        ref = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-5) * weight.to(dtype).double()
        err = (pair.view(5, 2, 256).double().sum(1) - ref).abs()
        assert bool((err <= ref.abs() * (U[dtype] ** 2 * 2 + 2.0 ** -20) + 2.0 ** -24).all())


def test_norm_pairs_past_the_range_of_half():
    """Value and remainder add up to what a single fp16 number could not hold."""
    from ipex_llm_b200.ops import cuda_ops
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(3, 512, device="cuda", generator=g).half()
    w = torch.full((512,), 30000.0, device="cuda").half()
    ref = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-5) * w.double()
    assert 65504 < float(ref.abs().max()) < 131008
    pair = cuda_ops.rms_norm_pairs(x, w, 1e-5).view(3, 2, 512).double()
    # the remainder of a value past the range is rounded to fp16 itself
    assert bool(((pair.sum(1) - ref).abs() <= ref.abs() * (U[torch.float16] ** 2 * 2 + 2.0 ** -20) +
                 (ref.abs() > 65504) * 65504 * U[torch.float16]).all())


@pytest.mark.parametrize("batch", [9, 20, 32])
def test_decode_steps_of_a_batch(batch):
    """Steps of a batch against the same sequences decoded eight at a time."""
    from transformers import LlamaConfig
    from ipex_llm_b200.engine.decoder_engine import DecoderEngine
    from ipex_llm_b200.transformers import AutoModelForCausalLM
    cfg = LlamaConfig(hidden_size=512, intermediate_size=1408, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=4, vocab_size=1024, max_position_embeddings=512, tie_word_embeddings=False)
    model = AutoModelForCausalLM.from_config(cfg, load_in_low_bit="sym_int4", device="cuda:0", torch_dtype=torch.float16)
    ids = torch.randint(0, 1024, (batch, 24), device="cuda", generator=torch.Generator(device="cuda").manual_seed(batch))

    def steps(rows):
        eng = DecoderEngine(model, max_batch=rows.shape[0], max_len=256, kv_fp8=False)
        eng.prefill(rows)
        out = []
        for i in range(3):
            eng.tokens[:rows.shape[0]] = rows[:, i]
            eng.decode_step(rows.shape[0])
            out.append(eng.logits[:rows.shape[0]].double().clone())
        return torch.stack(out)

    whole = steps(ids)
    parts = torch.cat([steps(ids[s:s + 8]) for s in range(0, batch, 8)], dim=1)
    # both round every activation to fp16 about thirty times on the way: 2^-11 each, and no more than a few of them add up
    assert float((whole - parts).norm() / parts.norm()) < 8 * 2.0 ** -11


def test_batch_whose_weights_begin_at_16_bytes():
    from transformers import LlamaConfig
    from ipex_llm_b200.engine.decoder_engine import DecoderEngine
    from ipex_llm_b200.transformers import AutoModelForCausalLM
    cfg = LlamaConfig(hidden_size=512, intermediate_size=1408, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=4, vocab_size=1024, max_position_embeddings=512, tie_word_embeddings=False)
    model = AutoModelForCausalLM.from_config(cfg, load_in_low_bit="sym_int4", device="cuda:0", torch_dtype=torch.float16)
    ids = torch.randint(0, 1024, (9, 24), device="cuda", generator=torch.Generator(device="cuda").manual_seed(9))

    def step(move):
        eng = DecoderEngine(model, max_batch=9, max_len=256, kv_fp8=False)
        if move:
            eng.layers[1].down.data = _at_16_bytes(eng.layers[1].down.data)
        eng.prefill(ids)
        eng.tokens[:9] = ids[:, 0]
        eng.decode_step(9)
        return eng.logits[:9].double().clone()

    want, got = step(False), step(True)
    assert float((got - want).norm() / want.norm()) < 8 * 2.0 ** -11


# the first four go to the product for few rows, the last two are formats that it would round and stay with the others
@pytest.mark.parametrize("name,dtype", [("sym_int4", torch.float16), ("nf4", torch.float16), ("fp8_e4m3", torch.bfloat16),
                                        ("sym_int8", torch.bfloat16), ("asym_int4", torch.float16), ("nf4", torch.bfloat16)])
@pytest.mark.parametrize("M,K", [(5, 8320), (7, 11008), (8, 8320)])
def test_long_rows_between_dependent_launches(name, dtype, M, K):
    """Five to eight rows of a long contraction: against float64, and in a chain of programmatic launches whose buffers are
    overwritten by the next round."""
    from ipex_llm_b200.ops import cuda_ops, tcgen05_gemm
    from ipex_llm_b200.quant import qtypes
    g = torch.Generator(device="cuda").manual_seed(M + K)
    N = 272
    few = tcgen05_gemm.few_exact(cuda_ops.QTYPE_TO_WF[qtypes.qtype_from_name(name)], dtype, M)
    assert few == (name != "asym_int4" and (name, dtype) != ("nf4", torch.bfloat16))
    few = few and (name in ("sym_int4", "fp8_e4m3") or M * K >= 1 << 16)      # fewer of the others fit beside their kernel's rings
    qu, pu, _ = _weights("sym_int4", K, 384, dtype, g)            # makes the long rows, the same ones every time
    q, packed, w = _weights(name, N, K, dtype, g)
    bias = torch.randn(N, device="cuda", generator=g).to(dtype)
    start = torch.randn(M, 384, device="cuda", generator=g).to(dtype)
    x, y, y2, z = (torch.empty(M, n, dtype=dtype, device="cuda") for n in (K, N, N, 384))

    def chain(pdl):
        z.copy_(start)
        seen = []
        for _ in range(4):
            # the long rows made, read, made again in the same place and read again, beside the first result
            for rows, out, res in ((z, y, z[:, :N]), (start, y2, y)):
                cuda_ops.gemv_lowbit(rows, pu, qu, K, 384, out=x, pdl=pdl)
                cuda_ops.gemv_lowbit(x, packed, q, N, K, out=out, bias=bias, residual=res, pdl=pdl)
                if not pdl:
                    seen.append((x.clone(), res.clone(), out.clone()))
            z[:, :N].copy_(y2 * 0.1)
        return y2.clone(), seen

    want, seen = chain(False)
    torch.cuda.synchronize()
    got, _ = chain(True)
    torch.cuda.synchronize()
    cuda_ops.check_error_flag(x.device)
    if few:
        assert torch.equal(got, want)                             # (kernels that add parts up in any order do not repeat)
    # what a product rounds: see the bounds of the product for few rows above; kernels for one to eight rows hold x in 15 bits
    for xs, zs, ys in seen:
        ref = xs.double() @ w.t() + bias.double() + zs.double()
        mag = xs.double().abs() @ w.abs().t()
        top = xs.double().abs().amax(1, keepdim=True) * w.abs().sum(1)
        bound = mag * ((8 if name == "asym_int4" else 1) * U[dtype] + K * 2.0 ** -23) + top * 2.0 ** -14 + \
            (ref.abs() + 1e-3) * U[dtype]
        assert bool(((ys.double() - ref).abs() <= bound).all())
    moved = cuda_ops.gemv_lowbit(x, _at_16_bytes(packed), q, N, K, bias=bias, residual=z[:, :N])
    torch.cuda.synchronize()
    ref = x.double() @ w.t() + bias.double() + z[:, :N].double()
    top = x.double().abs().amax(1, keepdim=True) * w.abs().sum(1)
    assert bool(((moved.double() - ref).abs() <= top * 2.0 ** -10 + ref.abs() * U[dtype]).all())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("name", ["sym_int4", "asym_int4", "nf4", "fp8_e4m3", "fp8_e5m2", "sym_int8"])
def test_wide_rows_through_long_rings(name, dtype):
    """25 to 64 rows on both sides of their column counts, over more stages than a ring holds, many tiles at once, again and again."""
    from ipex_llm_b200.ops import cuda_ops, tcgen05_gemm
    g = torch.Generator(device="cuda").manual_seed(9)
    N, K = 3088, 4224
    q, packed, w = _weights(name, N, K, dtype, g)
    for M in (24, 25, 32, 33, 48, 49, 64):
        x = torch.randn(M, K, device="cuda", generator=g).to(dtype)
        mag, ref = x.double().abs() @ w.abs().t(), x.double() @ w.t()
        codes = M <= 32 or name.startswith("fp8")
        roundings = (8 if name == "asym_int4" else 3) if not codes else 1 if name == "nf4" else 0
        spread = x.double().abs().sum(1, keepdim=True) * 0.5 * K ** 0.5 * 2.0 ** -23 if name == "asym_int4" else 0.0
        bound = mag * (roundings * U[dtype] + K * 2.0 ** -23) + spread + ref.abs() * U[dtype] + 1e-6
        for split in (0, 1, 5):
            first = None
            for _ in range(6):
                out = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
                assert tcgen05_gemm.gemm_few(x, packed, N, K, out, cuda_ops.QTYPE_TO_WF[q], lut=cuda_ops.lut_for(q, x.device),
                                             split=split, pdl=True)
                first = out if first is None else first
                assert torch.equal(out, first)
            assert bool(((first.double() - ref).abs() <= bound).all())
    cuda_ops.check_error_flag(x.device)


# A kernel that lets its dependents start at once, ends `ns` later and only then leaves the tokens behind.
LATE = r"""
extern "C" __global__ void late(const uint4* from, uint4* to, int n, unsigned long long ns) {
  asm volatile("griddepcontrol.launch_dependents;");
  unsigned long long t0, t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
  t = t0;
  for (int i = 0; i < 1 << 22 && t - t0 < ns; ++i) {
    __nanosleep(1000);
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) to[i] = from[i];
}
"""


def _ok(result):
    assert int(result[0]) == 0, result
    return result[1] if len(result) > 1 else None


@pytest.mark.parametrize("M", [8, 40])
def test_kernel_in_front_may_take_its_time(M):
    """The bounded waits (half a second) count the product's own copies, not how long the kernel in front still runs."""
    import ctypes
    from cuda.bindings import driver, nvrtc
    from ipex_llm_b200.ops import cuda_ops, tcgen05_gemm
    prog = _ok(nvrtc.nvrtcCreateProgram(LATE.encode(), b"late.cu", 0, [], []))
    _ok(nvrtc.nvrtcCompileProgram(prog, 1, [b"--gpu-architecture=sm_100a"]))
    cubin = bytes(_ok(nvrtc.nvrtcGetCUBINSize(prog)))
    _ok(nvrtc.nvrtcGetCUBIN(prog, cubin))
    g = torch.Generator(device="cuda").manual_seed(M)
    N, K = 272, 1152
    q, packed, w = _weights("sym_int4", N, K, torch.float16, g)
    x = torch.randn(M, K, device="cuda", generator=g).half()
    late, out = torch.zeros_like(x), torch.empty(M, N, dtype=torch.float16, device="cuda")
    want = torch.empty_like(out)
    wf = cuda_ops.QTYPE_TO_WF[q]
    assert tcgen05_gemm.gemm_few(x, packed, N, K, want, wf)
    torch.cuda.synchronize()
    module = _ok(driver.cuModuleLoadData(cubin))
    kernel = _ok(driver.cuModuleGetFunction(module, b"late"))
    args = ((x.data_ptr(), late.data_ptr(), x.numel() // 8, 3_000_000_000),
            (ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_uint64))
    _ok(driver.cuLaunchKernel(kernel, 1, 1, 1, 128, 1, 1, 0, torch.cuda.current_stream().cuda_stream, args, 0))
    assert tcgen05_gemm.gemm_few(late, packed, N, K, out, wf, pdl=True)
    torch.cuda.synchronize()
    _ok(driver.cuModuleUnload(module))
    cuda_ops.check_error_flag(x.device)
    assert torch.equal(out, want)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M", [1, 8, 9, 17, 25, 32, 40])
def test_infinite_tokens_of_a_format_with_minima(M, dtype):
    """An infinite token times a weight is an infinity of the weight's sign, whatever its code and its block's minimum are; two of
    both signs are no number; the other rows do not notice."""
    from ipex_llm_b200.ops import cuda_ops, cuda_quant, tcgen05_gemm
    from ipex_llm_b200.quant import qtypes as qt
    g = torch.Generator(device="cuda").manual_seed(M)
    N, K = 272, 832
    q = qt.qtype_from_name("asym_int4")
    # rows of one sign, away from zero: with 4 bits between them, no weight rounds to it
    w = (1 + torch.rand(N, K, device="cuda", generator=g)) * torch.where(torch.arange(N, device="cuda") % 2 == 0, 1, -1)[:, None]
    packed = cuda_quant.quantize_to_device_layout(w.to(dtype), q)
    wd = cuda_ops.dequantize_device(packed, (N, K), q, torch.float32).double()
    x = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    bad = x.clone()
    bad[0, 700] = float("inf")
    bad[M // 2, [3, 130]] = float("-inf")
    if M > 2:
        bad[M - 1, 5], bad[M - 1, 400] = float("inf"), float("-inf")
    ref = bad.double() @ wd.t()
    hit = torch.isinf(bad).any(1)
    for split in (0, 1, 3):
        out, clean = (torch.empty(M, N, dtype=dtype, device="cuda") for _ in range(2))
        assert tcgen05_gemm.gemm_few(bad, packed, N, K, out, cuda_ops.QTYPE_TO_WF[q], split=split)
        assert tcgen05_gemm.gemm_few(x, packed, N, K, clean, cuda_ops.QTYPE_TO_WF[q], split=split)
        torch.cuda.synchronize()
        cuda_ops.check_error_flag(x.device)
        assert torch.equal(out[hit].double().nan_to_num(7.0, 9.0, -9.0), ref[hit].nan_to_num(7.0, 9.0, -9.0))
        assert torch.equal(out[~hit], clean[~hit])


@pytest.mark.parametrize("K", [128, 448, 12288, 12416])
@pytest.mark.parametrize("M", [16, 17, 32])
def test_minima_of_many_stages(M, K):
    """Minima up to 32 rows are not rounded on either side of the row count from which their product is made at the end, and of
    the number of stages that it has room for (96 of a CTA)."""
    from ipex_llm_b200.ops import cuda_ops, tcgen05_gemm
    g = torch.Generator(device="cuda").manual_seed(M + K)
    N = 400
    for dtype in (torch.float16, torch.bfloat16):
        q, packed, w = _weights("asym_int4", N, K, dtype, g)
        x = torch.randn(M, K, device="cuda", generator=g).to(dtype)
        mag, ref = x.double().abs() @ w.abs().t(), x.double() @ w.t()
        spread = x.double().abs().sum(1, keepdim=True) * 0.5 * K ** 0.5 * 2.0 ** -23
        for split in (0, 1, 2):
            out = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
            assert tcgen05_gemm.gemm_few(x, packed, N, K, out, cuda_ops.QTYPE_TO_WF[q], split=split)
            torch.cuda.synchronize()
            assert bool(((out.double() - ref).abs() <= mag * K * 2.0 ** -23 + spread + ref.abs() * U[dtype] + 1e-6).all())
    cuda_ops.check_error_flag(x.device)


@pytest.mark.parametrize("name", ["sym_int4", "asym_int4", "nf4", "fp8_e4m3", "fp8_e5m2", "sym_int8"])
@pytest.mark.parametrize("M,K", [(4, 8320), (5, 8320), (8, 11008)])
def test_rows_of_every_format_between_dependent_launches(name, M, K):
    """Where the product for few rows is the one that runs, a chain of programmatic launches whose buffers are overwritten by the
    next round repeats one without them bit for bit."""
    from ipex_llm_b200.ops import cuda_ops, tcgen05_gemm
    from ipex_llm_b200.quant import qtypes
    g = torch.Generator(device="cuda").manual_seed(M + K)
    N, dtype = 272, torch.float16
    assert tcgen05_gemm.few_faster(cuda_ops.QTYPE_TO_WF[qtypes.qtype_from_name(name)], dtype, M)
    qu, pu, _ = _weights("sym_int8", K, 384, dtype, g)
    q, packed, _ = _weights(name, N, K, dtype, g)
    start = torch.randn(M, 384, device="cuda", generator=g).to(dtype)
    x, y, z = (torch.empty(M, n, dtype=dtype, device="cuda") for n in (K, N, 384))

    def chain(pdl):
        z.copy_(start)
        seen = []
        for _ in range(6):
            cuda_ops.gemv_lowbit(z, pu, qu, K, 384, out=x, pdl=pdl)
            cuda_ops.gemv_lowbit(x, packed, q, N, K, out=y, residual=z[:, :N], pdl=pdl)
            z[:, :N].copy_(y * 0.1)
            seen.append(y.clone())
        return torch.stack(seen)

    want = chain(False)
    assert torch.equal(chain(True), want)
    cuda_ops.check_error_flag(x.device)
