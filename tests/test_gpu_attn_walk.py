"""The decode attention's walk over cached tokens at the edges of its batches and splits, against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [(4, 4, 1), (8, 2, 1), (8, 2, 3), (16, 1, 1)])     # one, four, twelve and sixteen rows a head
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("kind", ["half", "bf16", "e5m2"])
def test_walk(kind, D, heads, monkeypatch):
    from ipex_llm_b200.ops import cuda_ops
    Hq, Hkv, Sq = heads
    dtype = torch.bfloat16 if kind == "bf16" else torch.float16
    u = 2.0 ** -8 if kind == "bf16" else 2.0 ** -11
    g = torch.Generator(device="cuda").manual_seed(D + Hq)
    for S in (3, 15, 16, 17, 63, 64, 65, 130, 257, 520):
        q = torch.randn(2, Hq, Sq, D, device="cuda", generator=g).to(dtype)
        k, v = (torch.randn(2, Hkv, S, D, device="cuda", generator=g).to(dtype) for _ in range(2))
        kk, vv = k, v
        if kind == "e5m2":
            k, v = cuda_ops.quantize_kv_e5m2(k), cuda_ops.quantize_kv_e5m2(v)
            kk, vv = cuda_ops.dequantize_kv_e5m2(k, dtype), cuda_ops.dequantize_kv_e5m2(v, dtype)
        kd, vd = (t.double().repeat_interleave(Hq // Hkv, 1) for t in (kk, vv))
        s = q.double() @ kd.transpose(-1, -2) / math.sqrt(D)
        hidden = torch.arange(S, device="cuda")[None] > torch.arange(S - Sq, S, device="cuda")[:, None]
        p = torch.softmax(s.masked_fill(hidden, float("-inf")), -1)
        ref = p @ vd
        # 32-bit sums and an approximate exponential (2^-20 of the weights, with scores up to a few dozen), then the rounding
        bound = ref.abs() * u + (p @ vd.abs()) * 2.0 ** -17 + 1e-7
        for n in (1, 2, 3, 8):
            monkeypatch.setattr(cuda_ops, "attn_splits", lambda *a, n=n: n)
            out = cuda_ops.sdpa_decode(q, k, v, None, 1.0 / math.sqrt(D), None, None)
            torch.cuda.synchronize()
            assert bool(((out.double() - ref).abs() <= bound).all()), (S, n)


@pytest.mark.parametrize("heads", [(4, 4, 1), (8, 2, 1), (4, 2, 3), (16, 1, 1)])     # one, four, six and sixteen rows a head
@pytest.mark.parametrize("kind", ["half", "e5m2"])
def test_hidden_values_do_not_count(kind, heads, monkeypatch):
    """A value row that a query does not see (left of its window, or of a later query's token) may hold anything."""
    from ipex_llm_b200.ops import cuda_ops
    Hq, Hkv, Sq = heads
    D, window = 128, 50
    g = torch.Generator(device="cuda").manual_seed(Hq + Sq)
    for S in (64, 65, 130, 300):
        q = torch.randn(1, Hq, Sq, D, device="cuda", generator=g).half()
        k, v = (torch.randn(1, Hkv, S, D, device="cuda", generator=g).half() for _ in range(2))
        code = cuda_ops.quantize_kv_e5m2 if kind == "e5m2" else (lambda t: t)
        k, v = code(k), code(v)
        bad = v.clone()
        unseen = S - Sq - window + 1                       # the first query sees the `window` positions from here on
        inf = 0x7C if kind == "e5m2" else float("inf")
        bad[:, :, :unseen] = inf
        if Sq > 1:
            bad[:, :, S - 1] = inf                         # only the last query sees the last position
        for n in (1, 3):
            monkeypatch.setattr(cuda_ops, "attn_splits", lambda *a, n=n: n)
            ref = cuda_ops.sdpa_decode(q, k, v, None, 1.0 / math.sqrt(D), None, window)
            out = cuda_ops.sdpa_decode(q, k, bad, None, 1.0 / math.sqrt(D), None, window)
            torch.cuda.synchronize()
            rows = slice(0, max(1, Sq - 1))
            assert torch.equal(out[:, :, rows], ref[:, :, rows]), (S, n)


@pytest.mark.parametrize("heads", [(4, 4, 1), (8, 2, 3), (16, 1, 1)])               # one, twelve and sixteen rows a head
@pytest.mark.parametrize("kind", ["half", "e5m2"])
@pytest.mark.parametrize("window,cap", [(0, 5.0), (1, 0.0), (50, 0.0), (50, 5.0)])
def test_walk_with_window_and_cap(window, cap, kind, heads, monkeypatch):
    from ipex_llm_b200.ops import cuda_ops
    Hq, Hkv, Sq = heads
    D, dtype, u = 128, torch.float16, 2.0 ** -11
    g = torch.Generator(device="cuda").manual_seed(Hq + window)
    for S in (3, 16, 49, 65, 130, 520):
        q = torch.randn(2, Hq, Sq, D, device="cuda", generator=g).to(dtype) * 3
        k, v = (torch.randn(2, Hkv, S, D, device="cuda", generator=g).to(dtype) for _ in range(2))
        kk, vv = k, v
        if kind == "e5m2":
            k, v = cuda_ops.quantize_kv_e5m2(k), cuda_ops.quantize_kv_e5m2(v)
            kk, vv = cuda_ops.dequantize_kv_e5m2(k, dtype), cuda_ops.dequantize_kv_e5m2(v, dtype)
        kd, vd = (t.double().repeat_interleave(Hq // Hkv, 1) for t in (kk, vv))
        s = q.double() @ kd.transpose(-1, -2) / math.sqrt(D)
        if cap:
            s = cap * torch.tanh(s / cap)
        last = torch.arange(S - Sq, S, device="cuda")[:, None]
        key = torch.arange(S, device="cuda")[None]
        hidden = (key > last) | ((key <= last - window) if window else False)
        p = torch.softmax(s.masked_fill(hidden, float("-inf")), -1)
        ref = p @ vd
        # as above; a capped score carries tanh's error too (2^-22 of the cap, in front of the exponential)
        bound = ref.abs() * u + (p @ vd.abs()) * 2.0 ** -17 + 1e-7
        for n in (1, 2, 8):
            monkeypatch.setattr(cuda_ops, "attn_splits", lambda *a, n=n: n)
            out = cuda_ops.sdpa_decode(q, k, v, None, 1.0 / math.sqrt(D), cap, window)
            torch.cuda.synchronize()
            assert bool(((out.double() - ref).abs() <= bound).all()), (S, n)


def test_splits_fit_the_gpu(monkeypatch):
    from ipex_llm_b200.ops import cuda_ops
    monkeypatch.delenv("IPEX_LLM_ATTN_STEPS", raising=False)
    monkeypatch.delenv("IPEX_LLM_ATTN_MIN_CTAS", raising=False)
    for B in (1, 3, 8, 32, 700):
        for Hkv, rows in ((32, 1), (8, 8), (1, 71)):
            for S in (1, 40, 1000, 100000):
                n = cuda_ops.attn_splits(B, Hkv, S, rows, 128, False, torch.bfloat16)
                per_sm = cuda_ops._attn_ctas_per_sm(128, rows, False, 1)
                assert 1 <= n <= 128 and (n == 1 or n * B * Hkv * -(-rows // 16) <= 148 * per_sm and S // n >= 160)


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("heads", [(4, 4), (8, 1)])
def test_queries_of_any_alignment(heads, D):
    """q rows that begin at two bytes, or lie apart by an odd number of elements, are read one by one: the same results."""
    from ipex_llm_b200.ops import cuda_ops
    Hq, Hkv = heads
    g = torch.Generator(device="cuda").manual_seed(D)
    q = torch.randn(2, Hq, 3, D, device="cuda", generator=g).half()
    k, v = (torch.randn(2, Hkv, 77, D, device="cuda", generator=g).half() for _ in range(2))
    want = cuda_ops.sdpa_decode(q, k, v, None, D ** -0.5, None, None)
    moved = torch.empty(q.numel() + 1, dtype=q.dtype, device="cuda")[1:].view(q.shape).copy_(q)
    apart = torch.empty(*q.shape[:3], D + 3, dtype=q.dtype, device="cuda")[..., :D].copy_(q)
    for other in (moved, apart):
        assert torch.equal(cuda_ops.sdpa_decode(other, k, v, None, D ** -0.5, None, None), want)


@pytest.mark.parametrize("D,rows,fp8,dtype,ctas", [
    (64, 1, False, torch.float16, 5), (64, 1, True, torch.float16, 7), (64, 4, False, torch.float16, 4), (64, 4, True, torch.float16, 4),
    (64, 16, False, torch.float16, 3), (64, 1, False, torch.bfloat16, 4), (64, 4, False, torch.bfloat16, 4),
    (128, 1, False, torch.float16, 4), (128, 1, True, torch.bfloat16, 4), (128, 4, False, torch.float16, 2)])
def test_ctas_that_an_sm_holds(D, rows, fp8, dtype, ctas):
    """The walk waits for memory: short heads, whose registers allow it, keep their CTAs beside one another."""
    from ipex_llm_b200.native import cuda_api as api
    from ipex_llm_b200.ops import cuda_ops
    assert cuda_ops._attn_ctas_per_sm(D, rows, fp8, api.dtype_code(dtype)) >= ctas


def test_walks_that_would_spill_have_a_cta_less():
    """One row of 128 a warp needs 168 registers in bf16, and in fp16 where keys are hidden: three CTAs, not four that spill."""
    from ipex_llm_b200.native import cuda_api as api
    from ipex_llm_b200.ops import cuda_ops
    fp16, bf16 = api.dtype_code(torch.float16), api.dtype_code(torch.bfloat16)
    assert [cuda_ops._attn_ctas_per_sm(128, 1, False, dt, h) for dt in (bf16, fp16) for h in (False, True)] == [3, 3, 4, 3]


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("heads", [(4, 4, 1), (8, 2, 1), (8, 1, 3)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_rotated_queries_of_any_alignment(dtype, heads, D):
    """New tokens behind a cache: queries, keys and rotary values that are read in runs and one by one."""
    import ctypes
    from ipex_llm_b200.native import cuda_api as api
    from ipex_llm_b200.native.lib import cuda_lib, current_stream, ptr
    from ipex_llm_b200.ops import cuda_ops
    Hq, Hkv, Sq = heads
    B, past, u = 2, 77, 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    g = torch.Generator(device="cuda").manual_seed(D + Hq)
    q, kn, vn = (torch.randn(B, Sq, h, D, device="cuda", generator=g).to(dtype) for h in (Hq, Hkv, Hkv))
    k, v = (torch.randn(B, Hkv, past + Sq, D, device="cuda", generator=g).to(dtype) for _ in range(2))
    angle = torch.arange(past + Sq, device="cuda")[:, None] / 100.0 ** (torch.arange(D // 2, device="cuda") * 2 / D)[None]
    cos, sin = angle.cos().contiguous(), angle.sin().contiguous()
    lengths = torch.full((B,), past, dtype=torch.int32, device="cuda")
    lib = cuda_lib()

    def moved(t):
        return torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape).copy_(t)

    def run(qq, cc, ss, n):
        kc, vc, out = k.clone(), v.clone(), torch.empty_like(q)
        scratch, counters = cuda_ops.attn_workspace(q.device, lib.ipex_attn_decode_scratch_floats(B, Hkv, Hq // Hkv, Sq, D, n),
                                                    lib.ipex_attn_decode_counter_ints(B, Hkv, Hq // Hkv, Sq))
        strides = (ctypes.c_int64 * 12)(*qq.stride()[:3], *kn.stride()[:3], *kc.stride()[:3], *out.stride()[:3])
        rc = lib.ipex_attn_decode(ptr(qq), ptr(kn), ptr(vn), ptr(kc), ptr(vc), ptr(out), ptr(lengths), 0, ptr(cc), ptr(ss),
                                  ptr(scratch), ptr(counters), strides, B, Sq, Hq, Hkv, D, n, 1, D, 1, 0, D ** -0.5, 0.0, 0,
                                  api.dtype_code(dtype), 0, current_stream())
        api.check(rc, "attn_decode")
        torch.cuda.synchronize()
        return out, kc

    def rotate(t):                                         # [B, Sq, heads, D] at positions past ..
        c, s = cos[past:past + Sq, None].double(), sin[past:past + Sq, None].double()
        a, b = t.double()[..., :D // 2], t.double()[..., D // 2:]
        return torch.cat([a * c - b * s, b * c + a * s], -1)

    for n in (1, 3):
        want, kc = run(q, cos, sin, n)
        qd = rotate(q).transpose(1, 2)
        kd, vd = (t.double().repeat_interleave(Hq // Hkv, 1) for t in (kc, torch.cat([v[:, :, :past], vn.transpose(1, 2)], 2)))
        hidden = torch.arange(past + Sq, device="cuda")[None] > torch.arange(past, past + Sq, device="cuda")[:, None]
        p = torch.softmax((qd @ kd.transpose(-1, -2) * D ** -0.5).masked_fill(hidden, float("-inf")), -1)
        # rotated queries are rounded to their type (the key that the kernel wrote is read back): every score moves by up to u
        # times its products' magnitude, every weight by twice the largest of that
        move = u * (qd.abs() @ kd.abs().transpose(-1, -2)).amax(-1, keepdim=True) * D ** -0.5
        bound = (p @ vd.abs()) * (torch.expm1(2 * move) + 2.0 ** -16) + (p @ vd).abs() * u + 1e-6
        for qq, cc, ss in ((q, cos, sin), (moved(q), cos, sin), (q, moved(cos), sin), (q, cos, moved(sin)), (moved(q), moved(cos), moved(sin))):
            out, key = run(qq, cc, ss, n)
            assert torch.equal(key, kc)
            assert bool(((out.double().transpose(1, 2) - p @ vd).abs() <= bound).all())
            assert bool(((out.double() - want.double()).abs().transpose(1, 2) <= bound).all())
