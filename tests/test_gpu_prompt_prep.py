"""The pass between a prompt's qkv product and its attention, at the edges of its 64-token tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("heads", [(1, 1, 128), (6, 2, 64), (3, 3, 80), (2, 1, 256)])
@pytest.mark.parametrize("B,S", [(1, 1), (2, 63), (1, 64), (3, 65), (2, 130)])
def test_prompt_prep(B, S, heads, fp8, dtype):
    from ipex_llm_b200.ops import cuda_ops
    Hq, Hkv, D = heads
    g = torch.Generator(device="cuda").manual_seed(S + D)
    ld = (Hq + 2 * Hkv) * D + 16                                           # rows are not packed one after another
    qkv = torch.randn(B * S, ld, device="cuda", generator=g).to(dtype)
    before = qkv.clone()
    angle = torch.rand(S + 5, D // 2, device="cuda", generator=g) * 6.28
    cos, sin = angle.cos(), angle.sin()
    kc, vc = (torch.full((B, Hkv, S + 3, D), 7, device="cuda", dtype=torch.uint8 if fp8 else dtype) for _ in range(2))
    vt = cuda_ops.prompt_prep(qkv, kc, vc, cos, sin, B, S, Hq, Hkv, D, True)
    x = before[:, :(Hq + 2 * Hkv) * D].view(B, S, Hq + 2 * Hkv, D)
    a, b = x[..., :Hq + Hkv, : D // 2].double(), x[..., :Hq + Hkv, D // 2:].double()
    c, s = cos[:S, None].double(), sin[:S, None].double()
    ref = torch.cat([a * c - b * s, b * c + a * s], -1)
    got = qkv[:, :(Hq + 2 * Hkv) * D].view(B, S, Hq + 2 * Hkv, D)
    # products and their sum in 32 bits, then the rounding
    u = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    size = torch.cat([a.abs() + b.abs()] * 2, -1)
    assert bool(((got[..., :Hq + Hkv, :].double() - ref).abs() <= ref.abs() * u + size * 2.0 ** -22 + 1e-7).all())
    assert torch.equal(got[..., Hq + Hkv:, :], x[..., Hq + Hkv:, :]) and torch.equal(qkv[:, -16:], before[:, -16:])
    k, v = got[..., Hq:Hq + Hkv, :].transpose(1, 2), got[..., Hq + Hkv:, :].transpose(1, 2)
    code = cuda_ops.quantize_kv_e5m2 if fp8 else (lambda t: t)
    assert torch.equal(kc[:, :, :S], code(k)) and torch.equal(vc[:, :, :S], code(v))
    assert bool((kc[:, :, S:] == 7).all()) and bool((vc[:, :, S:] == 7).all())
    assert torch.equal(vt[..., :S], v.transpose(2, 3)) and bool((vt[..., S:] == 0).all())


@pytest.mark.parametrize("kv_fp8", [False, True])
def test_cache_that_was_changed_between_prompts(kv_fp8):
    """The engine keeps its caches: one whose rows were selected, or whose storage was cut, is not written by raw strides."""
    from transformers import LlamaConfig
    from ipex_llm_b200.engine.decoder_engine import DecoderEngine
    from ipex_llm_b200.transformers import AutoModelForCausalLM
    cfg = LlamaConfig(hidden_size=512, intermediate_size=1408, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=2, vocab_size=1024, max_position_embeddings=512, tie_word_embeddings=False)
    model = AutoModelForCausalLM.from_config(cfg, load_in_low_bit="sym_int4", device="cuda:0", torch_dtype=torch.float16)
    ids = torch.randint(0, 1024, (2, 70), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    eng = DecoderEngine(model, max_batch=2, max_len=256, kv_fp8=kv_fp8)
    want = eng.prefill(ids)
    layer = eng.cache.layers[1]
    layer._k, layer._v = layer._k[:, :, :64].clone(), layer._v[:, :, :64].clone()      # too short by now: it grows again
    got = eng.prefill(ids)
    # the other way rounds where this one does: to fp16, some thirty times on the way
    assert float((got.double() - want.double()).norm() / want.double().norm()) < 8 * 2.0 ** -11 and layer._k.shape[2] >= 70
    layer.batch_select_indices(torch.tensor([0, 1, 1], device="cuda"))
    with pytest.raises(RuntimeError):
        eng.prefill(ids)
