"""What the pass between a prompt's qkv product and its attention refuses (it writes the cache by raw strides)."""
import pytest
import torch

B, S, HQ, HKV, D = 2, 40, 4, 2, 32


def _operands(dtype=torch.float16, cache=None):
    cache = cache or dtype
    return dict(qkv=torch.zeros(B * S, (HQ + 2 * HKV) * D, dtype=dtype), k_cache=torch.zeros(B, HKV, 64, D, dtype=cache),
                v_cache=torch.zeros(B, HKV, 64, D, dtype=cache), cos=torch.zeros(64, D // 2), sin=torch.zeros(64, D // 2))


BAD = {
    "fewer rows in the cache": lambda o: o.update(k_cache=o["k_cache"][:1], v_cache=o["v_cache"][:1]),
    "a cache that is too short": lambda o: o.update(k_cache=o["k_cache"][:, :, :S - 1], v_cache=o["v_cache"][:, :, :S - 1]),
    "fewer heads in the cache": lambda o: o.update(k_cache=o["k_cache"][:, :1], v_cache=o["v_cache"][:, :1]),
    "another head size": lambda o: o.update(k_cache=o["k_cache"][..., :16], v_cache=o["v_cache"][..., :16]),
    "a shorter value cache": lambda o: o.update(v_cache=o["v_cache"][:, :, :S - 1]),
    "other strides of the values": lambda o: o.update(v_cache=torch.zeros(B, 64, HKV, D, dtype=torch.float16).transpose(1, 2)),
    "rows that are not contiguous": lambda o: o.update(
        k_cache=torch.zeros(B, HKV, D, 64, dtype=torch.float16).transpose(2, 3),
        v_cache=torch.zeros(B, HKV, D, 64, dtype=torch.float16).transpose(2, 3)),
    "a cache of another type": lambda o: o.update(k_cache=o["k_cache"].float(), v_cache=o["v_cache"].float()),
    "values of another type": lambda o: o.update(v_cache=o["v_cache"].to(torch.uint8)),
    "fewer angles than tokens": lambda o: o.update(cos=o["cos"][:S - 1], sin=o["sin"][:S - 1]),
    "angles in half precision": lambda o: o.update(cos=o["cos"].half(), sin=o["sin"].half()),
    "angles of another head size": lambda o: o.update(cos=torch.zeros(64, D), sin=torch.zeros(64, D)),
    "angles with gaps": lambda o: o.update(cos=torch.zeros(64, D)[:, ::2], sin=torch.zeros(64, D)[:, ::2]),
    "fewer tokens": lambda o: o.update(qkv=o["qkv"][:-1]),
    "fewer heads": lambda o: o.update(qkv=o["qkv"][:, D:]),
}


@pytest.mark.parametrize("what", sorted(BAD))
def test_refused(what):
    from ipex_llm_b200.ops import cuda_ops
    o = _operands()
    BAD[what](o)
    with pytest.raises(ValueError):
        cuda_ops.prompt_prep(**o, B=B, S=S, Hq=HQ, Hkv=HKV, D=D, transpose_v=True)


def test_what_a_cache_layer_has_to_hold():
    from ipex_llm_b200.ops import cuda_ops
    for dtype, cache in ((torch.float16, torch.float16), (torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.uint8)):
        o = _operands(dtype, cache)
        assert cuda_ops.prompt_prep_fits(o["k_cache"], o["v_cache"], o["cos"], o["sin"], dtype, B, S, HKV, D)
        assert cuda_ops.prompt_prep_fits(o["k_cache"], o["v_cache"], o["cos"], o["sin"], dtype, B, 64, HKV, D)
        assert not cuda_ops.prompt_prep_fits(o["k_cache"], o["v_cache"], o["cos"], o["sin"], dtype, B, 65, HKV, D)
        assert not cuda_ops.prompt_prep_fits(o["k_cache"], o["v_cache"], o["cos"], o["sin"], dtype, B + 1, S, HKV, D)
        assert not cuda_ops.prompt_prep_fits(None, None, o["cos"], o["sin"], dtype, B, S, HKV, D)
