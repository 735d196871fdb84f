"""What the product for few rows refuses: it builds a tensor map of ``x``, and writes ``out``, from the sizes it is given."""
import pytest
import torch

M, N, K = 5, 32, 128


def _operands(pairs):
    f16 = dict(dtype=torch.float16)
    return dict(x=torch.zeros(2 * M if pairs else M, K, **f16), w_data=torch.zeros(4096 + 32, dtype=torch.uint8),
                out=torch.zeros(M, N, **f16), bias=torch.zeros(N, **f16), residual=torch.zeros(M, N, **f16))


BAD = {
    "fewer rows": lambda o: o.update(x=o["x"][:-1]),
    "more rows": lambda o: o.update(out=o["out"][:-1], residual=o["residual"][:-1]),
    "shorter rows": lambda o: o.update(x=o["x"][:, :K - 8]),
    "rows with gaps": lambda o: o.update(x=torch.zeros(o["x"].shape[0], 2 * K, dtype=torch.float16)[:, ::2]),
    "rows of an odd stride": lambda o: o.update(x=torch.zeros(o["x"].shape[0], K + 4, dtype=torch.float16)[:, :K]),
    "rows that begin at 8 bytes": lambda o: o.update(x=torch.zeros(o["x"].shape[0], K + 8, dtype=torch.float16)[:, 4:K + 4]),
    "rows in 32 bits": lambda o: {k: o.update({k: o[k].float()}) for k in ("x", "out", "bias", "residual")},
    "an output in 32 bits": lambda o: o.update(out=o["out"].float()),
    "an output with gaps": lambda o: o.update(out=torch.zeros(M, 2 * N, dtype=torch.float16)[:, ::2]),
    "an output that is too narrow": lambda o: o.update(out=o["out"][:, :N - 1]),
    "a weight that begins at 16 bytes": lambda o: o.update(
        w_data=o["w_data"][(16 - o["w_data"].data_ptr()) % 32:]),
    "a bias that is too short": lambda o: o.update(bias=o["bias"][:-1]),
    "a bias of another type": lambda o: o.update(bias=o["bias"].float()),
    "a bias with gaps": lambda o: o.update(bias=torch.zeros(2 * N, dtype=torch.float16)[::2]),
    "a residual of fewer rows": lambda o: o.update(residual=o["residual"][:-1]),
    "a residual that is too narrow": lambda o: o.update(residual=o["residual"][:, :-1]),
    "a residual of another type": lambda o: o.update(residual=o["residual"].bfloat16()),
}


@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("what", sorted(BAD))
def test_refused(what, pairs):
    from ipex_llm_b200.native import cuda_api as api
    from ipex_llm_b200.ops import tcgen05_gemm
    o = _operands(pairs)
    o["w_data"] = o["w_data"][-o["w_data"].data_ptr() % 32:]
    BAD[what](o)
    assert tcgen05_gemm.gemm_few(o["x"], o["w_data"], N, K, o["out"], api.WF_SYM_INT4, bias=o["bias"], residual=o["residual"],
                                 pairs=pairs) is False


def test_pairs_need_two_rows_for_each_token():
    from ipex_llm_b200.native import cuda_api as api
    from ipex_llm_b200.ops import tcgen05_gemm
    o = _operands(False)
    o["w_data"] = o["w_data"][-o["w_data"].data_ptr() % 32:]
    assert tcgen05_gemm.gemm_few(o["x"], o["w_data"], N, K, o["out"], api.WF_SYM_INT4, pairs=True) is False


def test_who_takes_one_to_eight_rows():
    """The product for few rows where it is the faster one: measured at these sizes."""
    from ipex_llm_b200.native import cuda_api as api
    from ipex_llm_b200.ops.tcgen05_gemm import few_faster
    f16, bf16 = torch.float16, torch.bfloat16
    four = [(4096, 4096), (8192, 8192), (4096, 11008), (5120, 13824)]
    gemv = [(22016, 4096), (28672, 8192), (5120, 5120), (10240, 4096)]
    for dtype in (f16, bf16):
        assert all(few_faster(api.WF_SYM_INT4, dtype, 4, *s) for s in four) and not any(few_faster(api.WF_SYM_INT4, dtype, 4, *s) for s in gemv)
        assert few_faster(api.WF_FP8_E4M3, dtype, 4, 22016, 4096) and not few_faster(api.WF_FP8_E4M3, dtype, 4, 5120, 5120)
        for s in four + gemv:
            assert not any(few_faster(wf, dtype, rows, *s) for wf in (api.WF_SYM_INT4, api.WF_FP8_E4M3) for rows in (1, 2, 3))
            assert all(few_faster(wf, dtype, 5, *s) for wf in (api.WF_SYM_INT4, api.WF_FP8_E4M3, api.WF_INT8))
            assert few_faster(api.WF_ASYM_INT4, dtype, 1, *s) and few_faster(api.WF_FP8_E5M2, dtype, 1, *s)
            assert few_faster(api.WF_LUT4, dtype, 1, *s) == (dtype == f16)
    assert few_faster(api.WF_INT8, f16, 1, 5120, 5120) and few_faster(api.WF_INT8, bf16, 1, 4096, 4096)
    assert not few_faster(api.WF_INT8, bf16, 1, 5120, 5120)


def test_rows_that_only_the_general_way_takes_are_not_prepared_for(monkeypatch):
    """bf16 code books of one to eight rows: known before an output is made or a library is asked."""
    from ipex_llm_b200.native import cuda_api as api
    from ipex_llm_b200.ops import cuda_ops

    def asked(*a, **k):
        raise AssertionError("prepared for a call that is refused")

    for name in ("cuda_lib", "lut_for", "error_flag"):
        monkeypatch.setattr(cuda_ops, name, asked)
    x = torch.zeros(3, K, dtype=torch.bfloat16)
    assert cuda_ops._linear_rows(x, None, 3, N, K, api.WF_LUT4) is None
    assert cuda_ops._linear_rows(x, None, 3, 5120, K, api.WF_INT8) is None
