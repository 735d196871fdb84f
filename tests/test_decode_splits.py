"""KV splits of the engine's decode steps as a reply grows (pure host logic)."""
import pytest
import torch


def _engine(monkeypatch, n_heads, n_kv, prompt, batch=1, max_len=4096):
    from ipex_llm_b200.engine.decoder_engine import DecoderEngine
    from ipex_llm_b200.ops import cuda_ops
    monkeypatch.delenv("IPEX_LLM_ATTN_STEPS", raising=False)
    monkeypatch.delenv("IPEX_LLM_ATTN_MIN_CTAS", raising=False)
    monkeypatch.setattr(cuda_ops, "_attn_ctas_per_sm", lambda *a: 2)
    monkeypatch.setattr(cuda_ops, "_sm_count", lambda: 148)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    eng = DecoderEngine.__new__(DecoderEngine)
    eng.n_heads, eng.n_kv, eng.hd, eng.kv_fp8, eng.dtype, eng.max_len = n_heads, n_kv, 128, True, torch.float16, max_len
    eng.past_len = torch.full((batch,), prompt, dtype=torch.int32)
    eng._kv_hint = prompt
    eng._seat_context(prompt)
    return eng


def _reply(eng, steps, new=1):
    counts = []
    for _ in range(steps):
        counts.append(eng._pick_splits(eng.past_len.shape[0], new))
        eng.past_len += new
    return counts


@pytest.mark.parametrize("heads", [(32, 32), (64, 8), (8, 1)])
@pytest.mark.parametrize("prompt", [16, 32, 100, 700])
def test_a_long_reply_gets_its_splits(monkeypatch, heads, prompt):
    from ipex_llm_b200.ops import cuda_ops
    eng = _engine(monkeypatch, *heads, prompt)
    counts = _reply(eng, 2000)
    wave = 148 * 2 // heads[1]
    for done, n in enumerate(counts):
        ctx = prompt + done
        # never far from what a prompt of this length would get, and no idle GPU behind a walk of some hundred tokens (192 is
        # where a walk of single rows is split, in the middle of a window of up to 73)
        assert n <= wave and (ctx < 192 + 37 or n >= min(4, wave))
        low, high = (cuda_ops.attn_splits(1, heads[1], c, heads[0] // heads[1], 128, True, torch.float16)
                     for c in (ctx * 3 // 4, ctx * 3 // 2 + 64))
        assert low <= n <= high, (ctx, n)
    assert counts == sorted(counts) and len(set(counts)) <= 7            # each is a captured graph
    assert counts[1999] >= min(8, wave)


def test_the_length_is_read_once_a_window(monkeypatch):
    """The same continuation again, or drafts that are taken back: the count stays, and the device is asked rarely."""
    eng = _engine(monkeypatch, 32, 32, 1024)
    first, reads = eng._pick_splits(1), []
    seat = eng._seat_context
    monkeypatch.setattr(eng, "_seat_context", lambda n: (reads.append(n), seat(n)), raising=False)
    for _ in range(1000):
        eng.past_len.fill_(1024)
        assert set(_reply(eng, 4)) == {first}
    assert 0 < len(reads) <= 4000 // 512 and max(reads) <= 1028 + 1
    eng.past_len.fill_(1024)
    for _ in range(200):
        eng._pick_splits(1, 8)                                           # a verification of eight tokens; three are kept
        eng.past_len += 3
    assert eng._kv_from <= 1024 + 600 and eng._kv_until >= 1024 + 600


def test_few_splits_are_four(monkeypatch):
    from ipex_llm_b200.ops import cuda_ops
    monkeypatch.delenv("IPEX_LLM_ATTN_STEPS", raising=False)
    monkeypatch.delenv("IPEX_LLM_ATTN_MIN_CTAS", raising=False)
    monkeypatch.setattr(cuda_ops, "_attn_ctas_per_sm", lambda *a: 2)
    monkeypatch.setattr(cuda_ops, "_sm_count", lambda: 148)
    for Hkv, rows, start in ((32, 1, 192), (8, 8, 96), (2, 7, 96), (1, 1, 192)):
        got = [cuda_ops.attn_splits(1, Hkv, kv, rows, 128, True, torch.float16) for kv in range(1, 5000)]
        assert got[:start - 1] == [1] * (start - 1) and got[start - 1] == 4 and got == sorted(got)
    assert cuda_ops.attn_splits(3, 32, 400, 1, 128, True, torch.float16) == 3        # what fits at once
    assert cuda_ops.attn_splits(8, 32, 400, 1, 128, True, torch.float16) == 1
    # rows of 256 by fours take shorter walks
    assert [cuda_ops.attn_splits(1, 1, 700, rows, D, True, torch.float16) for rows, D in ((8, 256), (16, 128), (16, 256))] == \
        [4, 4, 6]
