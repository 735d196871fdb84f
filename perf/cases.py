"""The workloads whose speed is watched: low-bit language models as a user of this package runs them.

A case is one call (or one short run of calls) of a public entry point on seeded data, at sizes that the package's own
benchmarks, tests and model configurations use:

``linear``    one ``LowBitLinear`` of a converted module: what every converted model is made of, one row while a token is
              decoded, some dozens or thousands of rows for a batch or a prompt.
``decode``    a converted decoder that serves ``batch`` sequences: after a prompt of ``ctx`` tokens, ``steps`` calls of
              ``model.decode_step`` with the tokens that the host chose, the logits kept for the sampler.
``prompt``    the prompt pass of the same engine: logits of the last position and a filled KV cache.
``experts``   a converted bank of mixture-of-experts feed-forwards on routed tokens.
``train``     forward and backward of a QLoRA step: frozen low-bit base, adapters on every projection, checkpointing on.
``quantize``  packing of a weight that is already on the GPU, and expanding it again.

``layers`` is the depth of the model (32 is a whole Llama-2-7B; where the depth is less, every layer has the full size of
the named model).  ``kv`` is how keys and values are cached: ``e5m2`` is what up to eight sequences get by default, ``half``
(the model's type) what larger batches get and what IPEX_LLM_QUANTIZE_KV_CACHE=0 asks for.
"""
import math
import os
import zlib

import torch
import torch.nn.functional as F
import torch.utils.checkpoint

ARCHS = {
    "llama2-7b": dict(hidden_size=4096, intermediate_size=11008, num_attention_heads=32, num_key_value_heads=32,
                      vocab_size=32000, rope_theta=10000.0),
    "llama2-13b": dict(hidden_size=5120, intermediate_size=13824, num_attention_heads=40, num_key_value_heads=40,
                       vocab_size=32000, rope_theta=10000.0),
    "llama3-70b": dict(hidden_size=8192, intermediate_size=28672, num_attention_heads=64, num_key_value_heads=8,
                       vocab_size=128256, rope_theta=500000.0),
}
EPS = 1e-5
STD = 0.02
LORA_R, LORA_ALPHA = 8, 16
PROJECTIONS = ("q_proj", "k_proj", "v_proj", "o_proj", "gate_proj", "up_proj", "down_proj")


def listed():
    return [
        # one projection for one token: the smallest call, where latency and launches count
        dict(name="linear-1-row", kind="linear", rows=1, n=4096, k=4096, low_bit="sym_int4", dtype="float16"),
        # an odd number of rows (a ragged batch, a drafted continuation) in the code-book format and bf16
        dict(name="linear-37-rows", kind="linear", rows=37, n=11008, k=4096, low_bit="nf4", dtype="bfloat16"),
        # the headline: Llama-2-7B int4, one sequence, a 1024-token prompt behind it
        dict(name="decode-7b", kind="decode", arch="llama2-7b", layers=32, low_bit="sym_int4", dtype="float16", batch=1,
             ctx=1024, steps=4, kv="e5m2"),
        # the same model serving a small batch with an odd context
        dict(name="decode-7b-batch-8", kind="decode", arch="llama2-7b", layers=32, low_bit="sym_int4", dtype="float16",
             batch=8, ctx=517, steps=4, kv="e5m2"),
        # and a batch that a server fills
        dict(name="decode-7b-batch-32", kind="decode", arch="llama2-7b", layers=32, low_bit="sym_int4", dtype="float16",
             batch=32, ctx=256, steps=4, kv="half"),
        # layers of the 70B model: fp8 weights, bf16, eight query heads to a key head
        dict(name="decode-70b-layers", kind="decode", arch="llama3-70b", layers=8, low_bit="fp8_e4m3", dtype="bfloat16",
             batch=1, ctx=2048, steps=4, kv="e5m2"),
        # first token of the headline model
        dict(name="prompt-7b", kind="prompt", arch="llama2-7b", layers=32, low_bit="sym_int4", dtype="float16", batch=1,
             tokens=1024, kv="e5m2"),
        # a batch of short prompts with an odd length, fp8 weights
        dict(name="prompt-7b-ragged", kind="prompt", arch="llama2-7b", layers=8, low_bit="fp8_e4m3", dtype="bfloat16",
             batch=3, tokens=333, kv="half"),
        # a long prompt: attention weighs in
        dict(name="prompt-7b-long", kind="prompt", arch="llama2-7b", layers=8, low_bit="sym_int4", dtype="float16", batch=1,
             tokens=4096, kv="half"),
        # Mixtral's feed-forward for a batch of eight sequences
        dict(name="experts-8-tokens", kind="experts", experts=8, top_k=2, hidden=4096, inter=14336, tokens=8,
             low_bit="sym_int4", dtype="float16"),
        # QLoRA as the finetuning benchmark runs it, four layers of the 13B model
        dict(name="train-13b-layers", kind="train", arch="llama2-13b", layers=4, low_bit="nf4", dtype="bfloat16", batch=4,
             tokens=512),
        # loading: one feed-forward matrix is packed on the GPU (and expanded, as merging adapters does)
        dict(name="quantize", kind="quantize", n=11008, k=4096, low_bit="sym_int4", dtype="float16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges; model cases are cut to a few layers."""
    kind = rng.choice(("linear", "linear", "decode", "decode", "prompt", "prompt", "experts", "train", "quantize"))
    dtype = rng.choice(("float16", "bfloat16"))
    if kind == "linear":
        low_bit = rng.choice(("sym_int4", "asym_int4", "nf4", "fp8_e4m3", "sym_int8"))
        block = 128 if low_bit == "fp8_e4m3" else 64
        return dict(kind=kind, rows=_log_int(rng, 1, 4096), n=32 * rng.randint(16, 700),
                    k=block * rng.randint(1024 // block, 11520 // block), low_bit=low_bit, dtype=dtype)
    if kind == "decode":
        # the larger models at one or two sequences: with more, a row of their feed-forward's width no longer fits beside
        # the others in the decode kernels, and the engine refuses
        arch = rng.choice(("llama2-7b", "llama2-7b", "llama2-13b", "llama3-70b"))
        batch = _log_int(rng, 1, 32) if arch == "llama2-7b" else rng.randint(1, 2)
        return dict(kind=kind, arch=arch, layers=rng.randint(2, 4),
                    low_bit=rng.choice(("sym_int4", "fp8_e4m3", "nf4")), dtype=dtype, batch=batch,
                    ctx=_log_int(rng, 32, 2048), steps=4, kv=rng.choice(("e5m2", "half")) if batch <= 8 else "half")
    if kind == "prompt":
        return dict(kind=kind, arch=rng.choice(("llama2-7b", "llama2-13b", "llama3-70b")), layers=rng.randint(2, 4),
                    low_bit=rng.choice(("sym_int4", "fp8_e4m3", "nf4")), dtype=dtype, batch=rng.randint(1, 4),
                    tokens=_log_int(rng, 24, 2048), kv=rng.choice(("e5m2", "half")))
    if kind == "experts":
        return dict(kind=kind, experts=8, top_k=2, hidden=128 * rng.randint(16, 32), inter=128 * rng.randint(56, 112),
                    tokens=_log_int(rng, 1, 512), low_bit=rng.choice(("sym_int4", "fp8_e4m3")), dtype=dtype)
    if kind == "train":
        return dict(kind=kind, arch=rng.choice(("llama2-7b", "llama2-13b")), layers=rng.randint(1, 3), low_bit="nf4",
                    dtype="bfloat16", batch=rng.randint(1, 4), tokens=rng.randint(65, 512))
    return dict(kind=kind, n=16 * rng.randint(64, 1800), k=128 * rng.randint(8, 112),
                low_bit=rng.choice(("sym_int4", "asym_int4", "nf4", "fp8_e4m3", "sym_int8")), dtype=dtype)


# ---- seeded data ------------------------------------------------------------------------------------------------------
def _gen(seed, name):
    return torch.Generator(device="cuda").manual_seed(zlib.crc32(("%d/%s" % (seed, name)).encode()))


def _normal(seed, name, shape, dtype, std=STD, mean=0.0):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(mean, std, generator=_gen(seed, name))


def _dtype(case):
    return getattr(torch, case["dtype"])


def _tokens(seed, name, shape, vocab):
    return torch.randint(0, vocab, shape, device="cuda", generator=_gen(seed, name))


def _weight(case, seed, name, shape):
    """A parameter of a model, by its name: norm scales near one; queries and keys N(0, 0.01) (scores whose soft-max is
    neither flat nor one-hot); projections that add to the residual stream N(0, 0.02 / sqrt(2 * 32)), beside embeddings
    of some size, as deep models are initialised; everything else N(0, 0.02)."""
    if len(shape) == 1:
        return _normal(seed, name, shape, _dtype(case), 0.1, 1.0)
    std = STD
    if ".q_proj." in name or ".k_proj." in name:
        std = STD / 2
    elif ".o_proj." in name or ".down_proj." in name:
        std = STD / 8
    elif ".embed_tokens." in name:
        std = 0.5
    return _normal(seed, name, shape, _dtype(case), std)


def _dense_model(case, seed):
    from ipex_llm_b200.transformers import model as hub
    arch = ARCHS[case["arch"]]
    cfg = hub.transformers.LlamaConfig(num_hidden_layers=case["layers"], rms_norm_eps=EPS, tie_word_embeddings=False,
                                       max_position_embeddings=8192, **arch)
    with torch.device("cuda"):
        model = hub.transformers.AutoModelForCausalLM.from_config(cfg, dtype=_dtype(case))
    for name, p in model.named_parameters():
        p.data.copy_(_weight(case, seed, name, tuple(p.shape)))
    return model.eval()


class _Bank(torch.nn.Module):
    """Fused expert weights in the layout that transformers gives them."""

    def __init__(self, gate_up, down):
        super().__init__()
        self.gate_up_proj = torch.nn.Parameter(gate_up, requires_grad=False)
        self.down_proj = torch.nn.Parameter(down, requires_grad=False)


def _routes(case, seed):
    """Experts and weights of every token, as a router hands them over."""
    score = torch.rand((case["tokens"], case["experts"]), device="cuda", generator=_gen(seed, "router"))
    top = torch.topk(score, case["top_k"], dim=-1)
    return top.indices, torch.softmax(top.values * 4.0, dim=-1)


# ---- what the program has in hand, and one pass -----------------------------------------------------------------------
def prepare(case, seed):
    with torch.set_grad_enabled(case["kind"] == "train"):
        return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def _prepare_linear(case, seed):
    from ipex_llm_b200 import optimize_model
    box = torch.nn.Sequential(torch.nn.Linear(case["k"], case["n"], bias=False, device="cuda", dtype=_dtype(case)))
    box[0].weight.data.copy_(_weight(case, seed, "weight", (case["n"], case["k"])))
    box = optimize_model(box, low_bit=case["low_bit"], optimize_llm=False)
    return dict(kind="linear", layer=box[0], x=_normal(seed, "x", (case["rows"], case["k"]), _dtype(case), 1.0))


def _run_linear(state):
    with torch.no_grad():
        return state["layer"](state["x"])


def _engine(case, seed, rows, length):
    from ipex_llm_b200 import optimize_model
    from ipex_llm_b200.engine import get_engine
    model = optimize_model(_dense_model(case, seed), low_bit=case["low_bit"], torch_dtype=_dtype(case))
    had = os.environ.get("IPEX_LLM_QUANTIZE_KV_CACHE")
    os.environ["IPEX_LLM_QUANTIZE_KV_CACHE"] = "1" if case["kv"] == "e5m2" else "0"
    try:
        return model, get_engine(model, rows, length)
    finally:
        del os.environ["IPEX_LLM_QUANTIZE_KV_CACHE"]
        if had is not None:
            os.environ["IPEX_LLM_QUANTIZE_KV_CACHE"] = had


def _prepare_decode(case, seed):
    vocab = ARCHS[case["arch"]]["vocab_size"]
    B, S, n = case["batch"], case["ctx"], case["steps"]
    model, engine = _engine(case, seed, B, S + n + 1)
    engine.prefill(_tokens(seed, "prompt", (B, S), vocab))
    chosen = [t.contiguous().cpu().pin_memory() for t in _tokens(seed, "chosen", (B, n), vocab).t()]
    return dict(kind="decode", model=model, engine=engine, chosen=chosen, batch=B, ctx=S)


def _run_decode(state):
    # the same continuation again: back to the end of the prompt, then one step per token that the host picked
    engine, B = state["engine"], state["batch"]
    engine.past_len[:B].fill_(state["ctx"])
    logits = []
    for tokens in state["chosen"]:
        state["model"].decode_step(tokens)
        logits.append(engine.logits[:B].clone())
    return logits


def _prepare_prompt(case, seed):
    B, S = case["batch"], case["tokens"]
    model, engine = _engine(case, seed, B, S + 1)
    return dict(kind="prompt", model=model, engine=engine, tokens=S,
                ids=_tokens(seed, "prompt", (B, S), ARCHS[case["arch"]]["vocab_size"]))


def _run_prompt(state):
    # the cache in the model's type is compared too; a byte cache is not (a key that moves by fp16's last place may round
    # to the neighbouring byte): the decode cases read it
    engine, S = state["engine"], state["tokens"]
    out = {"logits": engine.prefill(state["ids"])}
    if not engine.kv_fp8:
        for i, layer in enumerate(engine.cache.layers):
            out["k%d" % i], out["v%d" % i] = layer._k[:, :, :S], layer._v[:, :, :S]
    return out


def _bank(case, seed):
    E, H, I = case["experts"], case["hidden"], case["inter"]
    return _weight(case, seed, "gate_up", (E, 2 * I, H)), _weight(case, seed, "down", (E, H, I))


def _prepare_experts(case, seed):
    from ipex_llm_b200 import optimize_model
    box = torch.nn.Sequential(_Bank(*_bank(case, seed)))
    box = optimize_model(box, low_bit=case["low_bit"], optimize_llm=False)
    index, weight = _routes(case, seed)
    return dict(kind="experts", bank=box[0], index=index, weight=weight,
                x=_normal(seed, "x", (case["tokens"], case["hidden"]), _dtype(case), 1.0))


def _run_experts(state):
    with torch.no_grad():
        return state["bank"](state["x"], state["index"], state["weight"])


def _lora(seed, layer, proj, which, shape):
    """Adapter weights in the middle of a run: neither side is zero."""
    std = 1.0 / math.sqrt(shape[1]) if which == "A" else 0.02
    return _normal(seed, "%d.%s.%s" % (layer, proj, which), shape, torch.bfloat16, std)


def _prepare_train(case, seed):
    from ipex_llm_b200 import optimize_model
    from ipex_llm_b200.transformers.qlora import (LoraConfig, cast_lora_weight, get_peft_model,
                                                  prepare_model_for_kbit_training)
    model = optimize_model(_dense_model(case, seed), low_bit=case["low_bit"], optimize_llm=False,
                           modules_to_not_convert=["lm_head"], torch_dtype=_dtype(case))
    model = prepare_model_for_kbit_training(model)
    model = get_peft_model(model, LoraConfig(r=LORA_R, lora_alpha=LORA_ALPHA, lora_dropout=0.0, training_mode="qlora",
                                             target_modules=list(PROJECTIONS)))
    cast_lora_weight(model, torch.bfloat16)
    model.train()
    trained = {}
    for i, block in enumerate(model.model.model.layers):
        for proj in PROJECTIONS:
            layer = getattr(block.self_attn if proj[0] in "qkvo" else block.mlp, proj)
            for which in "AB":
                p = getattr(layer, "lora_" + which)["default"].weight
                p.data.copy_(_lora(seed, i, proj, which, tuple(p.shape)))
                trained["%d.%s.%s" % (i, proj, which)] = p
    ids = _tokens(seed, "ids", (case["batch"], case["tokens"]), ARCHS[case["arch"]]["vocab_size"])
    return dict(kind="train", model=model, trained=trained, ids=ids)


def _run_train(state):
    for p in state["trained"].values():
        p.grad = None
    with torch.autocast("cuda", dtype=torch.bfloat16):
        loss = state["model"](input_ids=state["ids"], labels=state["ids"]).loss
    loss.backward()
    return {"loss": loss.detach(), "grad": {name: p.grad for name, p in state["trained"].items()}}


def _prepare_quantize(case, seed):
    from ipex_llm_b200.quant import qtypes
    return dict(kind="quantize", qtype=qtypes.qtype_from_name(case["low_bit"]), dtype=_dtype(case),
                w=_weight(case, seed, "weight", (case["n"], case["k"])))


def _run_quantize(state):
    from ipex_llm_b200.quant.params import FP4Params
    p = FP4Params(state["w"], requires_grad=False, quantized=False, qtype=state["qtype"]).to("cuda")
    return {"packed": p.data, "dense": p.dequantize(state["dtype"])}


_PREPARE = dict(linear=_prepare_linear, decode=_prepare_decode, prompt=_prepare_prompt, experts=_prepare_experts,
                train=_prepare_train, quantize=_prepare_quantize)
_RUN = dict(linear=_run_linear, decode=_run_decode, prompt=_run_prompt, experts=_run_experts, train=_run_train,
            quantize=_run_quantize)


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
_BITS = {"sym_int4": 4 + 16 / 64, "asym_int4": 4 + 32 / 64, "nf4": 4 + 16 / 64, "fp8_e4m3": 8 + 32 / 128,
         "sym_int8": 8 + 16 / 64}


def _layer_weights(arch):
    hd = arch["hidden_size"] // arch["num_attention_heads"]
    H, I, kv = arch["hidden_size"], arch["intermediate_size"], arch["num_key_value_heads"] * hd
    return H * (H + 2 * kv) + H * H + 3 * H * I


def work(case):
    per = _BITS[case["low_bit"]] / 8
    kind = case["kind"]
    if kind == "linear":
        M, N, K = case["rows"], case["n"], case["k"]
        return {"bytes": N * K * per + 2 * M * (N + K), "flops": 2.0 * M * N * K}
    if kind == "quantize":
        N, K = case["n"], case["k"]
        return {"bytes": N * K * (2 + per + per + 2), "flops": 0}
    if kind == "experts":
        T, H, I, E, k = case["tokens"], case["hidden"], case["inter"], case["experts"], case["top_k"]
        hit = E * (1 - (1 - k / E) ** T)
        return {"bytes": hit * 3 * H * I * per + 4 * T * H, "flops": 2.0 * T * k * 3 * H * I}
    arch = ARCHS[case["arch"]]
    H, V, L = arch["hidden_size"], arch["vocab_size"], case["layers"]
    hd = H // arch["num_attention_heads"]
    kv = arch["num_key_value_heads"] * hd
    body = L * _layer_weights(arch)
    B = case["batch"]
    if kind == "decode":
        kv_bytes = 1 if case["kv"] == "e5m2" else 2
        ctx = case["ctx"] + case["steps"] / 2
        step = (body + V * H) * per + 2 * B * ctx * kv * L * kv_bytes + 2 * B * V
        flops = 2.0 * B * (body + V * H) + 4.0 * B * ctx * H * L
        return {"bytes": case["steps"] * step, "flops": case["steps"] * flops}
    T = B * case["tokens"]
    attention = 4.0 * B * case["tokens"] ** 2 / 2 * H * L
    if kind == "prompt":
        kv_bytes = 1 if case["kv"] == "e5m2" else 2
        return {"bytes": (body + V * H) * per + 2 * T * kv * L * kv_bytes + 2 * T * H + 2 * B * V,
                "flops": 2.0 * T * body + 2.0 * B * V * H + attention}
    # training: forward, once more under checkpointing, gradients of the activations (attention: two and a half times)
    # and of the adapters; the output layer forward and backward
    lora = 0
    for n, k in _proj_shapes(arch).values():
        lora += LORA_R * (n + k)
    lora *= L
    return {"bytes": 2 * body * per + 2 * 2 * V * H + 2 * T * H + 2 * lora,
            "flops": 2.0 * T * (3 * body + 4 * lora + 2 * V * H) + 4.5 * attention}


def tolerance(case):
    if case["kind"] == "quantize":
        return "exact"
    # about four times what each differs by from 64 bits: one product (fp16 2e-4, with a second product behind it 4e-4; bf16
    # 3e-3), a whole model (fp16 3e-3, bf16 up to 1.7e-2)
    if case["kind"] in ("linear", "experts"):
        return {"rel": 2e-3 if case["dtype"] == "float16" else 1.2e-2}
    return {"rel": 1.2e-2 if case["dtype"] == "float16" else 3e-2}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------
_NF4 = (-1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453, -0.28444138169288635, -0.18477343022823334,
        -0.09105003625154495, 0.0, 0.07958029955625534, 0.16093020141124725, 0.24611230194568634, 0.33791524171829224,
        0.44070982933044434, 0.5626170039176941, 0.7229568362236023, 1.0)


def _rounded(w, low_bit):
    """The values that a packed weight stands for (scales are stored in fp16, those of fp8 blocks in fp32)."""
    shape, w = w.shape, w.float()
    if low_bit == "fp8_e4m3":
        b = w.reshape(-1, 128)
        d = b.abs().amax(1, keepdim=True) / 448.0
        q = (b * torch.where(d > 0, 1.0 / d, torch.zeros_like(d))).to(torch.float8_e4m3fn)
        return (q.double() * d.double()).reshape(shape)
    b = w.reshape(-1, 64)
    if low_bit == "sym_int4":
        top = b.gather(1, b.abs().argmax(1, keepdim=True))
        d = top / -8.0
        q = (b * torch.where(d != 0, 1.0 / d, torch.zeros_like(d)) + 8.5).trunc().clamp(0, 15) - 8.0
        return (q.double() * d.half().double()).reshape(shape)
    if low_bit == "asym_int4":
        lo, hi = b.amin(1, keepdim=True), b.amax(1, keepdim=True)
        d = (hi - lo) / 15.0
        q = ((b - lo) * torch.where(d != 0, 1.0 / d, torch.zeros_like(d)) + 0.5).trunc().clamp(0, 15)
        return (q.double() * d.half().double() + lo.half().double()).reshape(shape)
    if low_bit == "sym_int8":
        d = b.abs().amax(1, keepdim=True) / 127.0
        q = (b * torch.where(d != 0, 1.0 / d, torch.zeros_like(d))).round().clamp(-128, 127)
        return (q.double() * d.half().double()).reshape(shape)
    d = b.abs().amax(1, keepdim=True).half().float()
    book = torch.tensor(_NF4, dtype=torch.float32, device=w.device)
    edges = (book[1:] + book[:-1]) / 2
    q = torch.bucketize(b * torch.where(d != 0, 1.0 / d, torch.zeros_like(d)), edges)
    return (book[q].double() * d.double()).reshape(shape)


def _proj_shapes(arch):
    H, I = arch["hidden_size"], arch["intermediate_size"]
    kv = arch["num_key_value_heads"] * (H // arch["num_attention_heads"])
    return dict(q_proj=(H, H), k_proj=(kv, H), v_proj=(kv, H), o_proj=(H, H), gate_proj=(I, H), up_proj=(I, H),
                down_proj=(H, I))


def _norm(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w.double()


def _rotate(x, theta):
    S, D = x.shape[-2], x.shape[-1]
    inv = theta ** (-torch.arange(0, D, 2, device=x.device, dtype=torch.float64) / D)
    a = torch.arange(S, device=x.device, dtype=torch.float64)[:, None] * inv
    c, s = a.cos(), a.sin()
    u, v = x[..., : D // 2], x[..., D // 2:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _attend(q, k, v, first):
    """Causal attention [heads, queries, D] of the queries at positions ``first`` and on, group by group of heads."""
    out = []
    mask = torch.arange(k.shape[1], device=q.device)[None, :] > torch.arange(first, first + q.shape[1],
                                                                            device=q.device)[:, None]
    group = q.shape[0] // k.shape[0]
    for h in range(k.shape[0]):
        s = q[h * group:(h + 1) * group] @ k[h].t() / math.sqrt(q.shape[-1])
        out.append(torch.softmax(s.masked_fill(mask, float("-inf")), -1) @ v[h])
    return torch.cat(out)


def _through_cache(x, case):
    """Keys and values as a decode step finds them."""
    x = x.to(_dtype(case))
    if case["kv"] == "e5m2":
        x = x.half().clamp(-57344.0, 57344.0).to(torch.float8_e5m2)
    return x.double()


def _layer(case, seed, i, x, cached_from=None, lora=None, keep=None):
    """One decoder layer on [B, S, H] in 64 bits.  From position ``cached_from`` on, queries read keys and values through
    the cache; ``lora``: {name: adapter}; ``keep``: called with the layer's keys and values."""
    arch = ARCHS[case["arch"]]
    shapes = _proj_shapes(arch)
    B, S, H = x.shape
    nq, nk = arch["num_attention_heads"], arch["num_key_value_heads"]
    D = H // nq
    at = "model.layers.%d." % i

    def project(y, proj):
        where = "self_attn." if proj[0] in "qkvo" else "mlp."
        with torch.no_grad():
            w = _rounded(_weight(case, seed, at + where + proj + ".weight", shapes[proj]), case["low_bit"])
        z = y @ w.t()
        if lora is not None:
            a, b = lora["%d.%s.A" % (i, proj)], lora["%d.%s.B" % (i, proj)]
            z = z + (y @ a.t()) @ b.t() * (LORA_ALPHA / LORA_R)
        return z

    def heads(y, n):
        return y.view(B, S, n, D).transpose(1, 2)

    y = _norm(x, _weight(case, seed, at + "input_layernorm.weight", (H,)))
    q = _rotate(heads(project(y, "q_proj"), nq), arch["rope_theta"])
    k = _rotate(heads(project(y, "k_proj"), nk), arch["rope_theta"])
    v = heads(project(y, "v_proj"), nk)
    if keep is not None:
        keep(k, v)
    split = S if cached_from is None else cached_from
    rows = []
    for b in range(B):
        o = [_attend(q[b, :, :split], k[b, :, :split], v[b, :, :split], 0)] if split else []
        if split < S:
            o.append(_attend(q[b, :, split:], _through_cache(k[b], case), _through_cache(v[b], case), split))
        rows.append(torch.cat(o, 1))
    o = torch.stack(rows).transpose(1, 2).reshape(B, S, H)
    x = x + project(o, "o_proj")
    y = _norm(x, _weight(case, seed, at + "post_attention_layernorm.weight", (H,)))
    return x + project(F.silu(project(y, "gate_proj")) * project(y, "up_proj"), "down_proj")


def _embedded(case, seed, ids):
    arch = ARCHS[case["arch"]]
    table = _weight(case, seed, "model.embed_tokens.weight", (arch["vocab_size"], arch["hidden_size"]))
    return table[ids].double()


def _scores(case, seed, x, packed=True):
    arch = ARCHS[case["arch"]]
    w = _weight(case, seed, "lm_head.weight", (arch["vocab_size"], arch["hidden_size"]))
    w = _rounded(w, case["low_bit"]) if packed else w.double()
    return _norm(x, _weight(case, seed, "model.norm.weight", (arch["hidden_size"],))) @ w.t()


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    with torch.no_grad():
        if kind == "linear":
            w = _rounded(_weight(case, seed, "weight", (case["n"], case["k"])), case["low_bit"])
            return _normal(seed, "x", (case["rows"], case["k"]), _dtype(case), 1.0).double() @ w.t()
        if kind == "quantize":
            w = _rounded(_weight(case, seed, "weight", (case["n"], case["k"])), case["low_bit"])
            return {"packed": None, "dense": w}
        if kind == "experts":
            return _exact_experts(case, seed)
        arch = ARCHS[case["arch"]]
        B = case["batch"]
        if kind == "prompt":
            x = _embedded(case, seed, _tokens(seed, "prompt", (B, case["tokens"]), arch["vocab_size"]))
            out = {}
            for i in range(case["layers"]):
                def keep(k, v, i=i):
                    if case["kv"] == "half":
                        out["k%d" % i], out["v%d" % i] = k, v
                x = _layer(case, seed, i, x, keep=keep)
            return {"logits": _scores(case, seed, x[:, -1]), **out}
        S, n = case["ctx"], case["steps"]
        ids = torch.cat([_tokens(seed, "prompt", (B, S), arch["vocab_size"]),
                         _tokens(seed, "chosen", (B, n), arch["vocab_size"])], 1)
        x = _embedded(case, seed, ids)
        for i in range(case["layers"]):
            x = _layer(case, seed, i, x, cached_from=S)
        return list(_scores(case, seed, x[:, S:]).unbind(1))


def _exact_experts(case, seed):
    gate_up, down = _bank(case, seed)
    index, weight = _routes(case, seed)
    x = _normal(seed, "x", (case["tokens"], case["hidden"]), _dtype(case), 1.0).double()
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        tok, pos = torch.where(index == e)
        if tok.numel():
            g, u = (x[tok] @ _rounded(gate_up[e], case["low_bit"]).t()).chunk(2, -1)
            y = (F.silu(g) * u) @ _rounded(down[e], case["low_bit"]).t()
            out.index_add_(0, tok, y * weight[tok, pos, None].double())
    return out


def _exact_train(case, seed):
    arch = ARCHS[case["arch"]]
    lora = {}
    for i in range(case["layers"]):
        for proj, (n, k) in _proj_shapes(arch).items():
            for which, shape in (("A", (LORA_R, k)), ("B", (n, LORA_R))):
                lora["%d.%s.%s" % (i, proj, which)] = _lora(seed, i, proj, which, shape).double().requires_grad_()
    ids = _tokens(seed, "ids", (case["batch"], case["tokens"]), arch["vocab_size"])
    x = _embedded(case, seed, ids)
    for i in range(case["layers"]):
        x = torch.utils.checkpoint.checkpoint(_layer, case, seed, i, x, None, lora, use_reentrant=False)
    z = _scores(case, seed, x, packed=False)[:, :-1]
    loss = F.cross_entropy(z.reshape(-1, z.shape[-1]), ids[:, 1:].reshape(-1))
    grads = torch.autograd.grad(loss, list(lora.values()))
    return {"loss": loss.detach(), "grad": dict(zip(lora, grads))}
