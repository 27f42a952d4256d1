"""The work that this framework is timed on: decode steps and prompts of Hunyuan dense layers in both precisions, mixtures of
experts, the gated delta rule, sampling, and a whole model's prompts through the engine.

`listed()` names the cases, `draw(rng)` gives more of the same ranges, `prepare` makes what a program holds before the call,
`run` makes one pass, `exact` says in plain 64-bit torch what that pass computes.

Layers are driven as the model drives them (`parts`, `cache`, `engine.make_context`): a step's context, the blocks one after
another, the prefetch stream joined behind them.  Steps of one token a sequence run as a captured CUDA graph, which is how the
framework decodes; prompts are launched from Python, which is how `Engine.step` runs them.  The rotation tables and everything
else that belongs to a step are made anew in every pass.
"""
from __future__ import annotations

import dataclasses
import math
import os
import random
import shutil
import tempfile

import numpy as np
import torch

DEV = "cuda:0"
BF = torch.bfloat16
F64 = torch.float64
EPS = 1e-5                     # of the norms
HEAD = 128                     # entries of an attention head
LAYERS = 2                     # layers that follow one another in a case of layers (a product prepares the next layer's norm)
TABLE_ROWS = 4096              # rows of the token table of a case of layers
ROPE_BASE = 10000.0 * 1000.0 ** (HEAD / (HEAD - 2))       # theta 10,000 with the dynamic-NTK factor 1,000
DELTA = dict(taps=4, rank=64)                             # the gated delta rule's short convolutions and inner vectors

# widths of the dense family: (hidden, heads, kv heads, intermediate)
WIDTHS = {"1.8b": (2048, 16, 4, 6144), "4b": (3072, 32, 8, 8192), "7b": (4096, 32, 8, 14336), "small": (1024, 8, 2, 2816)}


def _layers(name, width, dtype, batch, new, past, ragged):
    return dict(name=name, kind="layers", width=width, dtype=dtype, batch=batch, new=new, past=past, ragged=ragged)


def listed() -> list:
    return [
        # one user at a terminal: a token at a time, where launches and dependent latency are everything
        _layers("decode_b1", "1.8b", "bf16", 1, 1, 700, 0),
        # the headline: eight conversations behind prompts of about 2,048 tokens
        _layers("decode_b8", "1.8b", "bf16", 8, 1, 2100, 1),
        # a server's batch of the larger model, lengths as they come
        _layers("decode_b64", "4b", "bf16", 64, 1, 2048, 2),
        # one prompt of a document's page
        _layers("prompt_2048", "1.8b", "bf16", 1, 2048, 0, 0),
        # a batch of unequal prompts, odd lengths, the larger model
        _layers("prompts_ragged", "4b", "bf16", 5, 3001, 0, 3),
        # the 32-bit engine decoding a batch
        _layers("f32_decode_b8", "1.8b", "f32", 8, 1, 1000, 4),
        # and its prompt
        _layers("f32_prompt_531", "1.8b", "f32", 1, 531, 0, 0),
        # a mixture of gated experts, routed in groups, beside a gated shared expert: a prompt, and a step of a small batch
        dict(name="experts_prompt", kind="experts", hidden=2048, experts=32, top=4, groups=8, keep=4, ff=1024, shared=2048, tokens=2048),
        dict(name="experts_decode_b8", kind="experts", hidden=2048, experts=32, top=4, groups=8, keep=4, ff=1024, shared=2048, tokens=8),
        # prompts of two sequences through the gated delta rule
        dict(name="delta_prompts", kind="delta", hidden=2048, heads=16, kv_heads=8, batch=2, new=1777, ragged=5),
        # the usual options of a chat (temperature, top-k, top-p, repetition penalty) on a wide vocabulary
        dict(name="sample_b8", kind="sample", rows=8, vocab=120818, top_k=20, top_p=0.6, temperature=0.7, penalty=1.05, window=64),
        # a short prompt through the whole model and engine, tokens to logits
        dict(name="engine_prompt_61", kind="engine", width="small", layers=8, vocab=32768, batch=1, new=61, ragged=0),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "f32", "experts", "delta", "sample", "engine"])
    ragged = rng.randint(1, 1 << 20)
    if kind == "decode":
        width = rng.choice(["1.8b", "4b", "small"])
        c = _layers("", width, "bf16", _log_int(rng, 1, 64), 1, _log_int(rng, 64, 4000), ragged)
    elif kind == "prompt":
        width = rng.choice(["1.8b", "4b", "small"])
        batch = rng.randint(1, 4)
        past = rng.choice([0, 0, rng.randint(1, 1000)])            # a whole prompt, or a further part of one
        c = _layers("", width, "bf16", batch, _log_int(rng, 130, 3500 if batch < 3 else 2000), past, ragged)
    elif kind == "f32":
        width = rng.choice(["1.8b", "small"])
        if rng.random() < 0.5:
            c = _layers("", width, "f32", _log_int(rng, 1, 32), 1, _log_int(rng, 64, 2000), ragged)
        else:
            c = _layers("", width, "f32", rng.randint(1, 2), _log_int(rng, 20, 600), 0, ragged)
    elif kind == "experts":
        c = dict(kind="experts", hidden=rng.choice([1024, 2048]), experts=rng.choice([16, 32]), top=rng.choice([2, 4]), groups=4, keep=2,
                 ff=rng.choice([512, 1024]), shared=rng.choice([1024, 2048]), tokens=_log_int(rng, 1, 4000))
    elif kind == "delta":
        c = dict(kind="delta", hidden=rng.choice([1024, 2048]), heads=rng.choice([8, 16]), kv_heads=rng.choice([4, 8]), batch=rng.randint(1, 4),
                 new=_log_int(rng, 20, 2000), ragged=ragged)
    elif kind == "sample":
        c = dict(kind="sample", rows=_log_int(rng, 1, 64), vocab=rng.choice([32768, 65536, 120818, 128167]), top_k=rng.randint(10, 100),
                 top_p=rng.choice([0.6, 0.8, 0.95]), temperature=rng.choice([0.6, 0.7, 1.0]), penalty=rng.choice([1.0, 1.05]), window=64)
    else:
        c = dict(kind="engine", width="small", layers=4, vocab=32768, batch=rng.randint(1, 4), new=_log_int(rng, 1, 500), ragged=ragged)
    c.pop("name", None)
    return c


# -- sizes that follow from a case -------------------------------------------------------------------------------------------
def _lengths(case) -> list:
    """(tokens that are there, new tokens) of every sequence: the first has the most, the others what `ragged` draws."""
    new, past, batch, ragged = case["new"], case.get("past", 0), case["batch"], case["ragged"]
    rng = random.Random(ragged)
    out = [(past, new)]
    for _ in range(batch - 1):
        n = new if new == 1 or not ragged else rng.randint(max(1, new // 8), new)
        p = past if past == 0 or not ragged else rng.randint(max(1, past // 8), past)
        out.append((p, n))
    return out


def _widths(case):
    return WIDTHS[case["width"]]


def _dtype(case):
    return torch.float32 if case.get("dtype") == "f32" else BF


# -- weights and inputs ------------------------------------------------------------------------------------------------------
class _Maker:
    """Tensors from one seed, in the order they are asked for."""

    def __init__(self, seed, device=DEV):
        self.device = device
        self.gen = torch.Generator(device=device)
        self.gen.manual_seed(int(seed) * 7919 + 13)

    def normal(self, *shape, scale=1.0, mean=0.0, dtype=BF):
        return (torch.randn(shape, generator=self.gen, dtype=torch.float32, device=self.device) * scale + mean).to(dtype)

    def matrix(self, rows, cols, scale=1.0):
        return self.normal(rows, cols, scale=scale / math.sqrt(cols))

    def gain(self, n):
        return self.normal(n, scale=0.1, mean=1.0)

    def uniform(self, *shape):
        return torch.rand(shape, generator=self.gen, dtype=torch.float32, device=self.device)

    def ids(self, n, below):
        return torch.randint(0, below, (n,), generator=self.gen, device=self.device)


def _dense_weights(make, prefix, widths):
    h, nh, nkv, f = widths
    p = prefix
    return {p + "self_attn.q_proj.weight": make.matrix(nh * HEAD, h), p + "self_attn.k_proj.weight": make.matrix(nkv * HEAD, h),
            p + "self_attn.v_proj.weight": make.matrix(nkv * HEAD, h), p + "self_attn.o_proj.weight": make.matrix(h, nh * HEAD),
            p + "self_attn.query_layernorm.weight": make.gain(HEAD), p + "self_attn.key_layernorm.weight": make.gain(HEAD),
            p + "mlp.gate_proj.weight": make.matrix(f, h), p + "mlp.up_proj.weight": make.matrix(f, h),
            p + "mlp.down_proj.weight": make.matrix(h, f), p + "input_layernorm.weight": make.gain(h),
            p + "post_attention_layernorm.weight": make.gain(h)}


def _layers_inputs(case, seed):
    """(weights by name, token table, token ids, per layer and sequence the keys and values that are there)."""
    h, nh, nkv, f = _widths(case)
    make = _Maker(seed)
    weights = {}
    for l in range(LAYERS):
        weights.update(_dense_weights(make, f"model.layers.{l}.", (h, nh, nkv, f)))
    table = make.normal(TABLE_ROWS, h)
    lens = _lengths(case)
    ids = make.ids(sum(n for _, n in lens), TABLE_ROWS)
    dtype = _dtype(case)
    past = [[(make.normal(p, nkv, HEAD, dtype=dtype), make.normal(p, nkv, HEAD, dtype=dtype)) for p, _ in lens] for _ in range(LAYERS)]
    return weights, table, ids, past


def _dense_config(case, layers, vocab):
    from hymt2sharp_b200.config import HunyuanDenseConfig
    h, nh, nkv, f = _widths(case)
    return HunyuanDenseConfig.from_dict(dict(
        architectures=["HunYuanDenseV1ForCausalLM"], num_hidden_layers=layers, hidden_size=h, num_attention_heads=nh, num_key_value_heads=nkv,
        head_dim=HEAD, intermediate_size=f, vocab_size=vocab, rope_theta=10000.0, rope_scaling={"type": "dynamic", "alpha": 1000.0},
        rms_norm_eps=EPS, use_qk_norm=True, tie_word_embeddings=True, max_position_embeddings=32768))


# -- prepare -----------------------------------------------------------------------------------------------------------------
def prepare(case: dict, seed: int) -> dict:
    return {"layers": _prepare_layers, "experts": _prepare_experts, "delta": _prepare_delta, "sample": _prepare_sample,
            "engine": _prepare_engine}[case["kind"]](case, seed)


def _context(cache, lens, ids, dtype, vocab):
    """A step of len(lens) sequences whose earlier tokens are in the cache already; the cache keeps its length, so that the same
    step can run again."""
    from hymt2sharp_b200.engine.engine import StepEntry, make_context
    from hymt2sharp_b200.kernels import ops
    slots = cache.alloc_slots(len(lens))
    earlier = [(s, p) for s, (p, _) in zip(slots, lens) if p]
    if earlier:
        cache.begin_step(earlier)
        cache.end_step(earlier)
    flat, entries, o = ids.tolist(), [], 0
    for s, (_, n) in zip(slots, lens):
        entries.append(StepEntry(s, flat[o:o + n], []))
        o += n
    ctx, _, _, _ = make_context(cache, entries, vocab, dtype, torch.device(DEV), ops.device_status(torch.device(DEV)))
    return ctx, slots


def _cache_tokens(lens):
    return sum(-(-(p + n) // 64) * 64 for p, n in lens)


def _captured(fn):
    """The pass as a CUDA graph: one run first (kernels set themselves up), then the capture."""
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        fn()
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = fn()
    return graph, out


def _prepare_layers(case, seed):
    from hymt2sharp_b200.cache import PagedCache
    from hymt2sharp_b200.engine.hunyuan_dense import build_spec
    from hymt2sharp_b200.engine.model import DecoderModel
    weights, table, ids, past = _layers_inputs(case, seed)
    dtype, lens = _dtype(case), _lengths(case)
    model = DecoderModel(build_spec(_dense_config(case, LAYERS, TABLE_ROWS)))
    for block in model.blocks:
        block.load(weights, DEV, dtype)
    cache = PagedCache(model.groups, dtype, DEV, _cache_tokens(lens), max_slots=case["batch"],
                       max_sequence_tokens=-(-max(p + n for p, n in lens) // 64) * 64)
    ctx, slots = _context(cache, lens, ids, dtype, TABLE_ROWS)
    table = table.to(dtype)
    for l in range(LAYERS):
        slot = model.slots[l][0]
        planes = cache.plane(slot.group, slot.plane)
        for s, (p, _), kv in zip(slots, lens, past[l]):
            blocks = -(-p // 64)
            rows = torch.as_tensor(cache.host_tables[slot.group][s, :blocks].astype(np.int64), device=DEV)
            for plane, x in zip(planes, kv):
                if p:
                    padded = torch.zeros((blocks * 64, *x.shape[1:]), dtype=dtype, device=DEV)
                    padded[:p] = x
                    plane[rows] = padded.view(blocks, 64, *x.shape[1:]).transpose(1, 2)
    state = dict(kind="layers", model=model, cache=cache, ctx=ctx, table=table)
    if ctx.decode:
        state["graph"], state["out"] = _captured(lambda: _run_blocks(state))
    return state


def _run_blocks(state):
    from hymt2sharp_b200.kernels import ops
    model = state["model"]
    ctx = dataclasses.replace(state["ctx"], shared={})
    residual = torch.empty((ctx.num_tokens, model.spec.hidden), dtype=torch.float32, device=ctx.device)
    ops.embed(residual, state["table"], ctx.tokens, ctx.status, 1.0)
    for i, block in enumerate(model.blocks):
        ahead = model.blocks[i + 1] if i + 1 < len(model.blocks) else None
        ctx.next_first_norm = ahead.first_norm() if ahead is not None else None
        ctx.block_ahead = ahead
        block.forward(residual, ctx, model.slots[i])
    ops.join_beside(ctx.device)
    return residual, state["cache"].storage[0]


def _experts_weights(case, seed):
    h, e, f, s = case["hidden"], case["experts"], case["ff"], case["shared"]
    make = _Maker(seed)
    w = {"router": make.matrix(e, h, 1.5), "shared.sg": make.matrix(1, h), "shared.gate": make.matrix(s, h), "shared.up": make.matrix(s, h),
         "shared.down": make.matrix(h, s)}
    for i in range(e):
        w[f"e{i}.gate"], w[f"e{i}.up"], w[f"e{i}.down"] = make.matrix(f, h), make.matrix(f, h), make.matrix(h, f)
    return w, make.normal(case["tokens"], h), make.normal(case["tokens"], h, dtype=torch.float32)


def _prepare_experts(case, seed):
    from hymt2sharp_b200.cache import PagedCache
    from hymt2sharp_b200.parts import PartSpec, build_part
    w, x, residual = _experts_weights(case, seed)
    shared = PartSpec("swiglu", dict(hidden=case["hidden"], intermediate=case["shared"], gate_proj="shared.gate", up_proj="shared.up",
                                     down_proj="shared.down"))
    part = build_part("feed_forward", PartSpec("routed_experts", dict(
        hidden=case["hidden"], experts=case["experts"], identity=0, top=case["top"], intermediate=case["ff"], activation="silu", router="router",
        scores="sigmoid", weights="chosen_share", share_eps=1e-20, groups=case["groups"], keep=case["keep"], gate_proj="e{}.gate",
        up_proj="e{}.up", down_proj="e{}.down", shared=shared, shared_gate="shared.sg")))
    part.load(w, DEV, BF)
    decode = case["tokens"] <= 64
    lens = [(0, 1)] * case["tokens"] if decode else [(0, case["tokens"])]
    cache = PagedCache([], BF, DEV, _cache_tokens(lens), max_slots=len(lens))
    ctx, _ = _context(cache, lens, torch.zeros(case["tokens"], dtype=torch.int64), BF, 8)
    state = dict(kind="experts", part=part, ctx=ctx, cache=cache, x=x, residual=residual)
    if decode:
        state["graph"], state["out"] = _captured(lambda: _run_experts(state))
    return state


def _run_experts(state):
    out = state["residual"].clone()
    state["part"].forward(state["x"], out, dataclasses.replace(state["ctx"], shared={}))
    return out


def _delta_weights(case, seed):
    W, H, G, d, r = case["hidden"], case["heads"], case["kv_heads"], HEAD, DELTA["rank"]
    make = _Maker(seed)
    w = {"q": make.matrix(G * d, W), "k": make.matrix(G * d, W), "v": make.matrix(H * d, W), "b": make.matrix(H, W), "a1": make.matrix(r, W),
         "a2": make.matrix(H * d, r, 0.5), "g1": make.matrix(r, W), "g2": make.matrix(H * d, r), "norm": make.gain(d), "o": make.matrix(W, H * d)}
    for name, c in (("q.conv", G * d), ("k.conv", G * d), ("v.conv", H * d)):
        w[name] = make.normal(c, DELTA["taps"], scale=0.4)
    w["A_log"] = (make.uniform(H) * 15.0 + 1.0).log()
    step = torch.exp(make.uniform(H * d) * math.log(100.0) + math.log(0.001))      # step sizes between 0.001 and 0.1
    w["dt"] = torch.log(torch.expm1(step))
    return w, make.normal(sum(n for _, n in _lengths(case)), W)


def _prepare_delta(case, seed):
    from hymt2sharp_b200.cache import PagedCache
    from hymt2sharp_b200.parts import MixerSlot, PartSpec, build_part
    w, x = _delta_weights(case, seed)
    part = build_part("mixer", PartSpec("gated_delta", dict(
        hidden=case["hidden"], heads=case["heads"], kv_heads=case["kv_heads"], dim=HEAD, vdim=HEAD, taps=DELTA["taps"], eps=EPS, q_proj="q",
        k_proj="k", v_proj="v", q_conv="q.conv", k_conv="k.conv", v_conv="v.conv", b_proj="b", a_log="A_log", a1_proj="a1", a2_proj="a2",
        dt_bias="dt", g1_proj="g1", g2_proj="g2", norm="norm", o_proj="o", decay_rank=DELTA["rank"], gate_rank=DELTA["rank"])))
    # (the part pads its stacked projections on the host)
    part.load({k: v.cpu() for k, v in w.items()}, DEV, BF)
    lens = _lengths(case)
    cache = PagedCache([], BF, DEV, _cache_tokens(lens), max_slots=len(lens), state_bytes=part.state_bytes())
    ctx, slots = _context(cache, lens, torch.zeros(len(x), dtype=torch.int64), BF, 8)
    state = dict(kind="delta", part=part, ctx=ctx, cache=cache, x=x, slot=MixerSlot(state_offset=0, state_bytes=part.state_bytes()),
                 rows=cache.state.view(torch.float32))
    return state


def _run_delta(state):
    ctx = dataclasses.replace(state["ctx"], shared={})
    out = torch.empty((ctx.num_tokens, state["part"].hidden), dtype=torch.float32, device=ctx.device)
    state["part"].forward(state["x"], out, ctx, state["slot"], store=True)
    return out, state["rows"]


def _sample_inputs(case, seed):
    make = _Maker(seed)
    # a model's logits: a wide bulk, and some tens of tokens far above it
    logits = make.normal(case["rows"], case["vocab"], scale=2.0, dtype=torch.float32)
    at = make.ids(case["rows"] * 40, case["vocab"]).view(case["rows"], 40)
    logits.scatter_add_(1, at, make.uniform(case["rows"], 40) * 14.0)
    history = make.ids(case["rows"] * case["window"], case["vocab"]).view(case["rows"], case["window"])
    history[:, :8] = at[:, :8]                                       # some of the likely ones were said before
    return logits, history


def _prepare_sample(case, seed):
    from hymt2sharp_b200.sampling import BatchSampler, SamplingParams
    logits, history = _sample_inputs(case, seed)
    params = [SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], repeat_penalty=case["penalty"],
                             penalty_window=case["window"], seed=seed * 1000 + i) for i in range(case["rows"])]
    sampler = BatchSampler(params, DEV, history.tolist())
    state = dict(kind="sample", sampler=sampler, logits=logits, work=torch.empty_like(logits),
                 tokens=torch.empty(case["rows"], dtype=torch.int32, device=DEV), snapshot=sampler.snapshot())
    state["graph"], state["out"] = _captured(lambda: _run_sample(state))
    return state


def _run_sample(state):
    """The step's logits as the head leaves them, the options that the batch came with, one token a row."""
    state["work"].copy_(state["logits"])
    state["sampler"].restore(state["snapshot"])
    state["sampler"].sample(state["work"], None, out=state["tokens"])
    return state["work"], state["tokens"]


def _engine_weights(case, seed):
    h = _widths(case)[0]
    make = _Maker(seed)
    weights = {"model.embed_tokens.weight": make.normal(case["vocab"], h, scale=1.0 / math.sqrt(h)), "model.norm.weight": make.gain(h)}
    for l in range(case["layers"]):
        weights.update(_dense_weights(make, f"model.layers.{l}.", _widths(case)))
    lens = _lengths(case)
    return weights, make.ids(sum(n for _, n in lens), case["vocab"])


def _prepare_engine(case, seed):
    import json

    import hymt2sharp_b200
    from hymt2sharp_b200.engine.engine import StepEntry
    from hymt2sharp_b200.weights import write_safetensors
    weights, ids = _engine_weights(case, seed)
    folder = tempfile.mkdtemp(prefix="hymt2_cases_")
    try:
        with open(os.path.join(folder, "config.json"), "w") as f:
            json.dump(_dense_config(case, case["layers"], case["vocab"]).to_dict(), f)
        write_safetensors(os.path.join(folder, "model.safetensors"), {k: v.cpu() for k, v in weights.items()}, metadata={"format": "pt"})
        engine = hymt2sharp_b200.load(folder, dtype="bfloat16", max_tokens=4096, max_batch=case["batch"], device=DEV)
    finally:
        shutil.rmtree(folder, ignore_errors=True)
    slots = engine.alloc_slots(case["batch"])
    flat, entries, o = ids.tolist(), [], 0
    for s, (_, n) in zip(slots, _lengths(case)):
        entries.append(StepEntry(s, flat[o:o + n], [n - 1]))
        o += n
    return dict(kind="engine", engine=engine, slots=slots, entries=entries)


def _run_engine(state):
    for s in state["slots"]:
        state["engine"].reset(s)
    return state["engine"].step(state["entries"])


# -- one pass ----------------------------------------------------------------------------------------------------------------
def run(state: dict):
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    return {"layers": _run_blocks, "experts": _run_experts, "delta": _run_delta, "engine": _run_engine}[state["kind"]](state)


# -- what a pass cannot do without -------------------------------------------------------------------------------------------
def _attention_work(lens, nh, nkv, size):
    pairs = sum(n * p + n * (n + 1) // 2 for p, n in lens)
    return dict(flops=4 * pairs * nh * HEAD, bytes=sum(2 * (p + 2 * n) * nkv * HEAD * size for p, n in lens))


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("layers", "engine"):
        h, nh, nkv, f = _widths(case)
        lens, size = _lengths(case), 4 if case.get("dtype") == "f32" else 2
        T, layers = sum(n for _, n in lens), LAYERS if kind == "layers" else case["layers"]
        entries = h * (nh + 2 * nkv) * HEAD + nh * HEAD * h + 3 * h * f
        a = _attention_work(lens, nh, nkv, size)
        # the residual leaves once as float32; between layers it can stay where it is
        total = dict(flops=layers * (2 * T * entries + a["flops"]), bytes=layers * (entries * size + a["bytes"]) + T * h * (size + 4))
        if kind == "engine":
            head = case["vocab"] * h
            total["flops"] += 2 * len(lens) * head
            total["bytes"] += head * 2 + len(lens) * case["vocab"] * 4 - T * h * 4
        return total
    if kind == "experts":
        h, e, f, s, T, top = case["hidden"], case["experts"], case["ff"], case["shared"], case["tokens"], case["top"]
        met = e * (1.0 - (1.0 - top / e) ** T)                    # experts that some token chooses
        return dict(flops=2 * T * (h * (e + 1) + 3 * h * f * top + 3 * h * s), bytes=2 * (met * 3 * h * f + 3 * h * s + (e + 1) * h) + T * h * (2 + 8))
    if kind == "delta":
        W, H, G, r = case["hidden"], case["heads"], case["kv_heads"], DELTA["rank"]
        lens = _lengths(case)
        T, entries = sum(n for _, n in lens), W * HEAD * (2 * G + 2 * H) + 2 * r * W + 2 * r * H * HEAD + W * H
        return dict(flops=2 * T * entries + 8 * T * H * HEAD * HEAD, bytes=2 * entries + T * W * (2 + 4) + len(lens) * H * HEAD * HEAD * 4)
    return dict(flops=4 * case["rows"] * case["vocab"], bytes=8 * case["rows"] * case["vocab"])


def tolerance(case: dict) -> dict:
    """About four times the distance to the 64-bit values that was measured."""
    kind = case["kind"]
    if kind == "sample":
        return {"rel": 1e-7}                                      # one float32 division; what survives and the tokens are whole
    if case.get("dtype") == "f32":
        return {"rel": 6e-6}
    return {"rel": {"layers": 1e-2, "experts": 3e-3, "delta": 1.5e-2, "engine": 4e-2}[kind]}


# -- the same in 64 bits -----------------------------------------------------------------------------------------------------
def exact(case: dict, seed: int):
    with torch.no_grad():
        return {"layers": _exact_layers, "experts": _exact_experts, "delta": _exact_delta, "sample": _exact_sample,
                "engine": _exact_engine}[case["kind"]](case, seed)


def _norm64(x, gain):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * gain.double()


def _rotate64(x, positions):
    """Pairs (i, i + d/2) by float32(position * frequency): the frequencies and the angle are float32 by definition."""
    half = HEAD // 2
    base = float(np.float32(np.float32(10000.0) * np.float32(math.pow(1000.0, float(np.float32(HEAD) / np.float32(HEAD - 2))))))
    freq = np.array([np.float32(1.0) / np.float32(math.pow(base, float(np.float32(i) / np.float32(half)))) for i in range(half)], dtype=np.float32)
    angle = (positions.float()[:, None] * torch.from_numpy(freq).to(x.device)[None]).double()
    c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, a * s + b * c], dim=-1)


def _dense_layer64(x, w, prefix, widths, lens, past):
    h, nh, nkv, f = widths
    p = prefix
    W = lambda name: w[p + name].double()
    y = _norm64(x, w[p + "input_layernorm.weight"])
    T = x.shape[0]
    positions = torch.cat([torch.arange(a, a + n, device=x.device) for a, n in lens])
    q = _norm64(_rotate64((y @ W("self_attn.q_proj.weight").T).view(T, nh, HEAD), positions), w[p + "self_attn.query_layernorm.weight"])
    k = _norm64(_rotate64((y @ W("self_attn.k_proj.weight").T).view(T, nkv, HEAD), positions), w[p + "self_attn.key_layernorm.weight"])
    v = (y @ W("self_attn.v_proj.weight").T).view(T, nkv, HEAD)
    out, o = torch.empty((T, nh, HEAD), dtype=F64, device=x.device), 0
    for b, (a, n) in enumerate(lens):
        ks, vs = k[o:o + n], v[o:o + n]
        if a:
            ks, vs = torch.cat([past[b][0].double(), ks]), torch.cat([past[b][1].double(), vs])
        hidden = torch.arange(a + n, device=x.device)[None] > torch.arange(a, a + n, device=x.device)[:, None]
        for g in range(nkv):
            group = slice(g * (nh // nkv), (g + 1) * (nh // nkv))
            s = torch.einsum("thd,kd->htk", q[o:o + n, group], ks[:, g]) / math.sqrt(HEAD)
            s.masked_fill_(hidden[None], -math.inf)
            out[o:o + n, group] = torch.einsum("htk,kd->thd", torch.softmax(s, -1), vs[:, g])
        o += n
    x = x + out.view(T, nh * HEAD) @ W("self_attn.o_proj.weight").T
    y = _norm64(x, w[p + "post_attention_layernorm.weight"])
    g = y @ W("mlp.gate_proj.weight").T
    return x + (g * torch.sigmoid(g) * (y @ W("mlp.up_proj.weight").T)) @ W("mlp.down_proj.weight").T


def _exact_layers(case, seed):
    weights, table, ids, past = _layers_inputs(case, seed)
    lens = _lengths(case)
    x = table[ids].double()
    for l in range(LAYERS):
        x = _dense_layer64(x, weights, f"model.layers.{l}.", _widths(case), lens, past[l])
    return x, None                  # the cache's blocks have no layout of their own outside this framework


def _exact_engine(case, seed):
    weights, ids = _engine_weights(case, seed)
    lens = _lengths(case)
    table = weights["model.embed_tokens.weight"]
    x = table[ids].double()
    for l in range(case["layers"]):
        x = _dense_layer64(x, weights, f"model.layers.{l}.", _widths(case), lens, None)
    last = torch.tensor([n for _, n in lens], device=x.device).cumsum(0) - 1
    return _norm64(x[last], weights["model.norm.weight"]) @ table.double().T


def _exact_experts(case, seed):
    w, x, residual = _experts_weights(case, seed)
    x, out = x.double(), residual.double()
    W = lambda name: w[name].double()

    def gated(rows, p):
        g = rows @ W(p + "gate").T
        return (g * torch.sigmoid(g) * (rows @ W(p + "up").T)) @ W(p + "down").T

    scores = torch.sigmoid(x @ W("router").T)
    per = case["experts"] // case["groups"]
    worth = scores.view(len(x), case["groups"], per).topk(min(2, per), dim=-1).values.sum(-1)
    kept = torch.zeros_like(worth, dtype=torch.bool).scatter_(1, worth.topk(case["keep"], dim=-1).indices, True)
    allowed = scores.masked_fill(~kept.repeat_interleave(per, dim=1), -1.0)
    best, chosen = allowed.topk(case["top"], dim=-1)
    share = best / (best.sum(-1, keepdim=True) + 1e-20)
    for e in range(case["experts"]):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if len(rows):
            out.index_add_(0, rows, gated(x[rows], f"e{e}.") * share[rows, place][:, None])
    return out + torch.sigmoid(x @ W("shared.sg").T) * gated(x, "shared.")


def _exact_delta(case, seed):
    w, x = _delta_weights(case, seed)
    H, G, d, taps = case["heads"], case["kv_heads"], HEAD, DELTA["taps"]
    W = {k: v.double() for k, v in w.items()}
    x = x.double()
    outs, states = [], []
    o = 0
    for _, n in _lengths(case):
        h = x[o:o + n]
        o += n
        raw = [h @ W[c].T for c in ("q", "k", "v")]

        def conv(u, f):
            padded = torch.cat([torch.zeros((taps - 1, u.shape[1]), dtype=F64, device=u.device), u])
            y = sum(padded[j:j + n] * f[:, j] for j in range(taps))
            return y * torch.sigmoid(y), padded[n:]

        (q, tq), (k, tk), (v, tv) = (conv(u, W[c + ".conv"]) for u, c in zip(raw, ("q", "k", "v")))
        unit = lambda u: (u := u.view(n, G, d)) / torch.sqrt((u * u).sum(-1, keepdim=True) + 1e-6)
        q, k = unit(q).repeat_interleave(H // G, 1) * d ** -0.5, unit(k).repeat_interleave(H // G, 1)
        v, beta = v.view(n, H, d), torch.sigmoid(h @ W["b"].T)
        step = torch.nn.functional.softplus((h @ W["a1"].T) @ W["a2"].T + W["dt"], threshold=1e9).view(n, H, d)
        decay = torch.exp(-torch.exp(W["A_log"])[None, :, None] * step)
        S = torch.zeros((H, d, d), dtype=F64, device=x.device)
        read = torch.empty((n, H, d), dtype=F64, device=x.device)
        for t in range(n):
            S = S * decay[t][:, :, None]
            u = beta[t][:, None] * (v[t] - torch.matmul(k[t][:, None], S)[:, 0])
            S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
            read[t] = torch.matmul(q[t][:, None], S)[:, 0]
        read = read / torch.sqrt((read * read).mean(-1, keepdim=True) + EPS) * W["norm"]
        gate = torch.sigmoid((h @ W["g1"].T) @ W["g2"].T)
        outs.append((read.reshape(n, H * d) * gate) @ W["o"].T)
        states.append(torch.cat([S.reshape(-1), torch.cat([tq, tk, tv], dim=1).reshape(-1)]))
    return torch.cat(outs), torch.stack(states)


def _exact_sample(case, seed):
    logits, history = _sample_inputs(case, seed)
    x = logits.double()
    if case["penalty"] != 1.0:
        for r in range(case["rows"]):
            for t in history[r].tolist():
                x[r, t] = x[r, t] * case["penalty"] if x[r, t] <= 0 else x[r, t] / case["penalty"]
    inv = float(np.float32(1.0) / np.float32(case["temperature"]))
    best, at = (x * inv).topk(case["top_k"], dim=-1)
    p = torch.exp(best - best[:, :1])
    keep = p.cumsum(-1) - p < case["top_p"] * p.sum(-1, keepdim=True)
    out = torch.full_like(x, -math.inf)
    rows = torch.arange(case["rows"], device=x.device)[:, None].expand_as(at)
    out[rows[keep], at[keep]] = x[rows[keep], at[keep]]
    return out, None
