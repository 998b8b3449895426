"""Performance cases: what users of the framework have it do, through its public entry points.

Six kinds of work, each over the range of sizes it is used at:

* ``decode``    greedy decode steps on prefilled KV slots (``QUICForCausalLM.decode``), from one
                row answered token by token to 64 ragged rows in bursts;
* ``prefill``   prompts into KV slots (``QUICForCausalLM.prefill``), from one short prompt to
                16 prompts of 2048 tokens;
* ``generate``  the token loop of the reference's scripts: ``forward`` on left-padded prompts,
                then ``forward`` once per token with the cache it returned, argmax by the caller;
* ``serve``     a request queue through ``Engine.run``;
* ``linear``    the stand-alone W4A16 linear at the model's four shapes;
* ``attention`` the stand-alone GQA decode attention on left-padded batches.

The model is the 24-layer architecture with seeded random weights.  Its linears have the spread
of the un-quantised initialisation (0.02) and the token's own embedding keeps a share of the
final hidden state, as in a trained model with tied embeddings; the final norm's signs make the
best next token of token t the one paired with it.  The greedy choice is therefore decided by a
wide margin, and two correct implementations generate the same ids.
"""

from __future__ import annotations

import functools
import importlib
from types import SimpleNamespace

import torch

import __graft_entry__ as entry

entry.load_package()
_model = importlib.import_module("quic_cu_b200.model")
_kernels = importlib.import_module("quic_cu_b200.kernels")
_engine = importlib.import_module("quic_cu_b200.engine")
_config = importlib.import_module("quic_cu_b200.config")
_checkpoint = importlib.import_module("quic_cu_b200.checkpoint")

LAYERS, VOCAB, HIDDEN, INTER, GROUP = 24, 151936, 896, 4864, 128
SHAPES = {"qkv": (896, 1152), "o_proj": (896, 896), "gate_up": (896, 9728), "down": (4864, 896)}  # (K, N)
LAYER_PARAMS = sum(k * n for k, n in SHAPES.values())
HEAD_BYTES = VOCAB * HIDDEN * 2
KV_TOKEN_BYTES = LAYERS * 512  # K and V of one token
DEVICE = "cuda"


# ---- the cases ---------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # one chat user: every token id comes from the host and goes back to it
        {"name": "decode-1-fed", "kind": "decode", "weights": "w4", "rows": 1, "shortest": 512, "longest": 512,
         "steps": 16, "fed": True},
        # one user far into a conversation, tokens taken a burst at a time
        {"name": "decode-1-long", "kind": "decode", "weights": "w4", "rows": 1, "shortest": 2100, "longest": 2100,
         "steps": 32, "fed": False},
        # a handful of users with contexts of different lengths
        {"name": "decode-5", "kind": "decode", "weights": "w4", "rows": 5, "shortest": 90, "longest": 701,
         "steps": 16, "fed": False},
        # a full serving batch
        {"name": "decode-64", "kind": "decode", "weights": "w4", "rows": 64, "shortest": 200, "longest": 1500,
         "steps": 16, "fed": False},
        # the un-quantised checkpoint
        {"name": "decode-fp16-1", "kind": "decode", "weights": "fp16", "rows": 1, "shortest": 512, "longest": 512,
         "steps": 16, "fed": False},
        # time to first token: a short question, a few documents, a full admission of long ones
        {"name": "prefill-1x87", "kind": "prefill", "weights": "w4", "seqs": 1, "shortest": 87, "longest": 87},
        {"name": "prefill-8x517", "kind": "prefill", "weights": "w4", "seqs": 8, "shortest": 130, "longest": 517},
        {"name": "prefill-16x2048", "kind": "prefill", "weights": "w4", "seqs": 16, "shortest": 2048,
         "longest": 2048},
        # a script in the reference's style: a fresh cache, then one forward per token
        {"name": "generate-4x128", "kind": "generate", "batch": 4, "shortest": 40, "longest": 128, "tokens": 32},
        # continuous batching with requests of the serving configuration's lengths
        {"name": "serve-96", "kind": "serve", "requests": 96, "slots": 64, "shortest": 64, "longest": 1024,
         "fewest": 128, "most": 512, "burst": 16, "batching": "continuous"},
        # single operators: the largest linear at a decode batch, attention over a long cache
        {"name": "linear-gate_up-16", "kind": "linear", "layer": "gate_up", "rows": 16},
        {"name": "attention-16x8192", "kind": "attention", "batch": 16, "context": 8192},
    ]


def _log(rng, low: int, high: int) -> int:
    """A size between ``low`` and ``high``, spread over the logarithm."""
    return max(low, min(high, round(low * (high / low) ** rng.random())))


def draw(rng) -> dict:
    kind = rng.choice(["decode"] * 4 + ["prefill"] * 3 + ["generate", "serve"] + ["linear"] * 2 + ["attention"] * 2)
    if kind == "decode":
        rows = _log(rng, 1, 64)
        longest = _log(rng, 48, min(8000, 120000 // rows))
        # token by token from the host is what one user or a few do
        fed = rows <= 4 and rng.random() < 0.5
        return {"kind": kind, "weights": "fp16" if rng.random() < 0.25 else "w4", "rows": rows,
                "shortest": max(16, longest // rng.choice((1, 2, 5))), "longest": longest,
                "steps": _log(rng, 4, 48), "fed": fed}
    if kind == "prefill":
        seqs = _log(rng, 1, 16)
        longest = _log(rng, 5, 2000)
        return {"kind": kind, "weights": "fp16" if rng.random() < 0.25 else "w4", "seqs": seqs,
                "shortest": max(1, longest // rng.choice((1, 2, 5))), "longest": longest}
    if kind == "generate":
        longest = _log(rng, 20, 600)
        return {"kind": kind, "batch": _log(rng, 1, 12), "shortest": max(8, longest // 2), "longest": longest,
                "tokens": _log(rng, 8, 64)}
    if kind == "serve":
        requests = _log(rng, 8, 64)
        longest, most = _log(rng, 40, 700), _log(rng, 20, 200)
        return {"kind": kind, "requests": requests, "slots": max(2, min(64, requests // rng.choice((1, 2, 4)))),
                "shortest": max(8, longest // 4), "longest": longest, "fewest": max(4, most // 3), "most": most,
                "burst": rng.choice((8, 16)), "batching": "static" if rng.random() < 0.25 else "continuous"}
    if kind == "linear":
        return {"kind": kind, "layer": rng.choice(sorted(SHAPES)), "rows": _log(rng, 1, 8192)}
    batch = _log(rng, 1, 256)
    return {"kind": kind, "batch": batch, "context": _log(rng, 100, min(32768, 2_000_000 // batch))}


def _lengths(count: int, shortest: int, longest: int) -> list[int]:
    """Ragged lengths from ``shortest`` to ``longest`` in no particular order; the first is the longest."""
    return [longest - int((longest - shortest) * ((i * 0.618034) % 1.0)) for i in range(count)]


# ---- models and inputs ----------------------------------------------------------------------
def _packed_linear(n: int, k: int, gen: torch.Generator, gain: float = 1.0) -> dict:
    """int4 values and zero points uniform in 0..15, scales |N(0, 0.01)| + 0.001 times ``gain``."""
    words = torch.randint(-2 ** 31, 2 ** 31, (n, k // 8), generator=gen, device=DEVICE, dtype=torch.int64)
    zeros = torch.randint(-2 ** 31, 2 ** 31, (n // 8, k // GROUP), generator=gen, device=DEVICE, dtype=torch.int64)
    scale = (torch.randn(n, k // GROUP, generator=gen, device=DEVICE).abs() * 0.01 + 1e-3) * gain
    return {"weight_packed": words.to(torch.int32), "weight_zero_point": zeros.to(torch.int32),
            "weight_scale": scale.half()}


@functools.cache
def _net(weights: str):
    """The model a program loads once and keeps; caches, prompts and requests come from the seed."""
    gen = torch.Generator(device=DEVICE).manual_seed(20)
    state = {}
    signs = torch.where(torch.rand(HIDDEN, generator=gen, device=DEVICE) < 0.5, -1.0, 1.0)
    half = torch.randn(VOCAB // 2, HIDDEN, generator=gen, device=DEVICE)
    state["model.embed_tokens.weight"] = torch.stack([half, half * signs], dim=1).view(VOCAB, HIDDEN).half()
    state["model.norm.weight"] = (signs * 0.5).half()
    for i in range(LAYERS):
        base = f"model.layers.{i}"
        for norm in ("input_layernorm", "post_attention_layernorm"):
            spread = torch.rand(HIDDEN, generator=gen, device=DEVICE)
            state[f"{base}.{norm}.weight"] = (0.75 + 0.5 * spread).half()
        for name, n, k, has_bias in _checkpoint.LAYER_LINEARS:
            if weights == "w4":
                for key, value in _packed_linear(n, k, gen, gain=0.3).items():
                    state[f"{base}.{name}.{key}"] = value
            else:
                state[f"{base}.{name}.weight"] = (torch.randn(n, k, generator=gen, device=DEVICE) * 0.02).half()
            if has_bias:
                state[f"{base}.{name}.bias"] = (torch.randn(n, generator=gen, device=DEVICE) * 0.02).half()
    return _model.from_state_dict(state, _checkpoint.qwen_config_dict(LAYERS, VOCAB), device=DEVICE)


def _prompts(lengths: list[int], seed: int) -> list[torch.Tensor]:
    gen = torch.Generator().manual_seed(seed)
    return [torch.randint(0, VOCAB, (n,), generator=gen) for n in lengths]


def prepare(case: dict, seed: int):
    kind = case["kind"]
    s = SimpleNamespace(case=case, kind=kind)
    if kind in ("decode", "prefill"):
        count = case["rows"] if kind == "decode" else case["seqs"]
        lengths = _lengths(count, case["shortest"], case["longest"])
        s.net, s.slots, s.prompts = _net(case["weights"]), list(range(count)), _prompts(lengths, seed)
        room = case["longest"] + (case["steps"] if kind == "decode" else 1)
        s.cache = s.net.new_cache(n_slots=count, s_max=(room + 63) // 64 * 64)
    if kind == "decode":
        for a in range(0, count, 16):  # admitted a few at a time
            s.net.prefill(s.cache, s.slots[a:a + 16], s.prompts[a:a + 16])
        s.tok, s.pos, s.lengths = s.cache.tok.clone(), s.cache.pos.clone(), list(s.cache.host_len)
        s.feed = torch.zeros(count, dtype=torch.int32).pin_memory()
        s.first = s.cache.tok.cpu().numpy()
        s.feed_values = s.feed.numpy()
    elif kind == "generate":
        s.net = _net("w4")
        lengths = _lengths(case["batch"], case["shortest"], case["longest"])
        s.ids = torch.zeros(case["batch"], case["longest"], dtype=torch.long)
        s.mask = torch.zeros_like(s.ids)
        for b, p in enumerate(_prompts(lengths, seed)):
            s.ids[b, -p.numel():] = p
            s.mask[b, -p.numel():] = 1
        s.ids, s.mask = s.ids.to(DEVICE), s.mask.to(DEVICE)
    elif kind == "serve":
        net = _net("w4")
        s.prompts = _prompts(_lengths(case["requests"], case["shortest"], case["longest"]), seed)
        s.budgets = _lengths(case["requests"], case["fewest"], case["most"])[::-1]
        room = case["longest"] + case["most"] + case["burst"]
        config = _config.EngineConfig(batching=case["batching"], decode_burst=case["burst"],
                                      max_context=(room + 127) // 128 * 128)
        s.engine = _engine.Engine(config=config, max_batch_size=case["slots"],
                                  model_module=SimpleNamespace(load=lambda **options: (net, None)))
    elif kind == "linear":
        k, n = SHAPES[case["layer"]]
        gen = torch.Generator(device=DEVICE).manual_seed(seed)
        s.weight = _kernels.W4Weight(n, k, torch.device(DEVICE, torch.cuda.current_device()))
        layer = _packed_linear(n, k, gen)
        s.weight.put(layer["weight_packed"], layer["weight_scale"], layer["weight_zero_point"])
        s.x = torch.randn(case["rows"], k, generator=gen, device=DEVICE).half()
        s.op = _kernels.w4a16()
    elif kind == "attention":
        b, ctx = case["batch"], case["context"]
        gen = torch.Generator(device=DEVICE).manual_seed(seed)
        s.q = torch.randn(b, 14, 1, 64, generator=gen, device=DEVICE, dtype=torch.float16)
        s.k = torch.randn(b, 2, ctx, 64, generator=gen, device=DEVICE, dtype=torch.float16)
        s.v = torch.randn(b, 2, ctx, 64, generator=gen, device=DEVICE, dtype=torch.float16)
        s.pads = torch.tensor(_pads(b, ctx), dtype=torch.int32, device=DEVICE)
        s.op = _kernels.flash_attn_decode()
    return s


def _pads(batch: int, context: int) -> list[int]:
    return [context // 4 - n for n in _lengths(batch, 0, context // 4)]


# ---- one pass ---------------------------------------------------------------------------------
def _rewind(s) -> None:
    """Back to the end of the prompts, as for another answer to the same question."""
    s.cache.tok.copy_(s.tok)
    s.cache.pos.copy_(s.pos)
    s.cache.host_len[:] = s.lengths


def run(s):
    case = s.case
    if s.kind == "decode":
        _rewind(s)
        if not case["fed"]:
            tokens = s.net.decode(s.cache, s.slots, case["steps"])
            return {"tokens": torch.tensor(tokens), "kv": s.cache.kv}
        tokens, values = [], s.feed_values
        values[:] = s.first
        for _ in range(case["steps"]):
            row = [t[0] for t in s.net.decode(s.cache, s.slots, 1, feed=s.feed)]
            tokens.append(row)
            values[:] = row
        return {"tokens": torch.tensor(tokens).t(), "kv": s.cache.kv}
    if s.kind == "prefill":
        first, logits = s.net.prefill(s.cache, s.slots, s.prompts)
        return {"first": first, "logits": logits, "kv": s.cache.kv, "pos": s.cache.pos}
    if s.kind == "generate":
        with torch.inference_mode():
            out = s.net(input_ids=s.ids, attention_mask=s.mask, use_cache=True)
            tokens = [out.logits[:, -1, :].argmax(dim=-1, keepdim=True)]
            for _ in range(case["tokens"] - 1):
                out = s.net(input_ids=tokens[-1], past_key_values=out.past_key_values, use_cache=True)
                tokens.append(out.logits[:, -1, :].argmax(dim=-1, keepdim=True))
            return {"tokens": torch.cat(tokens, dim=1), "logits": out.logits, "kv": out.past_key_values.kv}
    if s.kind == "serve":
        for prompt, budget in zip(s.prompts, s.budgets):
            s.engine.add_request_ids(prompt, max_tokens=budget)
        outputs = s.engine.run()
        return {"lengths": torch.tensor([len(o) for o in outputs]),
                "tokens": torch.tensor([t for o in outputs for t in o])}
    if s.kind == "linear":
        return s.op.forward(s.weight, s.x)
    return s.op.forward(s.q, s.k, s.v, 0.125, s.pads)


# ---- what a pass cannot do without --------------------------------------------------------------
def _weight_bytes(weights: str) -> float:
    """All linears of the layers with their scales and zero points, the norms and the biases."""
    per_param = 2.0 if weights == "fp16" else 0.5 + (2 + 0.5) / GROUP
    return LAYERS * (LAYER_PARAMS * per_param + 2 * (1152 + 2 * HIDDEN))


def _forward_flops(tokens: int, attended: float, heads: int) -> float:
    """Linears for ``tokens`` rows, attention over ``attended`` (query, key) pairs, ``heads`` rows of logits."""
    return 2.0 * LAYERS * LAYER_PARAMS * tokens + 4.0 * LAYERS * HIDDEN * attended + 2.0 * VOCAB * HIDDEN * heads


def _prefill_work(weights: str, lengths: list[int]) -> dict:
    rows, pairs = sum(lengths), sum(n * (n + 1) / 2 for n in lengths)
    return {"bytes": _weight_bytes(weights) + HEAD_BYTES + rows * (2 * HIDDEN + KV_TOKEN_BYTES) +
            2 * len(lengths) * VOCAB, "flops": _forward_flops(rows, pairs, len(lengths))}


def _decode_work(weights: str, rows: int, context: float, steps: int) -> dict:
    """``steps`` dependent steps; ``context`` = tokens cached over all rows before the first."""
    attended = steps * (context + rows * (steps + 1) / 2)
    return {"bytes": steps * (_weight_bytes(weights) + HEAD_BYTES) + KV_TOKEN_BYTES * (attended + steps * rows),
            "flops": _forward_flops(steps * rows, attended, steps * rows)}


def _plus(*parts: dict) -> dict:
    return {key: sum(p[key] for p in parts) for key in ("bytes", "flops")}


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "decode":
        lengths = _lengths(case["rows"], case["shortest"], case["longest"])
        return _decode_work(case["weights"], case["rows"], sum(lengths), case["steps"])
    if kind == "prefill":
        return _prefill_work(case["weights"], _lengths(case["seqs"], case["shortest"], case["longest"]))
    if kind == "generate":
        lengths = _lengths(case["batch"], case["shortest"], case["longest"])
        return _plus(_prefill_work("w4", lengths),
                     _decode_work("w4", case["batch"], sum(lengths), case["tokens"] - 1))
    if kind == "serve":
        # every slot busy: a step reads the weights once for `slots` rows
        prompts = _lengths(case["requests"], case["shortest"], case["longest"])
        budgets = _lengths(case["requests"], case["fewest"], case["most"])[::-1]
        steps = max(max(budgets), sum(budgets) / case["slots"])
        attended = sum(m * (p + (m + 1) / 2) for p, m in zip(prompts, budgets))
        decode = {"bytes": steps * (_weight_bytes("w4") + HEAD_BYTES) + KV_TOKEN_BYTES * attended,
                  "flops": _forward_flops(sum(budgets), attended, sum(budgets))}
        return _plus(_prefill_work("w4", prompts), decode)
    if kind == "linear":
        (k, n), m = SHAPES[case["layer"]], case["rows"]
        return {"bytes": n * k * (0.5 + 2.5 / GROUP) + 2 * m * (k + n), "flops": 2.0 * m * n * k}
    tokens = sum(case["context"] - p for p in _pads(case["batch"], case["context"]))
    return {"bytes": 512.0 * tokens + 4 * 896 * case["batch"], "flops": 4.0 * 896 * tokens}


def tolerance(case: dict) -> dict:
    if case["kind"] == "linear":
        return {"rel": 1e-3}  # fp32 sums rounded to fp16
    if case["kind"] == "attention":
        return {"rel": 2e-3}  # probabilities and outputs in fp16
    # fp16 activations through 24 layers; token ids are decided by a wide margin
    return {"rel": 1e-2}
