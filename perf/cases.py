"""What a user of this framework has it do, as a list of timed cases: serving (prompts in, given tokens after them), training steps, and
the two kernel families that are also called on their own, packed attention and routed experts, in both directions.

Models are the presets of this repository with random weights; ``layers`` cuts their depth so that three states fit one GPU (every
layer of a model does the same work). Weights and inputs come from the seed alone. ``exact`` restates each path in 64 bits with plain
torch.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

DEV = "cuda"


# ----------------------------------------------------------------------------------------------------------------- cases
def listed() -> list[dict]:
    return [
        # one chat turn: a short prompt, then token by token; launches and latency are all there is
        _serve("chat_one_stream", "qwen2.5-0.5b", 12, streams=1, prompt=100, steps=16),
        # rollouts of a small policy: many streams of uneven length decoded together
        _serve("rollout_small_policy", "qwen2.5-0.5b", 12, streams=128, prompt=96, steps=24),
        # rollouts of an 8B-shaped policy: weights stream from memory at every step
        _serve("rollout_8b_shape", "llama-3-8b", 8, streams=32, prompt=72, steps=16),
        # a wave of prompts entering the cache together, lengths as they come
        _serve("prefill_ragged", "qwen2.5-0.5b", 12, streams=16, prompt=1000, steps=0),
        # one long document, small and 8B-shaped model
        _serve("prefill_long_small", "qwen2.5-0.5b", 12, streams=1, prompt=16384, steps=0),
        _serve("prefill_long_8b_shape", "llama-3-8b", 8, streams=1, prompt=8192, steps=0),
        # a latent-attention layer stack: prompts, then a few tokens
        _serve("latent_prompt_and_decode", "lulezen-1b", 8, streams=4, prompt=2048, steps=8),
        # an update of a small policy on sampled completions (GRPO), sequences shorter than the batch is wide
        _train("grpo_update_small", "qwen2.5-0.5b", 4, batch=16, seq=512, micro=16, loss="grpo"),
        # supervised training of the 8B shape at its usual length
        _train("sft_step_8b_shape", "llama-3-8b", 2, batch=1, seq=4096, micro=1, loss="sft"),
        # packed attention of a training step, documents of uneven length, both directions
        _attention("attention_packed_train", 32, 8, 128, docs=5, longest=6000, window=0),
        # the same with the small heads, few kv heads and short sequences of policy updates
        _attention("attention_short_train", 14, 2, 64, docs=24, longest=640, window=0),
        # one layer's routed experts in training, 8 of 128
        _experts("experts_train", tokens=4096, top=8, experts=128, width=2048, ff=768),
    ]


def _serve(name, model, layers, streams, prompt, steps):
    return _named(name, dict(kind="serve", model=model, layers=layers, streams=streams, prompt=prompt, steps=steps))


def _train(name, model, layers, batch, seq, micro, loss):
    return _named(name, dict(kind="train", model=model, layers=layers, batch=batch, seq=seq, micro=micro, loss=loss))


def _attention(name, heads, kv_heads, dim, docs, longest, window):
    return _named(name, dict(kind="attention", heads=heads, kv_heads=kv_heads, dim=dim, docs=docs, longest=longest, window=window))


def _experts(name, tokens, top, experts, width, ff):
    return _named(name, dict(kind="experts", tokens=tokens, top=top, experts=experts, width=width, ff=ff))


def _named(name, case):
    return case if name is None else {"name": name, **case}


def _spread(rng, lo: int, hi: int) -> int:
    """A whole number, its logarithm uniform over [lo, hi]."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng) -> dict:
    kind = rng.choice(("serve", "serve", "train", "attention", "attention", "experts"))
    if kind == "serve":
        model, layers, most = rng.choice((("qwen2.5-0.5b", 12, 16384), ("llama-3-8b", 8, 8192), ("lulezen-1b", 8, 8192)))
        streams = _spread(rng, 1, 128)
        steps = rng.choice((0, 0, 4, 8, 16))
        return _serve(None, model, layers, streams, _spread(rng, 2, min(most // streams, most // 2)), steps)
    if kind == "train":
        if rng.random() < 0.5:
            batch = _spread(rng, 1, 16)
            return _train(None, "qwen2.5-0.5b", 4, batch, _spread(rng, 64, 8192 // batch), rng.choice((1, batch)) if batch <= 4 else batch,
                          rng.choice(("grpo", "sft")))
        return _train(None, "llama-3-8b", 2, 1, _spread(rng, 64, 4096), 1, rng.choice(("grpo", "sft")))
    if kind == "attention":
        heads, kv_heads, dim = rng.choice(((32, 8, 128), (32, 4, 128), (14, 2, 64), (16, 16, 128), (8, 8, 64)))
        docs = _spread(rng, 1, 48)
        longest = _spread(rng, 16, min(8192, 20000 // docs))
        return _attention(None, heads, kv_heads, dim, docs, longest, rng.choice((0, 0, 0, 1024, 333)))
    top, experts, width, ff = rng.choice(((8, 128, 2048, 768), (2, 8, 4096, 3584), (2, 8, 1024, 1408)))
    return _experts(None, _spread(rng, 16, 4096), top, experts, width, ff)


def _lengths(count: int, longest: int) -> list[int]:
    """Uneven lengths between a quarter of the longest and the longest, the same for every seed."""
    room = max(1, longest - longest // 4)
    return [longest - (i * 7919 * 31) % room for i in range(count)]


# --------------------------------------------------------------------------------------------------------------- weights
def _gen(seed: int, salt: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(seed * 100003 + salt)


def _normal(seed, salt, shape, std, mean=0.0, dtype=torch.bfloat16):
    t = torch.empty(shape, dtype=dtype, device=DEV)
    return t.normal_(mean, std, generator=_gen(seed, salt))


def _sizes(case) -> dict:
    """Sizes of the dense presets, as published for these shapes."""
    if case["model"] == "qwen2.5-0.5b":
        return dict(vocab=151936, width=896, heads=14, kv_heads=2, dim=64, ff=4864, theta=1e6, eps=1e-6, bias=True, tied=True)
    if case["model"] == "llama-3-8b":
        return dict(vocab=128256, width=4096, heads=32, kv_heads=8, dim=128, ff=14336, theta=5e5, eps=1e-5, bias=False, tied=False)
    return dict(vocab=32000, width=2048, heads=16, dim=128, rot=64, vdim=128, kv_rank=512, q_rank=1024, window=4096, ff=8192, theta=5e5,
                eps=1e-6, limit=7.0, cap=30.0)


def _dense_weights(case, seed) -> dict[str, torch.Tensor]:
    """Projections at the usual scale, query and key projections such that scores spread by about one, norm weights near one."""
    z = _sizes(case)
    d, hd = z["width"], z["dim"]
    out, salt = {}, 0

    def put(name, shape, std, mean=0.0):
        nonlocal salt
        salt += 1
        out[name] = _normal(seed, salt, shape, std, mean)

    put("model.embed_tokens.weight", (z["vocab"], d), 0.02)
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        put(p + "input_layernorm.weight", (d,), 0.1, 1.0)
        put(p + "post_attention_layernorm.weight", (d,), 0.1, 1.0)
        for name, heads in (("q", z["heads"]), ("k", z["kv_heads"]), ("v", z["kv_heads"])):
            put(f"{p}self_attn.{name}_proj.weight", (heads * hd, d), 0.02 if name == "v" else 1.1 / math.sqrt(d))
            if z["bias"]:
                put(f"{p}self_attn.{name}_proj.bias", (heads * hd,), 0.1)
        put(p + "self_attn.o_proj.weight", (d, z["heads"] * hd), 0.02)
        put(p + "mlp.gate_proj.weight", (z["ff"], d), 0.02)
        put(p + "mlp.up_proj.weight", (z["ff"], d), 0.02)
        put(p + "mlp.down_proj.weight", (d, z["ff"]), 0.02)
    put("model.norm.weight", (d,), 0.1, 1.0)
    if not z["tied"]:
        put("lm_head.weight", (z["vocab"], d), 0.02)
    return out


def _latent_weights(case, seed) -> dict[str, torch.Tensor]:
    z = _sizes(case)
    d, H = z["width"], z["heads"]
    out, salt = {}, 0

    def put(name, shape, std, mean=0.0):
        nonlocal salt
        salt += 1
        out[name] = _normal(seed, salt, shape, std, mean)

    put("embed", (z["vocab"], d), 0.02)
    for i in range(case["layers"]):
        m = f"l{i}.mix."
        for n in ("1", "2"):
            put(f"l{i}.norm{n}", (d,), 0.1, 1.0)
            put(f"l{i}.norm{n}.b", (d,), 0.02)
            put(f"l{i}.ls{n}", (d,), 0.02, 0.2)
        put(m + "dq", (z["q_rank"], d), 0.02)
        put(m + "dq.norm", (z["q_rank"],), 0.1, 1.0)
        put(m + "uq", (H * (z["dim"] + z["rot"]), z["q_rank"]), 0.02)
        put(m + "dkv", (z["kv_rank"] + z["rot"], d), 0.02)
        put(m + "dkv.norm", (z["kv_rank"],), 0.1, 1.0)
        put(m + "uk", (H * z["dim"], z["kv_rank"]), 0.03)
        put(m + "uv", (H * z["vdim"], z["kv_rank"]), 0.03)
        put(m + "sink", (H,), 0.5)
        put(m + "g", (H, d), 0.02)
        put(m + "o", (d, H * z["vdim"]), 0.02)
        put(f"l{i}.mlp.gate", (z["ff"], d), 0.02)
        put(f"l{i}.mlp.up", (z["ff"], d), 0.02)
        put(f"l{i}.mlp.down", (d, z["ff"]), 0.02)
    put("final.norm", (d,), 0.1, 1.0)
    put("final.norm.b", (d,), 0.02)
    put("head", (z["vocab"], d), 0.02)
    return out


def _weights(case, seed):
    return _latent_weights(case, seed) if case["model"] == "lulezen-1b" else _dense_weights(case, seed)


def _model_config(case):
    from research_b200.models import get_preset

    cfg = get_preset(case["model"])
    if case["model"] == "lulezen-1b":
        return get_preset(case["model"], vocab_size=_sizes(case)["vocab"], layers=cfg.layers[:case["layers"]])
    return get_preset(case["model"], num_layers=case["layers"])


def _tokens(case, seed, vocab, shape) -> torch.Tensor:
    return torch.randint(0, vocab, shape, generator=torch.Generator().manual_seed(seed * 7 + 3))


# ----------------------------------------------------------------------------------------------------------------- serve
def _prepare_serve(case, seed) -> dict:
    from research_b200.inference import EngineConfig, InferenceEngine

    lengths, steps = _lengths(case["streams"], case["prompt"]), case["steps"]
    batch = case["streams"] + case["streams"] % 2
    most = max(lengths) + steps + 16
    engine = InferenceEngine(EngineConfig(
        cache_type="none", max_batch_size=batch, max_model_len=most, max_tokens_per_batch=sum(lengths) + sum(lengths) % 2,
        num_kv_blocks=sum(-(-(n + steps) // 16) for n in lengths) + 8, graph_batch_sizes=(batch,), ignore_eos=True),
        _model_config(case), _weights(case, seed), device=DEV)
    return {"case": case, "engine": engine, **_streams(case, seed)}


def _streams(case, seed) -> dict:
    lengths, vocab = _lengths(case["streams"], case["prompt"]), _sizes(case)["vocab"]
    flat = _tokens(case, seed, vocab, (sum(lengths) + case["streams"] * case["steps"],)).tolist()
    prompts, at = [], 0
    for n in lengths:
        prompts.append(flat[at:at + n])
        at += n
    after = [[flat[at + s * case["streams"] + i] for i in range(case["streams"])] for s in range(case["steps"])]
    return {"prompts": prompts, "after": after}


def _run_serve(s) -> list[torch.Tensor]:
    """Prompts into the cache, then the given tokens one by one; the logits behind every prompt and every given token."""
    engine = s["engine"]
    ids = [engine.open_stream() for _ in s["prompts"]]
    out = [engine.feed([(i, p, [len(p) - 1]) for i, p in zip(ids, s["prompts"])])]
    for tokens in s["after"]:
        out.append(engine.feed([(i, [t], [0]) for i, t in zip(ids, tokens)]))
    for i in ids:
        engine.close_stream(i)
    return out


def _work_serve(case) -> dict:
    z, L, n, steps = _sizes(case), case["layers"], case["streams"], case["steps"]
    lengths = _lengths(n, case["prompt"])
    d = z["width"]
    if case["model"] == "lulezen-1b":
        qk, vd = z["dim"] + z["rot"], z["vdim"]
        layer = d * z["q_rank"] + z["q_rank"] * z["heads"] * qk + d * (z["kv_rank"] + z["rot"]) + z["kv_rank"] * z["heads"] * (z["dim"] + vd)
        layer += z["heads"] * vd * d + 3 * d * z["ff"]
        per_pair, cached = 2 * z["heads"] * (qk + vd), 2 * (z["kv_rank"] + z["rot"])
    else:
        layer = d * (z["heads"] + 2 * z["kv_heads"]) * z["dim"] + z["heads"] * z["dim"] * d + 3 * d * z["ff"]
        per_pair, cached = 4 * z["heads"] * z["dim"], 4 * z["kv_heads"] * z["dim"]
    head = z["vocab"] * d
    tokens = sum(lengths) + n * steps
    pairs = sum((x + steps) * (x + steps + 1) // 2 for x in lengths)
    flops = 2 * L * layer * tokens + 2 * head * n * (1 + steps) + L * per_pair * pairs
    read_back = sum(x * steps + steps * (steps + 1) // 2 for x in lengths)       # keys that the single tokens read
    nbytes = (1 + steps) * 2 * (L * layer + head) + L * cached * (tokens + read_back) + 4 * z["vocab"] * n * (1 + steps)
    return {"bytes": nbytes, "flops": flops}


# ----------------------------------------------------------------------------------------------------------------- train
def _batch(case, seed) -> dict[str, torch.Tensor]:
    """Host tensors, as a data loader or a rollout hands them over: completions of uneven length behind a prompt quarter, in training on
    text every position."""
    B, T = case["batch"], case["seq"]
    ids = _tokens(case, seed, _sizes(case)["vocab"], (B, T))
    if case["loss"] == "sft":
        mask = torch.ones(B, T)
    else:
        ends = torch.tensor(_lengths(B, T))
        pos = torch.arange(T)[None]
        mask = ((pos >= T // 4) & (pos < ends[:, None])).float()
    g = torch.Generator().manual_seed(seed + 99)
    return {"input_ids": ids, "labels": ids.clone(), "loss_mask": mask, "advantages": torch.randn(B, generator=g)}


def _prepare_train(case, seed) -> dict:
    from research_b200.training import TrainerConfig
    from research_b200.training.backends import PyTorchTrainingBackend

    backend = PyTorchTrainingBackend(_model_config(case), _weights(case, seed), device=DEV, loss_fn=case["loss"], lr=1e-6,
                                     trainer_config=TrainerConfig(micro_batch_size=case["micro"]), need_entropy=False)
    return {"case": case, "backend": backend, "batch": _batch(case, seed), "names": list(_dense_names(case))}


def _dense_names(case):
    z = _sizes(case)
    yield "model.embed_tokens.weight"
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        yield p + "input_layernorm.weight"
        yield p + "post_attention_layernorm.weight"
        for n in "qkv":
            yield f"{p}self_attn.{n}_proj.weight"
            if z["bias"]:
                yield f"{p}self_attn.{n}_proj.bias"
        yield p + "self_attn.o_proj.weight"
        for n in ("gate", "up", "down"):
            yield f"{p}mlp.{n}_proj.weight"
    yield "model.norm.weight"
    if not z["tied"]:
        yield "lm_head.weight"


def _run_train(s) -> dict:
    """One step: forward, backward, clipping and AdamW; the loss and every gradient."""
    backend = s["backend"]
    metrics = backend.forward_backward(s["batch"]).wait()
    backend.optim_step().wait()
    return {"loss": metrics["loss" if s["case"]["loss"] == "sft" else "pg_loss"],
            "grads": {n: backend.buckets.grad_view(n) for n in s["names"]}}


def _work_train(case) -> dict:
    z, L, tokens = _sizes(case), case["layers"], case["batch"] * case["seq"]
    d = z["width"]
    layer = d * (z["heads"] + 2 * z["kv_heads"]) * z["dim"] + z["heads"] * z["dim"] * d + 3 * d * z["ff"]
    head = z["vocab"] * d
    params = L * layer + head * (1 if z["tied"] else 2)
    pairs = case["batch"] * case["seq"] * (case["seq"] + 1) // 2
    flops = 6 * (L * layer + head) * tokens + 3.5 * L * 4 * z["heads"] * z["dim"] * pairs
    # weights read in each direction, gradients written and read, 30 bytes a parameter for the update, the stream both ways
    return {"bytes": params * (2 + 2 + 2 + 30) + 8 * L * tokens * d * 2, "flops": flops}


# ------------------------------------------------------------------------------------------------------------- attention
def _prepare_attention(case, seed) -> dict:
    lengths = _lengths(case["docs"], case["longest"])
    T, H, Hkv, D = sum(lengths), case["heads"], case["kv_heads"], case["dim"]
    cu = torch.tensor([0] + [sum(lengths[:i + 1]) for i in range(len(lengths))], dtype=torch.int32, device=DEV)
    q, k, v = (_normal(seed, i, (T, h, D), 1.0).requires_grad_(True) for i, h in ((1, H), (2, Hkv), (3, Hkv)))
    return {"case": case, "q": q, "k": k, "v": v, "cu": cu, "longest": max(lengths), "dout": _normal(seed, 4, (T, H, D), 1.0)}


def _run_attention(s) -> list[torch.Tensor]:
    from research_b200 import ops

    q, k, v, n = s["q"], s["k"], s["v"], s["longest"]
    out = ops.flash_attention(q, k, v, s["cu"], s["cu"], n, n, causal=True, window=s["case"]["window"])
    return [out, *torch.autograd.grad(out, (q, k, v), s["dout"])]


def _seen(n: int, window: int) -> int:
    """Query and key pairs of a causal sequence of ``n``, with a window over the last so many keys or none (0)."""
    w = min(window, n) if window > 0 else n
    return w * (w + 1) // 2 + (n - w) * w


def _work_attention(case) -> dict:
    lengths = _lengths(case["docs"], case["longest"])
    T, D = sum(lengths), case["dim"]
    pairs = sum(_seen(n, case["window"]) for n in lengths)
    # q, k, v, dout read; out, dq, dk, dv written
    return {"bytes": 2 * T * D * (4 * case["heads"] + 4 * case["kv_heads"]), "flops": 3.5 * 4 * case["heads"] * D * pairs}


# --------------------------------------------------------------------------------------------------------------- experts
class _Fresh:
    """Every gradient view is written for the first time."""

    @staticmethod
    def accumulate_into(view) -> bool:
        return False


def _expert_inputs(case, seed) -> dict:
    T, E, d, f = case["tokens"], case["experts"], case["width"], case["ff"]
    score = _normal(seed, 5, (T, E), 1.0, dtype=torch.float32) + _normal(seed, 6, (E,), 0.5, dtype=torch.float32)     # some experts are liked better
    wt, idx = score.softmax(-1).topk(case["top"], dim=-1)
    return {"h": _normal(seed, 1, (T, d), 0.5), "wgu": _normal(seed, 2, (E * 2 * f, d), 0.02), "wd": _normal(seed, 3, (E * d, f), 0.02),
            "dout": _normal(seed, 4, (T, d), 0.1), "wt": (wt / wt.sum(-1, keepdim=True)).contiguous(), "idx": idx.to(torch.int32).contiguous()}


def _prepare_experts(case, seed) -> dict:
    s = _expert_inputs(case, seed)
    s["h"].requires_grad_(True)
    s["wt"].requires_grad_(True)
    return {"case": case, **s, "ggu": torch.empty_like(s["wgu"]), "gd": torch.empty_like(s["wd"])}


def _run_experts(s) -> dict:
    from research_b200.ops.moe_train import GroupedExperts, GroupedPlan

    c = s["case"]
    plan = GroupedPlan(s["idx"], c["experts"], c["width"], c["ff"])
    out = GroupedExperts.apply(s["h"], s["wt"], s["wgu"], s["ggu"], s["wd"], s["gd"], plan, _Fresh)
    dh, dwt = torch.autograd.grad(out, (s["h"], s["wt"]), s["dout"])
    return {"out": out, "dh": dh, "dwt": dwt, "ggu": s["ggu"], "gd": s["gd"]}


def _work_experts(case) -> dict:
    rows, E, d, f = case["tokens"] * case["top"], case["experts"], case["width"], case["ff"]
    used = min(E, rows)
    return {"bytes": 2 * 3 * d * f * (used + E) + 2 * 4 * case["tokens"] * d, "flops": 3 * 2 * rows * 3 * d * f}


# ------------------------------------------------------------------------------------------------------------- interface
_KINDS = {"serve": (_prepare_serve, _run_serve, _work_serve), "train": (_prepare_train, _run_train, _work_train),
          "attention": (_prepare_attention, _run_attention, _work_attention), "experts": (_prepare_experts, _run_experts, _work_experts)}


def prepare(case: dict, seed: int) -> dict:
    return _KINDS[case["kind"]][0](case, seed)


def run(state: dict):
    return _KINDS[state["case"]["kind"]][1](state)


def work(case: dict) -> dict:
    return _KINDS[case["kind"]][2](case)


def tolerance(case: dict) -> dict:
    """bf16 activations between the layers of a whole model, rounded at other places (another attention kernel, norms outside the
    products), moved its logits by up to 2 % and its gradients by 2 %, single gradients by more; one kernel alone by less."""
    if case["kind"] == "serve":
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 0.03, "max": 0.95} if case["kind"] == "train" else {"rel": 0.01, "max": 0.2}


# ----------------------------------------------------------------------------------------------------------------- exact
def exact(case: dict, seed: int):
    with torch.no_grad():
        return {"serve": _exact_serve, "train": _exact_train, "attention": _exact_attention, "experts": _exact_experts}[case["kind"]](case, seed)


def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _layer_norm(x, w, b, eps):
    return F.layer_norm(x, x.shape[-1:], w, b, eps)


def _rotated(x, theta, dims):
    """Pairs ``(i, i + dims / 2)`` of the last axis turned by the position (first axis) times ``theta ** (-2 i / dims)``."""
    half = dims // 2
    angle = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * theta ** (
        -torch.arange(half, dtype=torch.float64, device=x.device) / half)
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _visible(rows, n, window):
    """``[len(rows), n]``: which keys the positions ``rows`` see."""
    j = torch.arange(n, device=rows.device)
    seen = j[None] <= rows[:, None]
    return seen & (j[None] > rows[:, None] - window) if window > 0 else seen


def _attend(q, k, v, scale, window=0, sink=None):
    """Causal attention of one sequence in 64 bits, in blocks of rows; ``q [n, H, D]``, ``k``/``v [n, Hkv, ·]``."""
    n, H = q.shape[:2]
    g = H // k.shape[1]
    out = torch.empty(n, H, v.shape[-1], dtype=q.dtype, device=q.device)
    for h in range(H):
        kh, vh = k[:, h // g], v[:, h // g]
        for r0 in range(0, n, 4096):
            rows = torch.arange(r0, min(n, r0 + 4096), device=q.device)
            top = int(rows[-1]) + 1
            s = (q[r0:top, h] @ kh[:top].T).mul_(scale).masked_fill_(~_visible(rows, top, window), -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(len(rows), 1)], -1)
            p = s.softmax(-1)
            out[r0:top, h] = p[:, :top] @ vh[:top]
    return out


def _dense_forward(z, w, layers, ids):
    """Final-normed rows of one sequence."""
    x = w["model.embed_tokens.weight"][ids].double()
    n = len(ids)
    for i in range(layers):
        p = f"model.layers.{i}."
        h = _rms(x, w[p + "input_layernorm.weight"], z["eps"])
        q, k, v = (F.linear(h, w[f"{p}self_attn.{s}_proj.weight"], w.get(f"{p}self_attn.{s}_proj.bias")).view(n, -1, z["dim"]) for s in "qkv")
        o = _attend(_rotated(q, z["theta"], z["dim"]), _rotated(k, z["theta"], z["dim"]), v, z["dim"] ** -0.5)
        x = x + o.reshape(n, -1) @ w[p + "self_attn.o_proj.weight"].T
        h = _rms(x, w[p + "post_attention_layernorm.weight"], z["eps"])
        x = x + (F.silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
    return _rms(x, w["model.norm.weight"], z["eps"])


def _latent_forward(z, w, layers, ids):
    x = w["embed"][ids].double()
    n, H, dim, rank, eps = len(ids), z["heads"], z["dim"], z["kv_rank"], z["eps"]
    scale = (dim + z["rot"]) ** -0.5
    for i in range(layers):
        m, f = f"l{i}.mix.", f"l{i}.mlp."
        q = (_rms(x @ w[m + "dq"].T, w[m + "dq.norm"], eps) @ w[m + "uq"].T).view(n, H, -1)
        down = x @ w[m + "dkv"].T
        c = _rms(down[:, :rank], w[m + "dkv.norm"], eps)
        kr = _rotated(down[:, None, rank:], z["theta"], z["rot"]).expand(n, H, z["rot"])
        q = torch.cat([q[..., :dim], _rotated(q[..., dim:], z["theta"], z["rot"])], -1)
        k = torch.cat([(c @ w[m + "uk"].T).view(n, H, dim), kr], -1)
        o = _attend(q, k, (c @ w[m + "uv"].T).view(n, H, -1), scale, z["window"], w[m + "sink"])
        o = o * torch.sigmoid(x @ w[m + "g"].T)[..., None]
        x = x + _layer_norm(o.reshape(n, -1) @ w[m + "o"].T, w[f"l{i}.norm1"], w[f"l{i}.norm1.b"], eps) * w[f"l{i}.ls1"]
        g, u = (x @ w[f + "gate"].T).clamp(max=z["limit"]), (x @ w[f + "up"].T).clamp(-z["limit"], z["limit"])
        y = (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[f + "down"].T
        x = x + _layer_norm(y, w[f"l{i}.norm2"], w[f"l{i}.norm2.b"], eps) * w[f"l{i}.ls2"]
    return _layer_norm(x, w["final.norm"], w["final.norm.b"], eps)


def _exact_serve(case, seed):
    z, s = _sizes(case), _streams(case, seed)
    w = {k: v.double() for k, v in _weights(case, seed).items()}
    latent = case["model"] == "lulezen-1b"
    head = w["head"] if latent else w["model.embed_tokens.weight" if z["tied"] else "lm_head.weight"]
    rows = []
    for i, p in enumerate(s["prompts"]):
        ids = torch.tensor(p + [t[i] for t in s["after"]], device=DEV)
        rows.append((_latent_forward if latent else _dense_forward)(z, w, case["layers"], ids)[len(p) - 1:])
    out = []
    for k in range(case["steps"] + 1):
        logits = torch.stack([r[k] for r in rows]) @ head.T
        out.append(z["cap"] * torch.tanh(logits / z["cap"]) if latent else logits)
    return out


def _rms_back(dy, x, w, eps):
    """Gradients of ``_rms`` to ``x`` and ``w``."""
    r = torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    g = dy * w
    return r * g - x * r ** 3 * (g * x).mean(-1, keepdim=True), (dy * x * r).sum(0)


def _attend_back(q, k, v, out, dout, scale, window=0):
    dq, dk, dv = torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
    n, H = q.shape[:2]
    g = H // k.shape[1]
    for h in range(H):
        kh, vh = k[:, h // g], v[:, h // g]
        for r0 in range(0, n, 4096):
            rows = torch.arange(r0, min(n, r0 + 4096), device=q.device)
            top = int(rows[-1]) + 1
            do = dout[r0:top, h]
            p = (q[r0:top, h] @ kh[:top].T).mul_(scale).masked_fill_(~_visible(rows, top, window), -math.inf).softmax(-1)
            dv[:top, h // g] += p.T @ do
            ds = p * (do @ vh[:top].T - (do * out[r0:top, h]).sum(-1, keepdim=True)) * scale
            dq[r0:top, h] = ds @ kh[:top]
            dk[:top, h // g] += ds.T @ q[r0:top, h]
    return dq, dk, dv


def _unrotated(x, theta, dims):
    """The turn of ``_rotated`` the other way: its transpose."""
    half = dims // 2
    swap = torch.cat([x[..., half:], x[..., :half]], -1)                # (a, b) -> (b, a) turns the rotation around
    y = _rotated(swap, theta, dims)
    return torch.cat([y[..., half:], y[..., :half]], -1)


def _exact_train(case, seed):
    """Forward with every intermediate kept, then backward by hand, sequence by sequence."""
    z, L, b = _sizes(case), case["layers"], _batch(case, seed)
    w = {k: v.double() for k, v in _dense_weights(case, seed).items()}
    head = "model.embed_tokens.weight" if z["tied"] else "lm_head.weight"
    grads = {k: torch.zeros_like(v) for k, v in w.items()}
    B, T, micro = case["batch"], case["seq"], case["micro"]
    eps, scale = z["eps"], z["dim"] ** -0.5
    loss = 0.0
    mask = b["loss_mask"][:, 1:].double().to(DEV)                       # position t is scored on token t + 1
    for i in range(B):
        ids = b["input_ids"][i].to(DEV)
        group = mask[i // micro * micro:(i // micro + 1) * micro]
        # weight of every position's log-probability in the mean over the micro-batches
        if case["loss"] == "sft":
            weight = -mask[i] / group.sum().clamp(min=1) * (micro / B)
        else:
            weight = -mask[i] / mask[i].sum().clamp(min=1) * float(b["advantages"][i]) / B
        x, kept = w["model.embed_tokens.weight"][ids], []
        for layer in range(L):
            p = f"model.layers.{layer}."
            h = _rms(x, w[p + "input_layernorm.weight"], eps)
            q, k, v = (F.linear(h, w[f"{p}self_attn.{s}_proj.weight"], w.get(f"{p}self_attn.{s}_proj.bias")).view(T, -1, z["dim"]) for s in "qkv")
            q, k = _rotated(q, z["theta"], z["dim"]), _rotated(k, z["theta"], z["dim"])
            o = _attend(q, k, v, scale)
            x1 = x + o.reshape(T, -1) @ w[p + "self_attn.o_proj.weight"].T
            h2 = _rms(x1, w[p + "post_attention_layernorm.weight"], eps)
            g, u = h2 @ w[p + "mlp.gate_proj.weight"].T, h2 @ w[p + "mlp.up_proj.weight"].T
            kept.append((x, h, q, k, v, o, x1, h2, g, u))
            x = x1 + (F.silu(g) * u) @ w[p + "mlp.down_proj.weight"].T
        hf = _rms(x, w["model.norm.weight"], eps)
        dhf = torch.zeros_like(hf)
        for r0 in range(0, T - 1, 1024):
            r1 = min(T - 1, r0 + 1024)
            lp = (hf[r0:r1] @ w[head].T).log_softmax(-1)
            tgt = ids[r0 + 1:r1 + 1, None]
            loss += float((lp.gather(-1, tgt)[:, 0] * weight[r0:r1]).sum())
            d = lp.exp_().mul_(-weight[r0:r1, None])
            d.scatter_add_(1, tgt, weight[r0:r1, None])
            grads[head] += d.T @ hf[r0:r1]
            dhf[r0:r1] = d @ w[head]
        dx, dw = _rms_back(dhf, x, w["model.norm.weight"], eps)
        grads["model.norm.weight"] += dw
        for layer in reversed(range(L)):
            p = f"model.layers.{layer}."
            x, h, q, k, v, o, x1, h2, g, u = kept[layer]
            sg = torch.sigmoid(g)
            grads[p + "mlp.down_proj.weight"] += dx.T @ (g * sg * u)
            dact = dx @ w[p + "mlp.down_proj.weight"]
            dg, du = dact * u * (sg + g * sg * (1 - sg)), dact * g * sg
            grads[p + "mlp.gate_proj.weight"] += dg.T @ h2
            grads[p + "mlp.up_proj.weight"] += du.T @ h2
            dn, dw = _rms_back(dg @ w[p + "mlp.gate_proj.weight"] + du @ w[p + "mlp.up_proj.weight"], x1, w[p + "post_attention_layernorm.weight"], eps)
            grads[p + "post_attention_layernorm.weight"] += dw
            dx = dx + dn
            grads[p + "self_attn.o_proj.weight"] += dx.T @ o.reshape(T, -1)
            dq, dk, dv = _attend_back(q, k, v, o, (dx @ w[p + "self_attn.o_proj.weight"]).view_as(o), scale)
            dq, dk = _unrotated(dq, z["theta"], z["dim"]), _unrotated(dk, z["theta"], z["dim"])
            dh = 0.0
            for s, t in (("q", dq), ("k", dk), ("v", dv)):
                t = t.reshape(T, -1)
                grads[f"{p}self_attn.{s}_proj.weight"] += t.T @ h
                if z["bias"]:
                    grads[f"{p}self_attn.{s}_proj.bias"] += t.sum(0)
                dh = dh + t @ w[f"{p}self_attn.{s}_proj.weight"]
            dn, dw = _rms_back(dh, x, w[p + "input_layernorm.weight"], eps)
            grads[p + "input_layernorm.weight"] += dw
            dx = dx + dn
        grads["model.embed_tokens.weight"].index_add_(0, ids, dx)
    return {"loss": loss, "grads": {n: grads[n] for n in _dense_names(case)}}


def _exact_attention(case, seed):
    s = _prepare_attention(case, seed)
    q, k, v, dout = (s[n].detach().double() for n in ("q", "k", "v", "dout"))
    scale, cu, window = case["dim"] ** -0.5, s["cu"].tolist(), case["window"]
    out, dq, dk, dv = torch.empty_like(q), torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    for a, b in zip(cu, cu[1:]):
        out[a:b] = _attend(q[a:b], k[a:b], v[a:b], scale, window)
        dq[a:b], dk[a:b], dv[a:b] = _attend_back(q[a:b], k[a:b], v[a:b], out[a:b], dout[a:b], scale, window)
    return [out, dq, dk, dv]


def _exact_experts(case, seed):
    s = _expert_inputs(case, seed)
    h, wt, dout, idx = s["h"].double(), s["wt"].double(), s["dout"].double(), s["idx"].long()
    E, d, f = case["experts"], case["width"], case["ff"]
    out, dh, dwt = torch.zeros_like(h), torch.zeros_like(h), torch.zeros_like(wt)
    ggu, gd = (torch.zeros_like(s[n], dtype=torch.float64) for n in ("wgu", "wd"))
    for e in range(E):
        tok, slot = (idx == e).nonzero(as_tuple=True)
        wgu, wd = s["wgu"][e * 2 * f:(e + 1) * 2 * f].double(), s["wd"][e * d:(e + 1) * d].double()
        x, c = h[tok], wt[tok, slot][:, None]
        g, u = (x @ wgu.T).split(f, -1)
        sg = torch.sigmoid(g)
        act = g * sg * u
        y = act @ wd.T
        out.index_add_(0, tok, y * c)
        dwt[tok, slot] = (dout[tok] * y).sum(-1)
        dy = dout[tok] * c
        dact = dy @ wd
        dgu = torch.cat([dact * u * (sg + g * sg * (1 - sg)), dact * g * sg], -1)
        gd[e * d:(e + 1) * d] = dy.T @ act
        ggu[e * 2 * f:(e + 1) * 2 * f] = dgu.T @ x
        dh.index_add_(0, tok, dgu @ wgu)
    return {"out": out, "dh": dh, "dwt": dwt, "ggu": ggu, "gd": gd}
