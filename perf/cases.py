"""What the framework is timed on: the work of its Llama-style decoder, from the smallest calls to the largest.

Four paths, each through the entry points a user's program calls:

* ``train``    one optimizer step of `SOTATrainer.train_step` on a host batch (copy, forward, loss, backward, clip, AdamW);
* ``serve``    requests through `EngineCore.execute`: prompts in chunks of the engine's token budget, then one token per
  request and step, batched continuously (a request decodes while another's prompt is still being read);
* ``fp8``      forward and backward of one projection of a layer that trains in fp8 (`ops.fp8.fp8_linear`);
* ``experts``  forward and backward of the routed feed-forward of the mixture models (`ops.moe.moe_ffn`).

Shapes are the presets of `models/llama.py` with fewer layers and, in the same proportion, a smaller vocabulary, so that a
step spends its time where the whole model's does.  Weights and tokens are random; lengths follow from the case alone.
"""
from __future__ import annotations

import math
import random

import torch
from torch.utils.checkpoint import checkpoint

from trainscale_b200.config.sota_config import SOTAConfig
from trainscale_b200.data.packing import cu_seqlens_from_document_ids
from trainscale_b200.inference.batch import StepEntry
from trainscale_b200.inference.engine import EngineConfig, EngineCore
from trainscale_b200.models.llama import build_model, preset_config
from trainscale_b200.ops.fp8 import fp8_linear
from trainscale_b200.ops.moe import moe_ffn
from trainscale_b200.trainer.sota_trainer import SOTATrainer

DEVICE = "cuda"
BLOCK = 16                      # tokens of a cache block
FP8_WEIGHTS = ("self_attn.wqkv", "self_attn.wo", "mlp.w_gate_up", "mlp.w_down")
LR, DECAY, BETAS, EPS, CLIP = 2e-5, 0.01, (0.9, 0.999), 1e-8, 1.0


def listed() -> list[dict]:
    return [
        # the tiny decoder of configs/llama_tiny_cpu_ddp.yaml on a GPU: packed documents, launches and latency count
        _train("train_tiny_packed", "tiny", 4, 32000, 8, 512, packed=True),
        # an ordinary fine-tuning batch of a small model: three sequences of an odd length, 64-wide heads, tied head
        _train("train_1b_odd", "llama3-1b", 4, 32064, 3, 1001),
        # the headline benchmark (Llama-3-8B, sequence 8192, operator-level recompute), an eighth of its depth and vocabulary
        _train("train_8b", "llama3-8b", 4, 16032, 1, 8192, recompute=True),
        # a long document: attention is half of the step
        _train("train_long", "llama3-8b", 2, 8016, 1, 32768, recompute=True),
        # the widest projection of configs/llama3_70b_tp4_pp2_fp8.yaml, one micro-batch
        _fp8("fp8_70b_gate_up", "llama3-70b", "mlp.w_gate_up", 4096),
        # the feed-forward of a mixture with few wide experts (Mixtral), and of one with many narrow ones
        _experts("experts_wide", 4096, 4096, 3584, 8, 2),
        _experts("experts_narrow", 3001, 2048, 1024, 64, 6),
        # one interactive request: nothing but latency
        _serve("serve_one", "llama3-1b", 16, 128256, 1, 97, 97, 32, 8192),
        # a dozen chats with short prompts: steps of few rows over the whole model
        _serve("serve_chat", "llama3-1b", 16, 128256, 12, 16, 64, 40, 8192),
        # a batch of requests with prompts of all lengths: chunked prompts beside decoding rows
        _serve("serve_batch", "llama3-1b", 16, 128256, 48, 64, 512, 24, 8192),
        # questions about long documents: prompts longer than the token budget, decoding over a long cache
        _serve("serve_long", "llama3-8b", 4, 16032, 3, 5000, 10000, 24, 8192),
    ]


def _train(name, model, layers, vocab, batch, seq, packed=False, recompute=False) -> dict:
    return {"name": name, "path": "train", "model": model, "layers": layers, "vocab": vocab, "batch": batch, "seq": seq,
            "packed": packed, "recompute": recompute}


def _fp8(name, model, weight, tokens) -> dict:
    return {"name": name, "path": "fp8", "model": model, "layers": 1, "vocab": 1000, "weight": weight, "tokens": tokens}


def _experts(name, tokens, hidden, ff, experts, top) -> dict:
    return {"name": name, "path": "experts", "tokens": tokens, "hidden": hidden, "ff": ff, "experts": experts, "top": top}


def _serve(name, model, layers, vocab, requests, shortest, longest, new, budget) -> dict:
    return {"name": name, "path": "serve", "model": model, "layers": layers, "vocab": vocab, "requests": requests,
            "shortest": shortest, "longest": longest, "new": new, "budget": budget}


def _spread(rng: random.Random, low: int, high: int) -> int:
    """An integer of [low, high], evenly over its logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng: random.Random) -> dict:
    most = max(_weight(c) for c in listed())
    while True:
        case = _drawn(rng)
        del case["name"]
        if _weight(case) <= most:
            return case


def _drawn(rng: random.Random) -> dict:
    path = rng.choices(("train", "fp8", "experts", "serve"), (4, 1, 2, 4))[0]
    if path == "train":
        model, most = rng.choice((("tiny", 4), ("llama3-1b", 4), ("llama3-8b", 3), ("mistral-7b", 2), ("llama3-70b", 1)))
        batch = rng.choice((1, 1, 2, 3, 4, 8))
        seq = _spread(rng, 100, 32768 if model in ("llama3-8b", "mistral-7b") else 8192)
        if rng.random() < 0.5:
            seq = -(-seq // 256) * 256
        return _train("", model, rng.randint(1, most), 8 * _spread(rng, 500, 4008), batch, seq, rng.random() < 0.35,
                      rng.random() < 0.4)
    if path == "fp8":
        tokens = _spread(rng, 200, 8192)
        return _fp8("", rng.choice(("llama3-1b", "llama3-8b", "llama3-70b")), rng.choice(FP8_WEIGHTS),
                    tokens if rng.random() < 0.25 else -(-tokens // 16) * 16)
    if path == "experts":
        experts, top = rng.choice(((4, 2), (8, 2), (16, 2), (32, 4), (64, 6)))
        return _experts("", _spread(rng, 64, 8192), rng.choice((512, 1024, 2048, 4096)), 128 * rng.randint(2, 28), experts, top)
    model, layers, vocab = rng.choice((("tiny", 4, 32000), ("llama3-1b", 16, 128256), ("llama3-8b", 4, 16032)))
    requests = _spread(rng, 1, 64)
    shortest = _spread(rng, 8, 2048)
    longest = min(12000, max(shortest, _spread(rng, 8, 24000 // requests + 8)))
    return _serve("", model, layers, vocab, requests, min(shortest, longest), longest, rng.randint(4, 40),
                  rng.choice((2048, 8192, 8192)))


# ------------------------------------------------------------------------------------------------ shapes and lengths
def _config(case: dict):
    return preset_config(case["model"], num_hidden_layers=case["layers"], vocab_size=case["vocab"])


def _rng(case: dict) -> random.Random:
    return random.Random(repr(sorted((k, v) for k, v in case.items() if k != "name")))


def _documents(case: dict) -> list[list[int]]:
    """Document lengths in every sequence of a training batch."""
    rng, rows = _rng(case), []
    for _ in range(case["batch"]):
        row = [] if case["packed"] else [case["seq"]]
        while sum(row) < case["seq"]:
            row.append(min(rng.randint(64, 512), case["seq"] - sum(row)))
        rows.append(row)
    return rows


def _prompts(case: dict) -> list[int]:
    rng = _rng(case)
    return [_spread(rng, case["shortest"], case["longest"]) for _ in range(case["requests"])]


def _schedule(case: dict) -> list[list[tuple[int, int, int]]]:
    """Steps of (request, first position, tokens): rows that decode first, then prompts up to the token budget."""
    prompts = _prompts(case)
    done, steps = [0] * len(prompts), []
    while True:
        step, left = [], case["budget"]
        for r, n in enumerate(prompts):
            if n <= done[r] < n + case["new"]:
                step.append((r, done[r], 1))
                left -= 1
        for r, n in enumerate(prompts):
            if done[r] < n and left > 0:
                take = min(n - done[r], left)
                step.append((r, done[r], take))
                left -= take
        if not step:
            return steps
        for r, _, n in step:
            done[r] += n
        steps.append(step)


def _shapes(case: dict) -> dict[str, tuple[int, ...]]:
    c = _config(case)
    H, I, D, q, kv = c.hidden_size, c.intermediate_size, c.head_dim, c.num_attention_heads, c.num_key_value_heads
    out = {"model.embed_tokens.weight": (c.vocab_size, H)}
    for i in range(c.num_hidden_layers):
        p = f"model.layers.{i}."
        out[p + "input_layernorm.weight"] = (H,)
        out[p + "self_attn.wqkv"] = ((q + 2 * kv) * D, H)
        out[p + "self_attn.wo"] = (H, q * D)
        out[p + "post_attention_layernorm.weight"] = (H,)
        out[p + "mlp.w_gate_up"] = (2 * I, H)
        out[p + "mlp.w_down"] = (H, I)
    out["model.norm.weight"] = (H,)
    if not c.tie_word_embeddings:
        out["lm_head"] = (c.vocab_size, H)
    return out


def _generator(seed: int, device: str = DEVICE) -> torch.Generator:
    return torch.Generator(device=device).manual_seed(seed)


def _weights(case: dict, seed: int) -> dict[str, torch.Tensor]:
    """bf16 weights by parameter name: every product keeps the size of its inputs, those that feed the residual stream are
    scaled down by the depth."""
    g, out = _generator(seed), {}
    std = 0.9 / math.sqrt(_config(case).hidden_size)
    for name, shape in _shapes(case).items():
        w = torch.empty(shape, dtype=torch.float32 if len(shape) == 1 else torch.bfloat16, device=DEVICE)
        if len(shape) == 1:
            out[name] = w.normal_(1.0, 0.1, generator=g).bfloat16()
        else:
            out[name] = w.normal_(0.0, std / math.sqrt(2 * case["layers"]) if name.endswith(("wo", "w_down")) else std, generator=g)
    return out


def _tokens(case: dict, seed: int, count: int) -> torch.Tensor:
    return torch.randint(0, case["vocab"], (count,), generator=_generator(seed + 1, "cpu"))


# ------------------------------------------------------------------------------------------------ prepare and run
def prepare(case: dict, seed: int):
    make = {"train": _prepare_train, "serve": _prepare_serve, "fp8": _prepare_fp8, "experts": _prepare_experts}
    return make[case["path"]](case, seed)


def run(state):
    return state["run"](state)


def _model(case: dict, seed: int):
    model = build_model(_config(case), dtype=torch.bfloat16, device=DEVICE)
    model.load_state_dict(_weights(case, seed))
    return model


def _batch(case: dict, seed: int) -> dict[str, torch.Tensor]:
    """A host batch as the collate function of the data pipeline gives it."""
    B, S = case["batch"], case["seq"]
    ids = _tokens(case, seed, B * S).view(B, S)
    batch = {"input_ids": ids, "attention_mask": torch.ones_like(ids), "labels": ids.clone()}
    if case["packed"]:
        rows = _documents(case)
        batch["document_ids"] = torch.stack([torch.repeat_interleave(torch.arange(len(r)), torch.tensor(r)) for r in rows])
        batch["position_ids"] = torch.stack([torch.cat([torch.arange(n) for n in r]) for r in rows])
        batch["cu_seqlens"], batch["max_seqlen"] = cu_seqlens_from_document_ids(batch["document_ids"])
    return {k: v.pin_memory() if torch.is_tensor(v) else v for k, v in batch.items()}


def _prepare_train(case: dict, seed: int):
    trainer = SOTATrainer(SOTAConfig.from_dict({
        "training_mode": "full",
        "optimizer": {"type": "adamw", "learning_rate": LR, "weight_decay": DECAY, "betas": list(BETAS), "eps": EPS,
                      "max_grad_norm": CLIP},
        "scheduler": {"type": "constant", "warmup_steps": 0, "warmup_ratio": 0.0},
        "loss": {"type": "chunked_ce"},
        "distributed": {"enabled": False, "strategy": "fsdp2", "gradient_checkpointing": False,
                        "fsdp_config": {"activation_checkpointing": False,
                                        "ac_mode": "op_selective" if case["recompute"] else "none"}},
        "hardware": {"precision": "bf16"},
        "data": {"max_seq_length": case["seq"]},
        "training": {"per_device_train_batch_size": case["batch"], "gradient_accumulation_steps": 1, "max_steps": 10 ** 6,
                     "logging_steps": 10 ** 9, "save_strategy": "no", "save_steps": 0, "eval_strategy": "no",
                     "early_stopping_patience": 0, "output_dir": "/tmp/trainscale_cases"},
    }))
    trainer.setup_model(model=_model(case, seed))
    trainer.setup_optimizer()
    trainer.setup_scheduler(10 ** 6)
    return {"run": _run_train, "trainer": trainer, "batch": _batch(case, seed)}


def _run_train(state):
    loss = state["trainer"].train_step(state["batch"])
    named = list(state["trainer"].model.named_parameters())
    return {"loss": loss, "grads": {n: p.main_grad for n, p in named}, "weights": {n: p.detach() for n, p in named}}


def _prepare_serve(case: dict, seed: int):
    prompts, new = _prompts(case), case["new"]
    config = EngineConfig(model=case["model"], device=DEVICE, enforce_eager=False)
    config.scheduler.max_num_seqs = max(64, case["requests"])
    config.scheduler.max_num_batched_tokens = case["budget"]
    config.cache.block_size = BLOCK
    config.cache.num_gpu_blocks = sum(-(-(n + new) // BLOCK) for n in prompts) + 64
    config.cache.max_model_len = max(prompts) + new
    core = EngineCore(config, model=_model(case, seed))
    ids = [t.tolist() for t in _tokens(case, seed, sum(prompts) + new * len(prompts)).split([n + new for n in prompts])]
    steps = [[StepEntry(r, ids[r][a:a + n], None if a + n >= prompts[r] else []) for r, a, n in step] for step in _schedule(case)]
    return {"run": _run_serve, "core": core, "steps": steps, "requests": len(prompts)}


def _run_serve(state):
    core, out = state["core"], []
    for entries in state["steps"]:
        logits = core.execute(entries)
        if logits is not None:
            out.append(logits.clone())        # a captured step's result is overwritten by the next
    for r in range(state["requests"]):
        core.release(r)
    return out


def _normal(g: torch.Generator, *shape: int, std: float = 1.0) -> torch.Tensor:
    return torch.empty(shape, dtype=torch.bfloat16, device=DEVICE).normal_(0.0, std, generator=g)


def _prepare_fp8(case: dict, seed: int):
    (N, K), T, g = _shapes(case)["model.layers.0." + case["weight"]], case["tokens"], _generator(seed)
    # a few features are ten times the others, as they are behind a norm
    x = _normal(g, T, K) * (1 + 9 * (torch.rand(K, generator=g, device=DEVICE) < 0.01).bfloat16())
    return {"run": _run_fp8, "x": x.requires_grad_(), "w": _normal(g, N, K, std=0.9 / math.sqrt(K)).requires_grad_(),
            "dy": _normal(g, T, N)}


def _run_fp8(s):
    y = fp8_linear(s["x"], s["w"], recipe="rowwise")
    return [y.detach(), *torch.autograd.grad(y, (s["x"], s["w"]), s["dy"])]


def _prepare_experts(case: dict, seed: int):
    T, H, I, E, k = (case[n] for n in ("tokens", "hidden", "ff", "experts", "top"))
    g = _generator(seed)
    # a router's choice: some experts are liked more than others
    scores = torch.randn(T, E, generator=g, device=DEVICE) + 0.5 * torch.randn(E, generator=g, device=DEVICE)
    top = torch.softmax(scores, -1).topk(k, dim=-1)
    return {"run": _run_experts, "x": _normal(g, T, H).requires_grad_(), "ids": top.indices,
            "weights": (top.values / top.values.sum(-1, keepdim=True)).requires_grad_(),
            "gate_up": _normal(g, E, 2 * I, H, std=0.02).requires_grad_(), "down": _normal(g, E, H, I, std=0.02).requires_grad_(),
            "dy": _normal(g, T, H)}


def _run_experts(s):
    y = moe_ffn(s["x"], s["ids"], s["weights"].to(s["x"].dtype), s["gate_up"], s["down"])
    return [y.detach(), *torch.autograd.grad(y, (s["x"], s["weights"], s["gate_up"], s["down"]), s["dy"])]


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _weight(case: dict) -> float:
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def _pairs(start: int, n: int, window: int | None = None) -> int:
    """Visible (query, key) pairs of n causal rows from position `start`."""
    full = n * start + n * (n + 1) // 2
    if not window or start + n <= window:
        return full
    return sum(min(window, start + i + 1) for i in range(n))


def work(case: dict) -> dict:
    if case["path"] == "fp8":
        (N, K), T = _shapes(case)["model.layers.0." + case["weight"]], case["tokens"]
        return {"bytes": 2 * (2 * T * K + 2 * T * N + 2 * N * K), "flops": 6 * T * N * K}
    if case["path"] == "experts":
        T, H, I, E, k = (case[n] for n in ("tokens", "hidden", "ff", "experts", "top"))
        used = min(E, T * k)
        # x, dy, y, dx, routing; the weights of the experts used, the gradients of all
        return {"bytes": 4 * T * H * 2 + 3 * T * k * 8 + (used + E) * 3 * H * I * 2, "flops": 3 * 2 * T * k * 3 * H * I}
    c = _config(case)
    layer = sum(math.prod(s) for n, s in _shapes(case).items() if len(s) == 2 and ".layers." in n)
    head = c.vocab_size * c.hidden_size
    q, kv = c.num_attention_heads * c.head_dim, c.num_key_value_heads * c.head_dim
    if case["path"] == "train":
        T = case["batch"] * case["seq"]
        pairs = sum(_pairs(0, n, c.sliding_window) for row in _documents(case) for n in row)
        params = sum(math.prod(s) for s in _shapes(case).values())
        # bf16 weight, fp32 master weight and moments in; the same and the gradient out
        return {"bytes": params * (2 + 12 + 14 + 2) + 3 * 8 * T, "flops": 6 * T * (layer + head) + 12 * c.num_hidden_layers * q * pairs}
    flops = size = 0
    for step in _schedule(case):
        rows = sum(n for _, _, n in step)
        wanted = sum(a + n >= p for (r, a, n) in step for p in (_prompts(case)[r],))
        flops += 2 * rows * layer + 2 * wanted * head + 4 * c.num_hidden_layers * q * sum(_pairs(a, n) for _, a, n in step)
        # weights once a step, keys and values of every request read once, those of the new tokens written, logits
        size += 2 * (layer + (head if wanted else 0)) + 4 * wanted * c.vocab_size
        size += 2 * 2 * kv * c.num_hidden_layers * (sum(a for _, a, _ in step) + rows)
    return {"bytes": size, "flops": flops}


def tolerance(case: dict) -> dict:
    """Four times what a pass with its sums in another order was seen to differ by, at most what the types leave: 16 layers in
    bf16 are 2.5e-2 from the same in 64 bits, a layer's forward and backward 1.5e-2, one product 4e-3."""
    if case["path"] in ("experts", "fp8"):
        return {"rel": 0.01, "max": 0.3}
    return {"rel": 0.03, "max": 0.9}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def exact(case: dict, seed: int):
    make = {"train": _exact_train, "serve": _exact_serve, "fp8": _exact_fp8, "experts": _exact_experts}
    return make[case["path"]](case, seed)


def _norm64(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _attention64(q, k, v, window):
    """Causal rows of one sequence and one key head: q [heads, n, D], k and v [n, D]; a strip of rows at a time."""
    def strip(qs, ks, vs, a):
        s = qs @ ks.t() / math.sqrt(qs.shape[-1])
        i = torch.arange(a, a + qs.shape[1], device=qs.device).unsqueeze(1)
        j = torch.arange(ks.shape[0], device=qs.device)
        hidden = (j > i) if not window else (j > i) | (j <= i - window)
        return torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ vs

    rows, out = max(64, min(2048, (1 << 27) // (q.shape[0] * k.shape[0]))), []
    for a in range(0, k.shape[0], rows):
        b = min(a + rows, k.shape[0])
        out.append(checkpoint(strip, q[:, a:b], k[:b], v[:b], a, use_reentrant=False))
    return torch.cat(out, 1)


def _decoder64(c, w, ids, positions, spans):
    """Final hidden states of tokens [T] at `positions`; `spans`: consecutive runs that attend within themselves."""
    q, kv, D = c.num_attention_heads, c.num_key_value_heads, c.head_dim
    angle = positions.double().unsqueeze(1) * c.rope_theta ** (-torch.arange(0, D, 2, device=ids.device).double() / D)
    cos, sin = angle.cos().unsqueeze(1), angle.sin().unsqueeze(1)

    def layer(x, p):
        y = _norm64(x, w[p + "input_layernorm.weight"], c.rms_norm_eps) @ w[p + "self_attn.wqkv"].t()
        y = y.view(len(ids), q + 2 * kv, D)
        a, b = y[:, :q + kv].chunk(2, -1)
        heads = torch.cat([a * cos - b * sin, b * cos + a * sin], -1)
        out = []
        for i, j in spans:
            out.append(torch.cat([_attention64(heads[i:j, h * (q // kv):(h + 1) * (q // kv)].transpose(0, 1), heads[i:j, q + h],
                                               y[i:j, q + kv + h], c.sliding_window) for h in range(kv)]).transpose(0, 1))
        x = x + torch.cat(out).reshape(len(ids), q * D) @ w[p + "self_attn.wo"].t()
        y = _norm64(x, w[p + "post_attention_layernorm.weight"], c.rms_norm_eps) @ w[p + "mlp.w_gate_up"].t()
        gate, up = y.chunk(2, -1)
        return x + (torch.nn.functional.silu(gate) * up) @ w[p + "mlp.w_down"].t()

    x = w["model.embed_tokens.weight"][ids]
    for i in range(c.num_hidden_layers):
        x = checkpoint(layer, x, f"model.layers.{i}.", use_reentrant=False)
    return _norm64(x, w["model.norm.weight"], c.rms_norm_eps)


def _spans(lengths: list[int]) -> list[tuple[int, int]]:
    out, at = [], 0
    for n in lengths:
        out.append((at, at + n))
        at += n
    return out


def _exact_train(case: dict, seed: int):
    c = _config(case)
    w = {n: t.double().requires_grad_() for n, t in _weights(case, seed).items()}
    ids = _tokens(case, seed, case["batch"] * case["seq"]).to(DEVICE)
    lengths = [n for row in _documents(case) for n in row]
    positions = torch.cat([torch.arange(n, device=DEVICE) for n in lengths])
    x = _decoder64(c, w, ids, positions, _spans(lengths))
    known = torch.cat([torch.arange(a, b - 1, device=DEVICE) for a, b in _spans(lengths)])     # rows with a next token
    head = w["lm_head" if "lm_head" in w else "model.embed_tokens.weight"]

    def part(xs, target):
        return torch.nn.functional.cross_entropy(xs @ head.t(), target, reduction="sum")

    loss = sum(checkpoint(part, x[r], ids[r + 1], use_reentrant=False) for r in known.split(4096)) / len(known)
    grads = dict(zip(w, torch.autograd.grad(loss, list(w.values()))))
    norm = math.sqrt(sum(float(g.pow(2).sum()) for g in grads.values()))
    clip = min(1.0, CLIP / (norm + 1e-6))
    updated = {}
    with torch.no_grad():
        for n, p in w.items():
            g = grads[n] * clip
            m, v = g * (1 - BETAS[0]) / (1 - BETAS[0]), g.pow(2) * (1 - BETAS[1]) / (1 - BETAS[1])
            updated[n] = p * (1 - LR * DECAY) - LR * m / (v.sqrt() + EPS)
    return {"loss": float(loss), "grads": grads, "weights": updated}


@torch.no_grad()
def _exact_serve(case: dict, seed: int):
    c, prompts, new = _config(case), _prompts(case), case["new"]
    w = {n: t.double() for n, t in _weights(case, seed).items()}
    lengths = [n + new for n in prompts]
    ids = _tokens(case, seed, sum(lengths)).to(DEVICE)
    positions = torch.cat([torch.arange(n, device=DEVICE) for n in lengths])
    spans, out = _spans(lengths), []
    x = _decoder64(c, w, ids, positions, spans)
    head = w["lm_head" if "lm_head" in w else "model.embed_tokens.weight"]
    for step in _schedule(case):
        rows = [spans[r][0] + a + n - 1 for r, a, n in step if a + n >= prompts[r]]
        if rows:
            out.append((x[rows] @ head.t()).float())
    return out


def _exact_fp8(case: dict, seed: int):
    """The product itself: what fp8 takes from it is part of the difference."""
    s = _prepare_fp8(case, seed)
    x, w, dy = (s[n].detach().double() for n in ("x", "w", "dy"))
    return [x @ w.t(), dy @ w, dy.t() @ x]


def _exact_experts(case: dict, seed: int):
    s = _prepare_experts(case, seed)
    x, weights, gate_up, down = (s[n].detach().double().requires_grad_() for n in ("x", "weights", "gate_up", "down"))
    y = torch.zeros_like(x)
    for e in range(case["experts"]):
        token, slot = (s["ids"] == e).nonzero(as_tuple=True)
        gate, up = (x[token] @ gate_up[e].t()).chunk(2, -1)
        y = y.index_add(0, token, (torch.nn.functional.silu(gate) * up) @ down[e].t() * weights[token, slot].unsqueeze(1))
    return [y.detach(), *torch.autograd.grad(y, (x, weights, gate_up, down), s["dy"].double())]
