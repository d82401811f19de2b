"""What the framework is timed on: training steps, evaluation, the autograd module and generation.

Each case is one call (or one short loop a user's program would write) through the public entry
points: `GPT2TrainEngine.train_step` / `eval_losses`, `GPT2.forward` / `generate`, `GPTLM.forward`.
Shapes are those of the presets in `zero_to_hero_b200.config`, of the tests and of `bench.py`, plus
ragged sizes between them. `draw` samples the same ranges.
"""
from __future__ import annotations

import math

import torch

from zero_to_hero_b200.config import get_preset
from zero_to_hero_b200.engine import GPT2TrainEngine
from zero_to_hero_b200.models.gpt import GPTLM
from zero_to_hero_b200.models.gpt2 import GPT2

REAL_VOCAB = 50257  # tokens are drawn below this; 50304 is the same vocabulary padded


def _case(name, kind, layers, heads, vocab, block, batch, **more):
    c = {"kind": kind, "layers": layers, "heads": heads, "vocab": vocab, "block": block, "batch": batch}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The smallest training step: the tiny preset of the smoke run (2 layers, 128 wide, 4 x 128
        # tokens, two micro-steps). Host work and launches are all there is.
        _case("train-tiny", "train", 2, 2, 512, 128, 4, accum=2, dropout=0.0, reproducible=False),
        # The benchmark's model and micro-batch, 16 x 1024 tokens; two of its 32 micro-steps and the
        # optimizer step, so that one pass stays short.
        _case("train-124m", "train", 12, 12, 50304, 1024, 16, accum=2, dropout=0.0, reproducible=False),
        # The 350M preset with its micro-batch of 8 x 1024: the largest case.
        _case("train-350m", "train", 24, 16, 50304, 1024, 8, accum=2, dropout=0.0, reproducible=False),
        # Training with dropout 0.2 at all four sites, as the GPT-2 trainer this framework follows does.
        _case("train-124m-dropout", "train", 12, 12, 50304, 1024, 8, accum=1, dropout=0.2, reproducible=False),
        # Ragged: odd batch and context, unpadded vocabulary, the bitwise reproducible mode.
        _case("train-ragged-reproducible", "train", 6, 6, 50257, 509, 5, accum=2, dropout=0.0, reproducible=True),
        # Validation loss of the trainer: forward only over one micro-batch.
        _case("eval-124m", "eval", 12, 12, 50304, 1024, 16, length=1024),
        # One HellaSwag example: four endings padded to 256 tokens, through the same forward pass.
        _case("eval-124m-4x256", "eval", 12, 12, 50304, 1024, 16, rows=4, length=256),
        # A program that keeps its own training loop: nn.Module forward and loss.backward().
        _case("module-124m", "module", 12, 12, 50304, 1024, 8, length=1024, ln_bias=False),
        # The same with a GPT-2 checkpoint's own vocabulary, LayerNorm biases and an odd length.
        _case("module-ragged", "module", 12, 12, 50257, 1024, 3, length=777, ln_bias=True),
        # The character-level model at its preset: 6 layers, 384 wide, 64 x 256 tokens, 65 characters.
        _case("char", "char", 6, 6, 65, 256, 64, length=256),
        # The sampling command's defaults: one sequence from a single token, 64 new ones.
        _case("generate-124m", "generate", 12, 12, 50257, 1024, 1, prompt=1, new=64),
        # Generation with the 1.5B model for a few prompts of odd length: prefill counts as well.
        _case("generate-1.5b", "generate", 48, 25, 50304, 1024, 4, prompt=203, new=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("train", "train", "train", "eval", "module", "char", "generate", "generate"))
    limit = max(work(c)["flops"] for c in listed())
    while True:
        if kind == "char":
            c = _case(None, kind, rng.randint(1, 8), rng.randint(2, 8), rng.randint(27, 128),
                      _log_int(rng, 32, 512), _log_int(rng, 1, 96))
            c["length"] = rng.randint(c["block"] // 2, c["block"])
        else:
            heads = rng.choice((4, 6, 8, 12, 12, 16, 20, 25))
            c = _case(None, kind, _log_int(rng, 2, 24), heads, rng.choice((512, 1000, 50257, 50304)),
                      _log_int(rng, 64, 1024), _log_int(rng, 1, 16))
            block = c["block"]
            if kind == "train":
                c.update(accum=rng.randint(1, 3), dropout=rng.choice((0.0, 0.0, 0.1, 0.2)),
                         reproducible=rng.random() < 0.25)
            elif kind == "eval":
                c.update(rows=rng.randint(1, c["batch"]), length=rng.randint(block // 2, block))
            elif kind == "module":
                c.update(length=rng.randint(block // 2, block), ln_bias=rng.random() < 0.5)
            else:
                c.update(prompt=_log_int(rng, 1, block), new=_log_int(rng, 4, 64))
                c["batch"] = _log_int(rng, 1, 8)
        if work(c)["flops"] <= limit:
            return c


def _config(case):
    cfg = get_preset("gpt2-124m")
    mc, tc = cfg.model, cfg.train
    mc.num_layers, mc.num_heads, mc.emb_dim = case["layers"], case["heads"], 64 * case["heads"]
    mc.vocab_size, mc.block_size = case["vocab"], case["block"]
    mc.dropout = case.get("dropout", 0.0)
    mc.ln_bias = case.get("ln_bias", False)
    tc.micro_batch = case["batch"]
    tc.deterministic = case.get("reproducible", False)
    tc.total_batch_tokens = case["batch"] * case["block"] * case.get("accum", 1)
    return cfg


def _tokens(case, rows, length, gen):
    """A batch as the loaders cut it: Y is X shifted by one."""
    high = min(case["vocab"], REAL_VOCAB)
    t = torch.randint(0, high, (rows * length + 1,), generator=gen, dtype=torch.int64)
    return t[:-1].view(rows, length).contiguous(), t[1:].view(rows, length).contiguous()


def prepare(case, seed):
    kind, gen = case["kind"], torch.Generator().manual_seed(seed)
    if kind in ("train", "eval"):
        # the trainer's handle: weights, moments, activations; batches in pinned host memory
        engine = GPT2TrainEngine(_config(case), "cuda", seed=seed)
        rows, length = (case["batch"], case["block"]) if kind == "train" else \
            (case.get("rows", case["batch"]), case["length"])
        batches = [tuple(t.pin_memory() for t in _tokens(case, rows, length, gen))
                   for _ in range(case.get("accum", 1))]
        return {"kind": kind, "engine": engine, "batches": batches}
    torch.manual_seed(seed)
    with torch.device("cuda"):
        if kind == "char":
            model = GPTLM(case["vocab"], case["block"], 64 * case["heads"], case["layers"], case["heads"], 0.0)
        else:
            model = GPT2(_config(case).model)
    if kind == "generate":
        # Token embeddings at the scale of trained GPT-2 weights (std 0.14): the next token is then
        # predicted with confidence, as a trained model does, and greedy decoding does not turn on
        # rounding errors.
        with torch.no_grad():
            model.transformer.wte.weight.normal_(0.0, 0.14)
        X, _ = _tokens(case, case["batch"], case["prompt"], gen)
        return {"kind": kind, "model": model.eval(), "X": X.cuda(), "new": case["new"]}
    X, Y = _tokens(case, case["batch"], case["length"], gen)
    return {"kind": kind, "model": model, "X": X.cuda(), "Y": Y.cuda()}


def run(state):
    kind = state["kind"]
    if kind == "train":
        # one optimizer step and the read of its loss, as the trainer logs it
        eng = state["engine"]
        eng.train_step(state["batches"])
        loss = eng.read_loss()
        k = eng.layout.n_decay  # matrices and embeddings first, then biases and LayerNorm weights
        return {"loss": loss, "grad_norm": eng.norm,
                "matrices": {"weights": eng.p32[:k], "m": eng.m[:k], "v": eng.v[:k]},
                "vectors": {"weights": eng.p32[k:], "m": eng.m[k:], "v": eng.v[k:]}}
    if kind == "eval":
        return state["engine"].eval_losses(*state["batches"][0])
    model, X = state["model"], state["X"]
    if kind == "generate":
        tokens = model.generate(X, state["new"], temperature=1.0, top_k=1)
        with torch.inference_mode():
            logits, _ = model(tokens[:, -model.config.block_size:])
        return {"tokens": tokens, "logits": logits}
    model.zero_grad(set_to_none=True)
    logits, loss = model(X, state["Y"])
    loss.backward()
    flat = torch.nn.utils.parameters_to_vector  # one tensor for each of AdamW's two groups
    return {"logits": logits.detach(), "loss": loss.detach(),
            "matrix_grads": flat(p.grad for p in model.parameters() if p.dim() >= 2),
            "vector_grads": flat(p.grad for p in model.parameters() if p.dim() < 2)}


def _counts(case):
    """(parameters, weights that take part in matrix products per token)."""
    C, L, V = 64 * case["heads"], case["layers"], case["vocab"]
    dense = 12 * C * C * L + V * C
    return dense + (13 * L + 2) * C + case["block"] * C + (V * C if case["kind"] == "char" else 0), dense


def work(case):
    """Model arithmetic (2 operations per weight and token forward, 4 more backward, causal attention
    at half the square) and the bytes of parameters, their state and results, each once; decoding
    reads the bf16 weights once per new token."""
    kind = case["kind"]
    params, dense = _counts(case)
    C, L, V, B = 64 * case["heads"], case["layers"], case["vocab"], case["batch"]
    if kind == "generate":
        T, block = case["prompt"] + case["new"], case["block"]
        body = dense - V * C  # the head is needed at one position per new token
        flops = 2.0 * B * (min(T, block) * body + (case["new"] + 1) * V * C) + 2.0 * B * min(T, block) ** 2 * C * L
        return {"bytes": 4.0 * params + 2.0 * dense * case["new"], "flops": flops}
    if kind == "train":
        T, passes = case["block"], case["accum"]
    else:
        T, passes = case["length"], 1
    B = case.get("rows", B)
    forward = 2.0 * dense * B * T + 2.0 * B * T * T * C * L
    attention_extra = 1.0 * B * T * T * C * L  # the backward recomputes the scores
    if kind == "eval":
        return {"bytes": 2.0 * params + 20.0 * B * T, "flops": forward}
    flops = passes * (3.0 * forward + attention_extra)
    if kind == "train":
        return {"bytes": 26.0 * params + 16.0 * passes * B * T, "flops": flops}
    return {"bytes": 8.0 * params + 2.0 * B * T * V, "flops": flops}


def tolerance(case):
    """Against the same network in fp64 (same weights, random tokens) the bf16 paths differ, as the
    norm of the difference over the norm: logits 0.7-1.7e-2, gradients and AdamW moments 0.6-1.9e-2 (largest
    single value 0.6 of the rms), mean loss 5e-6, losses per token 5e-4 (largest 2e-3). Two correct bf16
    implementations may be sqrt(2) of that apart."""
    if case["kind"] == "eval":
        return {"rel": 0.002, "max": 0.01}
    return {"rel": 0.03, "max": 0.9}


# ---------------------------------------------------------------------------------------------
# the same results in 64 bits, in plain torch
# ---------------------------------------------------------------------------------------------
def _norm64(x, w, b):
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), w, b, 1e-5)


def _attention64(q, k, v, heads):
    T, C = q.shape
    q, k, v = (t.view(T, heads, C // heads).transpose(0, 1) for t in (q, k, v))
    scores = (q @ k.transpose(1, 2)) / math.sqrt(C // heads)
    scores = scores.masked_fill(torch.ones(T, T, dtype=torch.bool, device=q.device).triu(1), -math.inf)
    return (scores.softmax(-1) @ v).transpose(0, 1).reshape(T, C)


def _logits64(case, p, x):
    """Logits [T, V] of one sequence of tokens; `p` holds 64-bit parameters by name."""
    linear, heads = torch.nn.functional.linear, case["heads"]
    if case["kind"] == "char":
        h = p["tok_to_emb.weight"][x] + p["pos_to_emb.weight"][:len(x)]
        for i in range(case["layers"]):
            b = f"blocks.{i}."
            n = _norm64(h, p[b + "ln1.weight"], p[b + "ln1.bias"])
            q, k, v = (torch.cat([linear(n, p[f"{b}attn.heads.{j}.{which}.weight"]) for j in range(heads)], -1)
                       for which in ("query", "key", "value"))
            h = h + linear(_attention64(q, k, v, heads), p[b + "attn.proj.weight"], p[b + "attn.proj.bias"])
            n = _norm64(h, p[b + "ln2.weight"], p[b + "ln2.bias"])
            n = linear(n, p[b + "ff.ff.0.weight"], p[b + "ff.ff.0.bias"]).relu()
            h = h + linear(n, p[b + "ff.ff.3.weight"], p[b + "ff.ff.3.bias"])
        return linear(_norm64(h, p["ln.weight"], p["ln.bias"]), p["head.weight"], p["head.bias"])
    h = p["transformer.wte.weight"][x] + p["transformer.wpe.weight"][:len(x)]
    for i in range(case["layers"]):
        b = f"transformer.h.{i}."
        n = _norm64(h, p[b + "ln_1.weight"], p.get(b + "ln_1.bias"))
        q, k, v = linear(n, p[b + "attn.c_attn.weight"], p[b + "attn.c_attn.bias"]).chunk(3, -1)
        h = h + linear(_attention64(q, k, v, heads), p[b + "attn.c_proj.weight"], p[b + "attn.c_proj.bias"])
        n = _norm64(h, p[b + "ln_2.weight"], p.get(b + "ln_2.bias"))
        n = linear(n, p[b + "mlp.c_fc.weight"], p[b + "mlp.c_fc.bias"])
        n = torch.nn.functional.gelu(n, approximate="tanh")
        h = h + linear(n, p[b + "mlp.c_proj.weight"], p[b + "mlp.c_proj.bias"])
    h = _norm64(h, p["transformer.ln_f.weight"], p.get("transformer.ln_f.bias"))
    return linear(h, p["transformer.wte.weight"])


def exact(case, seed):
    kind = case["kind"]
    if kind == "generate" or case.get("dropout", 0.0) > 0.0 or work(case)["flops"] > 1.2e14:
        return None  # tokens of its own, a mask that is this framework's own, or too long in 64 bits
    state = prepare(case, seed)
    if kind in ("train", "eval"):
        eng = state["engine"]
        p = {n: v.double() for n, v in eng.state_dict().items() if n != "lm_head.weight"}
        batches = [(x.cuda(), y.cuda()) for x, y in state["batches"]]
    else:
        p = {n: v.detach().double() for n, v in state["model"].named_parameters()}
        batches = [(state["X"], state["Y"])]
    grad = kind != "eval"
    for v in p.values():
        v.requires_grad_(grad)
    tokens = sum(x.numel() for x, _ in batches)
    per_token, logits, loss = [], [], 0.0
    with torch.set_grad_enabled(grad):
        for X, Y in batches:
            for x, y in zip(X, Y):
                z = _logits64(case, p, x)
                ce = torch.nn.functional.cross_entropy(z, y, reduction="none")
                if grad:
                    (ce.sum() / tokens).backward()
                per_token.append(ce.detach())
                loss += ce.detach().sum() / tokens
                if kind in ("module", "char"):
                    logits.append(z.detach())
    if kind == "eval":
        return torch.stack(per_token)
    if kind != "train":
        flat = torch.nn.utils.parameters_to_vector
        return {"logits": torch.stack(logits), "loss": loss,
                "matrix_grads": flat(v.grad for v in p.values() if v.dim() >= 2),
                "vector_grads": flat(v.grad for v in p.values() if v.dim() < 2)}
    # first AdamW step, in the order of the engine's flat buffers (gaps between tensors stay 0)
    oc, k = eng.cfg.optim, eng.layout.n_decay
    norm = torch.sqrt(sum(v.grad.square().sum() for v in p.values()))
    clip = min(1.0, oc.clip_norm / (norm.item() + 1e-6))
    lr = oc.lr_max / oc.warmup_steps
    w, m, s = (torch.zeros(eng.layout.total, dtype=torch.float64, device="cuda") for _ in range(3))
    for name, spec in eng.layout.specs.items():
        at, v = slice(spec.offset, spec.offset + spec.numel), p[name]
        g = clip * v.grad.flatten()
        m[at], s[at] = (1 - oc.beta1) * g, (1 - oc.beta2) * g * g
        step = lr * g / (g.abs() + oc.eps)
        w[at] = v.detach().flatten() * (1 - lr * oc.weight_decay if spec.decay else 1.0) - step
    return {"loss": loss, "grad_norm": norm.reshape(1),
            "matrices": {"weights": w[:k], "m": m[:k], "v": s[:k]},
            "vectors": {"weights": w[k:], "m": m[k:], "v": s[k:]}}
