"""Cached-key/value decoding of a `models.gpt2.GPT2` (csrc/decode/decode.cu).

`DecodeSession` lives for one `generate` call: it packs the model's weights into one bf16 buffer, fills
the cache with a batched pass over the prompt and then runs one persistent kernel per new token. Nothing
outlives the call.
"""
from __future__ import annotations

import ctypes

import torch
import torch.nn as nn

from . import _lib, gemm as G, native as N

MAX_BATCH = 8            # sequences of one decode launch (the n of its tensor-core instruction)
# Sequences of a session, in groups of MAX_BATCH that each read all weights; more take the batched forward per
# token, whose time hardly depends on their number while the window is short. Session / forward, ms for 8 tokens,
# prompts of 8: 24 sequences 10.7 / 17.7 (124M) and 65 / 64 (1.5B), 32 14.0 / 17.7 and 85 / 64, 48 20.5 / 17.9 and
# 126 / 65; prompts of 256: 32 15.3 / 22.3 and 110 / 229, 48 22.5 / 26.4 and 162 / 325.
MAX_SEQUENCES = 32
# A prompt of up to this many tokens (before its last one) goes through the decode kernel one by one, a longer
# one through the batched pass, which is bound by its launches. Stepwise / batched, ms: 124M, one sequence, 4
# tokens 0.74 / 1.09, 6 tokens 1.11 / 1.08; eight sequences, 4 tokens 1.02 / 1.08; 1.5B, 4 tokens 4.4 / 5.0,
# 6 tokens 6.6 / 5.0.
STEPWISE_PROMPT = 4

_sigs = {
    "z2h_decode_scratch_bytes": ([ctypes.c_int] * 3, ctypes.c_longlong),
    "z2h_decode_epochs": ([ctypes.c_int] * 3, ctypes.c_uint),
    "z2h_decode_step": ([ctypes.c_void_p] * 4 + [ctypes.c_longlong] + [ctypes.c_void_p] * 2 + [ctypes.c_uint] +
                        [ctypes.c_int] * 7 + [ctypes.c_void_p] * 2, ctypes.c_int),
    "z2h_pack_bf16": ([ctypes.c_void_p] * 3 + [ctypes.c_int] * 2 + [ctypes.c_void_p] * 2, ctypes.c_int),
    "z2h_kv_from_qkv": ([ctypes.c_void_p] * 2 + [ctypes.c_int] * 4 + [ctypes.c_void_p], ctypes.c_int),
}
_fns: dict = {}


def _f(name: str):
    fn = _fns.get(name)
    if fn is None:
        fn = getattr(_lib.cuda_lib(), name)
        fn.argtypes, fn.restype = _sigs[name]
        _fns[name] = fn
    return fn


def _call(name: str, *args) -> None:
    rc = _f(name)(*args)
    if rc != 0:
        raise RuntimeError(f"{name} failed with code {rc} (1 bad argument, 3 launch)")


def packed_layout(cfg) -> tuple[dict[str, int], list[int], int]:
    """(element offset of every parameter, the 18 numbers of `DecodeLayout`, total elements)."""
    C, L, V, T, F = cfg.emb_dim, cfg.num_layers, cfg.vocab_size, cfg.block_size, 4 * cfg.emb_dim
    off: dict[str, int] = {}
    at = 0

    def put(name, n):
        nonlocal at
        off[name] = at
        at += (n + 63) // 64 * 64

    put("transformer.wte.weight", V * C)
    put("transformer.wpe.weight", T * C)
    parts = [("attn.c_attn.weight", 3 * C * C), ("attn.c_proj.weight", C * C), ("mlp.c_fc.weight", F * C),
             ("mlp.c_proj.weight", C * F), ("ln_1.weight", C), ("ln_1.bias", C), ("attn.c_attn.bias", 3 * C),
             ("attn.c_proj.bias", C), ("ln_2.weight", C), ("ln_2.bias", C), ("mlp.c_fc.bias", F), ("mlp.c_proj.bias", C)]
    layer0, inner = at, {}
    for i in range(L):
        start = at
        for name, n in parts:
            if cfg.ln_bias or name not in ("ln_1.bias", "ln_2.bias"):
                inner[name] = at - start
                put(f"transformer.h.{i}.{name}", n)
    stride = (at - layer0) // L if L else 0
    put("transformer.ln_f.weight", C)
    if cfg.ln_bias:
        put("transformer.ln_f.bias", C)
    o = off.get
    numbers = [off["transformer.wte.weight"], off["transformer.wpe.weight"], layer0, stride,
               off["transformer.ln_f.weight"], o("transformer.ln_f.bias", -1)] + [inner.get(n, -1) for n, _ in parts]
    return off, numbers, at


def _plain(module: nn.Module) -> bool:
    """Calling `module` runs its class's forward and nothing else."""
    return not (module._forward_hooks or module._forward_pre_hooks or "forward" in module.__dict__)


def plain_model(model) -> bool:
    """A GPT2 whose forward is that of this package's modules and nothing else: tied head, dropout off,
    no hooks, no replaced layers or parameters, contiguous fp32 or bf16 weights of one type and device."""
    from ..models import gpt2 as M
    from torch.nn.modules import module as nnm

    if type(model) is not M.GPT2 or nnm._global_forward_hooks or nnm._global_forward_pre_hooks:
        return False
    cfg = model.config
    known = (M.GPT2, M.Transformer, M.Block, M.Attention, M.MLP, M.LayerNorm, nn.Linear, nn.Embedding, nn.ModuleList)
    for m in model.modules():
        if type(m) not in known or not _plain(m):
            return False
        if type(m) is M.LayerNorm and m.eps != 1e-5:
            return False
        if type(m) is M.Attention and m.num_heads != cfg.num_heads:
            return False
        if type(m) is nn.Embedding and m.max_norm is not None:
            return False
        if m.training and (cfg.dropout > 0.0 or getattr(m, "dropout", 0.0) > 0.0):
            return False
    if model.lm_head.weight is not model.transformer.wte.weight:
        return False
    want, have = expected_shapes(cfg), dict(model.named_parameters())
    if set(have) != set(want):
        return False
    first = have["transformer.wte.weight"]
    return first.dtype in (torch.float32, torch.bfloat16) and all(
        type(p) is nn.Parameter and p.dtype == first.dtype and p.device == first.device and tuple(p.shape) == want[n]
        and p.is_contiguous() and p.data_ptr() % 16 == 0 for n, p in have.items())


def supports(model, X: torch.Tensor) -> bool:
    """Whether a decoding session computes what the module's own forward would, for this model and these
    prompts. Anything else (hooks, replaced layers, other types and shapes) keeps the general path."""
    cfg = model.config
    if type(X) is not torch.Tensor or not X.is_cuda or X.dim() != 2 or X.dtype not in (torch.int64, torch.int32):
        return False
    if not 1 <= X.shape[0] <= MAX_SEQUENCES or X.shape[1] < 1:
        return False
    if cfg.emb_dim != 64 * cfg.num_heads or cfg.emb_dim > 2048 or cfg.num_layers < 1:
        return False
    if torch.is_autocast_enabled() or torch.compiler.is_compiling() or X.device.index != torch.cuda.current_device():
        return False
    return plain_model(model) and model.lm_head.weight.device == X.device and \
        kernel_takes(X.shape[0], cfg.emb_dim, cfg.num_layers)


def group_sizes(batch: int) -> list[int]:
    """Sequences of the launches that a step of `batch` sequences takes."""
    return [min(MAX_BATCH, batch - b0) for b0 in range(0, batch, MAX_BATCH)]


def kernel_takes(batch: int, C: int, layers: int) -> bool:
    """The kernel's own rule, which depends on the device (2048 columns need 128 SMs)."""
    return all(_f("z2h_decode_epochs")(n, C, layers) != 0 for n in set(group_sizes(batch)))


def expected_shapes(cfg) -> dict[str, tuple[int, ...]]:
    from ..engine import ParamLayout

    return {n: tuple(s.shape) for n, s in ParamLayout(cfg).specs.items()}


class DecodeSession:
    """Weights, cache and scratch of one generation over `batch` sequences of at most `max_len` tokens."""

    def __init__(self, model, batch: int, max_len: int):
        cfg = self.cfg = model.config
        self.batch, self.max_len = batch, max_len
        self.C, self.H, self.L, self.V = cfg.emb_dim, cfg.num_heads, cfg.num_layers, cfg.vocab_size
        params = dict(model.named_parameters())
        self.device = params["transformer.wte.weight"].device
        self.offsets, numbers, total = packed_layout(cfg)
        self.numbers = (ctypes.c_longlong * len(numbers))(*numbers)
        self.w = torch.empty(total, device=self.device, dtype=torch.bfloat16)
        self._pack([(params[n], at) for n, at in self.offsets.items()])
        self.shapes = {n: tuple(p.shape) for n, p in params.items()}
        self.groups = []
        for i, n in enumerate(group_sizes(batch)):
            b0 = i * MAX_BATCH
            kv = torch.empty(self.L, 2, n, max_len, self.C, device=self.device, dtype=torch.bfloat16)
            scratch = torch.zeros(_f("z2h_decode_scratch_bytes")(n, self.C, self.H), device=self.device, dtype=torch.uint8)
            epochs = _f("z2h_decode_epochs")(n, self.C, self.L)
            self.groups.append({"rows": slice(b0, b0 + n), "n": n, "kv": kv, "scratch": scratch, "epochs": epochs, "base": 1})
        self.logits = torch.empty(batch, self.V, device=self.device, dtype=torch.float32)

    def _pack(self, tensors) -> None:
        n = len(tensors)
        src = (ctypes.c_void_p * n)(*[t.data_ptr() for t, _ in tensors])
        dst = (ctypes.c_longlong * n)(*[at for _, at in tensors])
        num = (ctypes.c_longlong * n)(*[t.numel() for t, _ in tensors])
        fp32 = int(tensors[0][0].dtype == torch.float32)
        _call("z2h_pack_bf16", src, dst, num, n, fp32, _lib.ptr(self.w), _lib.stream_ptr())

    def view(self, name: str) -> torch.Tensor | None:
        if name not in self.offsets:
            return None
        shape = self.shapes[name]
        n = 1
        for d in shape:
            n *= d
        return self.w[self.offsets[name]:self.offsets[name] + n].view(shape)

    def step(self, tokens: torch.Tensor, pos: int, head: bool = True) -> torch.Tensor:
        """Runs the tokens [batch] (int64, any stride) at position `pos`; returns fp32 logits [batch, V]."""
        status = _lib.ptr(_lib.status_word(self.device))
        stream = _lib.stream_ptr()
        stride = tokens.stride(0)
        for g in self.groups:
            b0 = g["rows"].start
            logits = ctypes.c_void_p(self.logits.data_ptr() + 4 * b0 * self.V) if head else None
            _call("z2h_decode_step", self.numbers, _lib.ptr(self.w), _lib.ptr(g["kv"]),
                  ctypes.c_void_p(tokens.data_ptr() + 8 * b0 * stride), stride, logits, _lib.ptr(g["scratch"]),
                  g["base"], g["n"], self.C, self.H, self.L, self.V, pos, self.max_len, status, stream)
            g["base"] += g["epochs"]  # 32 bits hold some 10^7 steps of the largest model
        return self.logits

    def prefill(self, tokens: torch.Tensor) -> None:
        """Fills the cache with positions 0 .. n-1 of `tokens` [batch, n] (int64)."""
        n = tokens.shape[1]
        if n * len(self.groups) <= STEPWISE_PROMPT:
            for pos in range(n):
                self.step(tokens[:, pos], pos, head=False)
            return
        for g in self.groups:
            self._prefill(tokens[g["rows"]].contiguous(), g["kv"])

    def _prefill(self, tokens: torch.Tensor, kv: torch.Tensor) -> None:
        """The module's forward over the prompt, with the keys and values of every layer kept. The last
        layer stops there: what follows it is needed at the last position only, which a step computes."""
        B, T = tokens.shape
        C, H, M = self.C, self.H, tokens.numel()
        w = self.view

        def buf(*shape, dtype=torch.bfloat16):
            return torch.empty(*shape, device=self.device, dtype=dtype)

        x, mid, xn, att = buf(M, C), buf(M, C), buf(M, C), buf(M, C)
        qkv, act, pre = buf(M, 3 * C), buf(M, 4 * C), buf(M, 4 * C)
        mean, rstd, lse = buf(M, dtype=torch.float32), buf(M, dtype=torch.float32), buf(B, H, T, dtype=torch.float32)
        N.embed_fwd(tokens, w("transformer.wte.weight"), w("transformer.wpe.weight"), x, T)
        for i in range(self.L):
            p = f"transformer.h.{i}."
            N.layernorm_fwd(x, w(p + "ln_1.weight"), w(p + "ln_1.bias"), xn, mean, rstd)
            if i == self.L - 1:
                G.gemm(xn, w(p + "attn.c_attn.weight")[C:], qkv[:, C:], bias=w(p + "attn.c_attn.bias")[C:])
            else:
                G.gemm(xn, w(p + "attn.c_attn.weight"), qkv, bias=w(p + "attn.c_attn.bias"))
            _call("z2h_kv_from_qkv", _lib.ptr(qkv), _lib.ptr(kv[i]), B, T, self.max_len, C, _lib.stream_ptr())
            if i == self.L - 1:
                return
            N.flash_fwd(qkv, att, lse, B, T, H)
            G.gemm(att, w(p + "attn.c_proj.weight"), mid, bias=w(p + "attn.c_proj.bias"), residual=x, epi=G.EPI_RESIDUAL)
            N.layernorm_fwd(mid, w(p + "ln_2.weight"), w(p + "ln_2.bias"), xn, mean, rstd)
            G.gemm(xn, w(p + "mlp.c_fc.weight"), act, bias=w(p + "mlp.c_fc.bias"), aux_out=pre, epi=G.EPI_GELU)
            G.gemm(act, w(p + "mlp.c_proj.weight"), x, bias=w(p + "mlp.c_proj.bias"), residual=mid, epi=G.EPI_RESIDUAL)


def generate(model, X: torch.Tensor, max_new_tokens: int, temperature: float, top_k: int | None,
             generator: torch.Generator | None) -> torch.Tensor | None:
    """`GPT2.generate` with cached keys and values; None where the memory for it is not there (nothing
    has been sampled then). Positions are absolute, so once the sequence outgrows the context every
    token shifts all of them: the window is then run through the batched pass again for each token. Raises when a
    kernel has reported a failure (an expired wait, a token out of range)."""
    from .sampling import sample_next

    B, T0 = X.shape
    block = model.config.block_size
    try:
        session = DecodeSession(model, B, min(block, T0 + max_new_tokens - 1))
        tokens = torch.zeros(B, T0 + max_new_tokens, device=X.device, dtype=torch.int64)
        tokens[:, :T0] = X
        session.prefill(tokens[:, max(0, T0 - block):T0 - 1])
    except torch.OutOfMemoryError:
        return None
    for T in range(T0, T0 + max_new_tokens):
        first = max(0, T - block)
        if T > T0 and first > 0:
            session.prefill(tokens[:, first:T - 1])
        logits = session.step(tokens[:, T - 1], T - 1 - first)
        sample_next(logits, temperature, top_k, generator, out=tokens[:, T])
    if not torch.cuda.is_current_stream_capturing():
        # A wait between CTAs that ran out leaves the step's results wrong and says so in the status word alone. Read
        # once a call, after the last launch: raises, as the engine does when it reads a loss. A caller that reads the
        # tokens waits here instead of there; one that goes on launching loses that overlap (15.4 -> 16.7 ms for 64
        # tokens of the 124M model and a forward pass).
        _lib.check_status(session.device)
    return torch.cat((X, tokens[:, T0:]), dim=1)
