"""Autograd-aware ops used by the model classes.

On a CUDA device every op runs the hand-written sm_100a kernels (bf16 activations, fp32
statistics / gradients) through `torch.autograd.Function`s; on CPU the same functions fall
back to plain PyTorch in the input dtype, which is also the fp32 oracle the kernel tests
compare against. There is no silent fallback on a GPU: if the native library is missing the
call raises.

Shapes the tensor-core GEMM cannot take (contracted sizes that are not multiples of 8 elements,
i.e. 16 bytes for TMA) are routed to `torch.matmul` in bf16 and counted in
`FALLBACK_COUNTS` so tests can assert the hot shapes never take that route.
"""
from __future__ import annotations

import math
from collections import Counter

import torch
import torch.nn.functional as F

from . import _lib, gemm as G, native as N

FALLBACK_COUNTS: Counter = Counter()


def _native(t: torch.Tensor) -> bool:
    return t.is_cuda


_sm_count: dict[int, int] = {}


def sm_count() -> int:
    """SMs of the current CUDA device (148 on a B200; the same figure is assumed without a GPU)."""
    if not torch.cuda.is_available():
        return 148
    d = torch.cuda.current_device()
    if d not in _sm_count:
        _sm_count[d] = torch.cuda.get_device_properties(d).multi_processor_count
    return _sm_count[d]


def pick_split_k(tiles: int, k_blocks: int, num_sms: int | None = None, min_kb: int = 16) -> int:
    """Split-K factor for a weight-gradient GEMM (few output tiles, very long K).

    `tiles` counts 128 x 256 output tiles (one per SM); the kernel that runs them works on CTA
    pairs with 256 x 256 tiles, so the model below uses half as many tiles and half as many
    workers. Cost of a factor s, in k-blocks of main loop: waves(s) * ceil(k_blocks / s) plus
    2 * s for the extra atomic accumulation traffic. Returns 1 (plain deterministic accumulation)
    when the tiles alone fill the machine for several waves.
    """
    if num_sms is None:
        num_sms = sm_count()
    if tiles >= 4 * num_sms or k_blocks < 2 * min_kb:
        return 1
    pair_tiles, workers = max(1, (tiles + 1) // 2), max(1, num_sms // 2)
    best, best_cost = 1, float("inf")
    for s in range(1, 17):
        if s > 1 and k_blocks // s < min_kb:
            break
        cost = math.ceil(pair_tiles * s / workers) * math.ceil(k_blocks / s) + 2 * s
        if cost < best_cost - 1e-9:
            best, best_cost = s, cost
    return best


def _gemm_ok(*dims: int) -> bool:
    return all(d % 8 == 0 for d in dims)


def _tight(t: torch.Tensor) -> torch.Tensor:
    """Contiguous and on the 16-byte boundary the tensor maps and the vector loads need."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


# --------------------------------------------------------------------------------------------
# linear
# --------------------------------------------------------------------------------------------
class _Linear(torch.autograd.Function):
    """y = act(x @ w.T + b) (+ residual) on the tcgen05 GEMM; act in {None, "gelu_tanh"}."""

    @staticmethod
    def forward(ctx, x, w, b, act, residual):
        K = x.shape[-1]
        Nout = w.shape[0]
        x2 = x.reshape(-1, K)
        if x2.dtype != torch.bfloat16:
            x2 = x2.bfloat16()
        x2 = x2.contiguous()
        w16 = w if w.dtype == torch.bfloat16 else w.detach().bfloat16()
        b16 = None if b is None else (b if b.dtype == torch.bfloat16 else b.detach().bfloat16())
        M = x2.shape[0]
        y = torch.empty(M, Nout, device=x.device, dtype=torch.bfloat16)
        pre = None
        if act == "gelu_tanh":
            pre = torch.empty_like(y)
            G.gemm(x2, w16, y, bias=b16, aux_out=pre, epi=G.EPI_GELU)
        elif residual is not None:
            r2 = residual.reshape(M, Nout)
            r2 = (r2 if r2.dtype == torch.bfloat16 else r2.bfloat16()).contiguous()
            G.gemm(x2, w16, y, bias=b16, residual=r2, epi=G.EPI_RESIDUAL)
        else:
            G.gemm(x2, w16, y, bias=b16)
        ctx.save_for_backward(x2, w16, pre)
        ctx.has_bias = b is not None
        ctx.has_res = residual is not None
        ctx.x_shape = x.shape
        ctx.w_dtype = w.dtype
        ctx.b_dtype = None if b is None else b.dtype
        ctx.x_dtype = x.dtype
        ctx.res_dtype = None if residual is None else residual.dtype
        return y.reshape(*x.shape[:-1], Nout)

    @staticmethod
    def backward(ctx, dy):
        x2, w16, pre = ctx.saved_tensors
        M, K = x2.shape
        Nout = w16.shape[0]
        dy2 = dy.reshape(M, Nout)
        dy2 = _tight(dy2 if dy2.dtype == torch.bfloat16 else dy2.bfloat16())
        dres = dy2.reshape(dy.shape).to(ctx.res_dtype) if ctx.has_res else None
        dx = dw = db32 = None
        want_db = ctx.has_bias and ctx.needs_input_grad[2]
        if want_db:
            db32 = torch.zeros(Nout, device=dy.device, dtype=torch.float32)
        if pre is not None:  # dpre = dy * gelu'(pre), its column sums on the way
            dpre = torch.empty_like(pre)
            N.gelu_bwd(dy2, pre, dpre, db32)
            dy2 = dpre
        elif want_db:
            N.colsum_bf16(dy2, db32, accumulate=True)
        if ctx.needs_input_grad[0]:
            dx2 = torch.empty(M, K, device=dy.device, dtype=torch.bfloat16)
            G.gemm(dy2, w16, dx2, b_mn=True)
            dx = dx2.reshape(ctx.x_shape).to(ctx.x_dtype)
        if ctx.needs_input_grad[1]:
            dw32 = torch.zeros(Nout, K, device=dy.device, dtype=torch.float32)
            tiles = math.ceil(Nout / 128) * math.ceil(K / 256)
            sk = pick_split_k(tiles, math.ceil(M / 64))
            G.gemm(dy2, x2, dw32, a_mn=True, b_mn=True, epi=G.EPI_ATOMIC_ADD, split_k=sk)
            dw = dw32.to(ctx.w_dtype)
        return dx, dw, None if db32 is None else db32.to(ctx.b_dtype), None, dres


def _transformed() -> bool:
    """Inside a function transform (vmap, torch.func.grad), forward-mode differentiation, a trace (compile, jit,
    make_fx) or a dispatch mode (fake tensors): a launch through plain addresses would be missing from what is
    transformed or recorded."""
    if torch.compiler.is_compiling() or torch.jit.is_tracing() or torch._C._len_torch_dispatch_stack() > 0:
        return True
    return torch._C._functorch.peek_interpreter_stack() is not None or torch.autograd.forward_ad._current_level >= 0


def _here(t: torch.Tensor) -> bool:
    """On the current device, where launches go; the library's operations run where their tensors are."""
    return t.device.index is None or t.device.index == torch.cuda.current_device()


def _any_width_ok(x, w, b) -> bool:
    """Whether `_LinearAnyWidth` computes what F.linear over bf16 casts does here. Anything that F.linear refuses,
    broadcasts or computes in another type or order goes to it: the kernels take plain addresses."""
    if w.dim() != 2 or x.dim() < 1 or w.shape[1] != x.shape[-1] or x.numel() == 0 or w.numel() == 0:
        return False
    if b is not None and b.shape != w.shape[:1]:
        return False
    if not _here(x) or any(t.device != x.device for t in (w, b) if t is not None):
        return False
    if torch.is_autocast_enabled(x.device.type) and torch.get_autocast_dtype(x.device.type) != torch.bfloat16:
        return False
    return not torch.are_deterministic_algorithms_enabled()  # the weight gradient may add with atomics


class _LinearAnyWidth(torch.autograd.Function):
    """y = x @ w.T + b over bf16 tensors for output widths that are no multiple of 8 (an unpadded
    vocabulary): the tensor cores work on a 16-byte pitch, the caller gets tight rows."""

    @staticmethod
    def forward(ctx, x, w, b):
        Nout, K = w.shape
        x2 = _tight(x.reshape(-1, K))
        M = x2.shape[0]
        wide = torch.empty(M, (Nout + 7) // 8 * 8, device=x.device, dtype=torch.bfloat16)
        G.gemm(x2, _tight(w), wide[:, :Nout], bias=None if b is None else _tight(b))
        y = torch.empty(M, Nout, device=x.device, dtype=torch.bfloat16)
        N.compact_rows(wide, y)
        ctx.save_for_backward(x, w)
        ctx.has_bias = b is not None
        return y.reshape(*x.shape[:-1], Nout)

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        Nout, K = w.shape
        need_x, need_w, need_b = ctx.needs_input_grad
        d2, x2 = dy.reshape(-1, Nout), x.reshape(-1, K)
        if torch.is_grad_enabled():  # a graph of this backward is wanted: plain operations
            return ((d2 @ w).reshape(x.shape) if need_x else None, d2.t() @ x2 if need_w else None,
                    d2.sum(0) if need_b else None)
        M = d2.shape[0]
        if d2.stride(1) != 1 or d2.stride(0) % 8 or d2.stride(0) < Nout or d2.data_ptr() % 16:
            d2 = d2.new_empty(M, (Nout + 7) // 8 * 8)[:, :Nout].copy_(d2)
        dx = dw = db = None
        if need_x:
            dx = torch.empty(M, K, device=dy.device, dtype=torch.bfloat16)
            G.gemm(d2, _tight(w), dx, b_mn=True)
            dx = dx.reshape(x.shape)
        if need_w:
            sk = pick_split_k(math.ceil(Nout / 128) * math.ceil(K / 256), math.ceil(M / 64))
            if sk == 1:
                dw = torch.empty(Nout, K, device=dy.device, dtype=torch.bfloat16)
                G.gemm(d2, _tight(x2), dw, a_mn=True, b_mn=True)
            else:
                dw = torch.zeros(Nout, K, device=dy.device, dtype=torch.float32)
                G.gemm(d2, _tight(x2), dw, a_mn=True, b_mn=True, epi=G.EPI_ATOMIC_ADD, split_k=sk)
                dw = dw.bfloat16()
        if need_b:
            db = d2.sum(0, dtype=torch.float32).bfloat16()
        return dx, dw, db


def linear(x, w, b=None, act: str | None = None, residual=None):
    """`act(x @ w.T + b) + residual`; act is None or "gelu_tanh" (not both act and residual)."""
    assert not (act and residual is not None)
    K, Nout = x.shape[-1], w.shape[0]
    if _native(x) and _gemm_ok(K, Nout):
        return _Linear.apply(x, w, b, act, residual)
    if _native(x) and _gemm_ok(K) and act is None and residual is None and not _transformed() and _any_width_ok(x, w, b):
        return _LinearAnyWidth.apply(x.bfloat16(), w.bfloat16(), None if b is None else b.bfloat16())
    if _native(x):
        FALLBACK_COUNTS["linear"] += 1
        y = F.linear(x.bfloat16(), w.bfloat16(), None if b is None else b.bfloat16())
    else:
        y = F.linear(x, w, b)
    if act == "gelu_tanh":
        y = F.gelu(y, approximate="tanh")
    if residual is not None:
        y = y + residual
    return y


# --------------------------------------------------------------------------------------------
# layer norm
# --------------------------------------------------------------------------------------------
class _LayerNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, b, eps):
        C = x.shape[-1]
        x2 = x.reshape(-1, C)
        x2 = (x2 if x2.dtype == torch.bfloat16 else x2.bfloat16()).contiguous()
        w16 = w if w.dtype == torch.bfloat16 else w.detach().bfloat16()
        b16 = None if b is None else (b if b.dtype == torch.bfloat16 else b.detach().bfloat16())
        M = x2.shape[0]
        y = torch.empty_like(x2)
        mean = torch.empty(M, device=x.device, dtype=torch.float32)
        rstd = torch.empty_like(mean)
        N.layernorm_fwd(x2, w16, b16, y, mean, rstd, eps)
        ctx.save_for_backward(x2, w16, mean, rstd)
        ctx.meta = (x.shape, x.dtype, w.dtype, None if b is None else b.dtype)
        return y.reshape(x.shape)

    @staticmethod
    def backward(ctx, dy):
        x2, w16, mean, rstd = ctx.saved_tensors
        shape, x_dtype, w_dtype, b_dtype = ctx.meta
        M, C = x2.shape
        dy2 = dy.reshape(M, C)
        dy2 = (dy2 if dy2.dtype == torch.bfloat16 else dy2.bfloat16()).contiguous()
        dx = torch.empty_like(x2)
        dw = torch.empty(C, device=dy.device, dtype=torch.float32)
        db = torch.empty_like(dw) if b_dtype is not None else None
        scratch = torch.empty(N.layernorm_bwd_num_partials(M) * 2 * C, device=dy.device,
                              dtype=torch.float32)
        N.layernorm_bwd(dy2, x2, w16, mean, rstd, None, dx, dw, db, scratch, accumulate=False)
        return (dx.reshape(shape).to(x_dtype), dw.to(w_dtype),
                None if db is None else db.to(b_dtype), None)


def layer_norm(x, w, b=None, eps: float = 1e-5):
    C = x.shape[-1]
    if _native(x) and C % 8 == 0 and C <= 2048:
        return _LayerNorm.apply(x, w, b, eps)
    if _native(x):
        FALLBACK_COUNTS["layer_norm"] += 1
    return F.layer_norm(x, (C,), w, b, eps)


# --------------------------------------------------------------------------------------------
# attention
# --------------------------------------------------------------------------------------------
class _FlashAttention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, num_heads):
        B, T, C3 = qkv.shape
        C = C3 // 3
        q2 = qkv.reshape(B * T, C3)
        q2 = (q2 if q2.dtype == torch.bfloat16 else q2.bfloat16()).contiguous()
        out = torch.empty(B * T, C, device=qkv.device, dtype=torch.bfloat16)
        lse = torch.empty(B, num_heads, T, device=qkv.device, dtype=torch.float32)
        N.flash_fwd(q2, out, lse, B, T, num_heads)
        ctx.save_for_backward(q2, out, lse)
        ctx.meta = (B, T, num_heads, qkv.dtype)
        return out.reshape(B, T, C)

    @staticmethod
    def backward(ctx, dout):
        q2, out, lse = ctx.saved_tensors
        B, T, H, dtype = ctx.meta
        C = H * 64
        d2 = dout.reshape(B * T, C)
        d2 = (d2 if d2.dtype == torch.bfloat16 else d2.bfloat16()).contiguous()
        dqkv = torch.empty_like(q2)
        dq_accum = torch.empty(N.flash_bwd_dq_elems(B, T, H), device=dout.device, dtype=torch.float32)
        stats = torch.empty(N.flash_bwd_stats_elems(B, T, H), device=dout.device, dtype=torch.float32)
        N.flash_bwd(q2, out, d2, lse, dqkv, dq_accum, stats, B, T, H)
        return dqkv.reshape(B, T, 3 * C).to(dtype), None


def causal_attention(qkv: torch.Tensor, num_heads: int, dropout_p: float = 0.0) -> torch.Tensor:
    """Causal multi-head self-attention over a packed [B, T, 3C] projection; returns [B, T, C]."""
    B, T, C3 = qkv.shape
    C = C3 // 3
    hd = C // num_heads
    if _native(qkv) and hd == 64 and dropout_p == 0.0:
        return _FlashAttention.apply(qkv, num_heads)
    if _native(qkv):
        FALLBACK_COUNTS["attention"] += 1
    q, k, v = qkv.split(C, dim=-1)
    q = q.view(B, T, num_heads, hd).transpose(1, 2)
    k = k.view(B, T, num_heads, hd).transpose(1, 2)
    v = v.view(B, T, num_heads, hd).transpose(1, 2)
    y = F.scaled_dot_product_attention(q, k, v, is_causal=True, dropout_p=dropout_p)
    return y.transpose(1, 2).contiguous().view(B, T, C)


# --------------------------------------------------------------------------------------------
# embedding
# --------------------------------------------------------------------------------------------
class _Embedding(torch.autograd.Function):
    @staticmethod
    def forward(ctx, idx, wte, wpe):
        B, T = idx.shape
        C = wte.shape[1]
        wte16 = wte if wte.dtype == torch.bfloat16 else wte.detach().bfloat16()
        wpe16 = None if wpe is None else (wpe if wpe.dtype == torch.bfloat16 else wpe.detach().bfloat16())
        out = torch.empty(B * T, C, device=idx.device, dtype=torch.bfloat16)
        idxc = idx.contiguous()
        N.embed_fwd(idxc, wte16, wpe16, out, T)
        ctx.save_for_backward(idxc)
        ctx.meta = (B, T, wte.shape, wte.dtype, None if wpe is None else (wpe.shape, wpe.dtype))
        return out.reshape(B, T, C)

    @staticmethod
    def backward(ctx, dout):
        (idx,) = ctx.saved_tensors
        B, T, wshape, wdtype, pmeta = ctx.meta
        C = wshape[1]
        d2 = dout.reshape(B * T, C)
        d2 = (d2 if d2.dtype == torch.bfloat16 else d2.bfloat16()).contiguous()
        dwte = torch.zeros(wshape, device=dout.device, dtype=torch.float32)
        dwpe = None
        if pmeta is not None:
            dwpe = torch.zeros(pmeta[0], device=dout.device, dtype=torch.float32)
        N.embed_bwd(idx, d2, dwte, dwpe, B, T)
        return None, dwte.to(wdtype), None if dwpe is None else dwpe.to(pmeta[1])


def embedding(idx: torch.Tensor, wte: torch.Tensor, wpe: torch.Tensor | None = None) -> torch.Tensor:
    """wte[idx] + wpe[arange(T)] (the position table may be longer than T)."""
    B, T = idx.shape
    if _native(idx) and wte.shape[1] % 8 == 0:
        return _Embedding.apply(idx, wte, wpe)
    out = F.embedding(idx, wte)
    if wpe is not None:
        out = out + wpe[:T]
    return out


# --------------------------------------------------------------------------------------------
# cross entropy
# --------------------------------------------------------------------------------------------
class _CrossEntropy(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, targets, v_real):
        M, V = logits.shape
        buf = logits.detach().bfloat16().clone() if logits.dtype == torch.bfloat16 else logits.detach().bfloat16()
        if buf.stride(0) % 8 != 0:
            raise ValueError("logits row pitch must be a multiple of 8 elements")
        losses = torch.empty(M, device=logits.device, dtype=torch.float32)
        N.ce_fwd_bwd(buf, targets.contiguous(), losses, v_real, 1.0 / M, write_grad=True)
        ctx.save_for_backward(buf)
        ctx.dtype = logits.dtype
        return losses.mean()

    @staticmethod
    def backward(ctx, g):
        (dlogits,) = ctx.saved_tensors
        return (dlogits.float() * g).to(ctx.dtype), None, None


class _CrossEntropySaved(torch.autograd.Function):
    """The same over bf16 logits whose rows are tight in memory, any vocabulary: one pass forward that keeps
    a copy of the logits (the caller's may change before the backward), one pass backward that rounds the
    gradient once. The copy is an output beside the loss: saved like any tensor and freed with the graph, and
    what a second derivative goes through. `skip_ignored`: the mean is over the targets that are not ignored,
    and a label that names neither a class nor -100 makes it NaN (and shows in the status word)."""

    @staticmethod
    def forward(ctx, logits, targets, v_real, skip_ignored):
        M, V = logits.shape
        targets = targets.contiguous()
        losses = torch.empty(M, device=logits.device, dtype=torch.float32)
        stats = torch.empty(M, 2, device=logits.device, dtype=torch.float32)
        copy = None
        ctx.set_materialize_grads(False)
        if ctx.needs_input_grad[0]:
            copy = torch.empty(M, (V + 7) // 8 * 8, device=logits.device, dtype=torch.bfloat16)
        N.ce_fwd_save(logits, targets, losses, stats, copy, v_real, strict=skip_ignored)
        count = (targets != -100).sum().float() if skip_ignored else None
        if copy is not None:
            ctx.save_for_backward(copy, targets, stats, count)
            ctx.meta = (M, V, v_real)
        return (losses.mean() if count is None else losses.sum() / count), copy

    @staticmethod
    def backward(ctx, g, g_copy):
        copy, targets, stats, count = ctx.saved_tensors
        M, V, v_real = ctx.meta
        skipping = count is not None
        if g_copy is not None:  # a second derivative, on its way to the logits
            g_copy = g_copy[:, :V]
        if g is None:
            return g_copy, None, None, None
        if torch.is_grad_enabled() and (g.requires_grad or skipping):  # a graph of this backward is wanted
            x = copy[:, :v_real].float()
            valid = ((targets >= 0) & (targets < v_real)).float()
            if skipping:
                valid = valid.masked_fill((valid == 0) & (targets != -100), math.nan)
            hit = (targets[:, None] == torch.arange(v_real, device=x.device)).float()
            grad = F.pad((x.softmax(1) - hit) * valid[:, None], (0, V - v_real))
            grad = (grad * (g / count if skipping else g / M)).bfloat16()
            return grad if g_copy is None else grad + g_copy, None, None, None
        grad = torch.empty_like(copy)
        up = g / count if skipping else g
        N.ce_bwd(copy, targets, stats, up.reshape(1), 1.0 if skipping else 1.0 / M, grad, V, v_real, strict=skipping)
        return grad[:, :V] if g_copy is None else grad[:, :V] + g_copy, None, None, None


def cross_entropy(logits: torch.Tensor, targets: torch.Tensor, v_real: int | None = None) -> torch.Tensor:
    """Mean softmax cross-entropy over rows; columns >= v_real are vocabulary padding."""
    V = logits.shape[-1]
    v_real = V if v_real is None else v_real
    if _native(logits):
        x, t = logits.reshape(-1, V), targets.reshape(-1)
        tight = (x.dtype == torch.bfloat16 and V <= N.CE_SAVE_MAX_COLUMNS and 1 <= v_real <= V and x.shape[0] > 0
                 and t.shape[0] == x.shape[0] and x.is_contiguous())
        if V % 8 == 0:
            if tight and t.dtype in (torch.int64, torch.int32):
                return _CrossEntropySaved.apply(x, t, v_real, False)[0]
            return _CrossEntropy.apply(x, t, v_real)
        if tight and t.dtype == torch.int64 and t.device == x.device and _here(x) and not _transformed():
            return _CrossEntropySaved.apply(x, t, v_real, True)[0]
    if _native(logits):
        FALLBACK_COUNTS["cross_entropy"] += 1
    return F.cross_entropy(logits.reshape(-1, V)[:, :v_real].float(), targets.reshape(-1))
