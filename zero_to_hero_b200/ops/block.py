"""One pre-norm transformer block as one autograd node.

    mid = x + proj(attention(ln1(x)));   out = mid + fc2(act(fc(ln2(mid))))

The single ops of `ops.functional` cost a block about 45 kernel launches and as many autograd nodes in
Python; here it is 8 launches forward (all parameters cast and packed by one of them) and about 17 backward,
in which the projection's bias gradient comes out of the LayerNorm backward, the QKV bias gradient out of
the attention backward and the c_fc bias gradient out of the activation's backward. Rounding points are
those of the single ops (the character model's residual sums round once instead of twice); nothing is dropped
out (blocks with active dropout take the single ops).
"""
from __future__ import annotations

import math

import torch

from . import gemm as G, native as N
from .functional import pick_split_k

_ORDER = ("ln1_w", "ln1_b", "b_qkv", "w_proj", "b_proj", "ln2_w", "ln2_b", "w_fc", "b_fc", "w_fc2", "b_fc2")
_BIASES = ("ln1_b", "b_qkv", "b_proj", "ln2_b", "b_fc", "b_fc2")
_SHAPES = {"w_proj": (1, 1), "w_fc": (4, 1), "w_fc2": (1, 4)}  # in units of C


def usable(x: torch.Tensor, num_heads: int, params) -> bool:
    """Whether `block` takes these: bf16 [B, T, 64 * heads] on a GPU (at most 2048 wide) and contiguous
    parameters of one type, fp32 or bf16, on x's device."""
    if not x.is_cuda or x.dtype != torch.bfloat16 or x.dim() != 3 or x.numel() == 0:
        return False
    if x.shape[2] != 64 * num_heads or x.shape[2] > 2048:
        return False
    first = params[0]
    return first is not None and first.dtype in (torch.float32, torch.bfloat16) and all(
        p is None or (p.dtype == first.dtype and p.device == x.device and p.is_contiguous() and p.data_ptr() % 16 == 0)
        for p in params)


def shaped(params, shapes) -> bool:
    """The parameters, those of `_ORDER` and the row blocks of the QKV weight, have these shapes; biases may be
    absent, and nothing else (the kernels would read a weight that is not there at address 0)."""
    return len(params) == len(shapes) and all(p is None or tuple(p.shape) == s for p, s in zip(params, shapes)) and \
        all(p is not None or name in _BIASES for p, name in zip(params, _ORDER + ("w_qkv",) * (len(params) - len(_ORDER))))


def plain_modules(pairs) -> bool:
    """Every (module, class): calling the module runs that class's forward and nothing else."""
    g = torch.nn.modules.module
    if g._global_forward_hooks or g._global_forward_pre_hooks or g._global_backward_hooks or g._global_backward_pre_hooks:
        return False
    return all(type(m) is c and not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or
                                     m._backward_pre_hooks or "forward" in m.__dict__) for m, c in pairs)


def _wgrad(dy, x, out):
    """out (fp32 zeros) = dy^T x"""
    sk = pick_split_k(math.ceil(out.shape[0] / 128) * math.ceil(out.shape[1] / 256), math.ceil(dy.shape[0] / 64))
    if sk == 1:
        G.gemm(dy, x, out, a_mn=True, b_mn=True)
    else:
        G.gemm(dy, x, out, a_mn=True, b_mn=True, epi=G.EPI_ATOMIC_ADD, split_k=sk)


def _split(flat, named, sizes, C):
    """(name -> view, the [3C, C] QKV view) of a buffer that holds the parameters `named` and then the row
    blocks of the QKV weight, `sizes` elements each."""
    pieces = flat.split([*sizes[:len(named)], 3 * C * C])
    views = dict.fromkeys(_ORDER)
    for n, t in zip(named, pieces):
        views[n] = t.view(_SHAPES[n][0] * C, _SHAPES[n][1] * C) if n in _SHAPES else t
    return views, pieces[-1].view(3 * C, C)


class _Block(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, num_heads, act, eps1, eps2, *params):
        B, T, C = x.shape
        M, F, dev = B * T, 4 * C, x.device
        x2 = x.reshape(M, C).contiguous()
        if x2.data_ptr() % 16:
            x2 = x2.clone()
        # bf16 copies of all parameters in one buffer; the QKV weight may come in several row blocks
        tensors = [p for p in params if p is not None]
        named = [n for n, p in zip(_ORDER, params) if p is not None]
        sizes = [p.numel() for p in tensors]
        flat = N.pack_bf16(tensors, sizes)
        w, w_qkv = _split(flat, named, sizes, C)

        def buf(*shape, dtype=torch.bfloat16):
            return torch.empty(*shape, device=dev, dtype=dtype)

        xn1, qkv, att, mid, xn2, hid, out = (buf(M, n) for n in (C, 3 * C, C, C, C, F, C))
        stats, lse = buf(4, M, dtype=torch.float32), buf(B, num_heads, T, dtype=torch.float32)
        N.layernorm_fwd(x2, w["ln1_w"], w["ln1_b"], xn1, stats[0], stats[1], eps1)
        G.gemm(xn1, w_qkv, qkv, bias=w["b_qkv"])
        N.flash_fwd(qkv, att, lse, B, T, num_heads)
        G.gemm(att, w["w_proj"], mid, bias=w["b_proj"], residual=x2, epi=G.EPI_RESIDUAL)
        N.layernorm_fwd(mid, w["ln2_w"], w["ln2_b"], xn2, stats[2], stats[3], eps2)
        pre = None
        if act == "gelu_tanh":
            pre = buf(M, F)
            G.gemm(xn2, w["w_fc"], hid, bias=w["b_fc"], aux_out=pre, epi=G.EPI_GELU)
        else:
            G.gemm(xn2, w["w_fc"], hid, bias=w["b_fc"])
            N.relu_(hid)
        G.gemm(hid, w["w_fc2"], out, bias=w["b_fc2"], residual=mid, epi=G.EPI_RESIDUAL)
        ctx.save_for_backward(x2, flat, xn1, qkv, att, lse, mid, xn2, pre, hid, stats)
        ctx.meta = (B, T, C, num_heads, named, sizes, params[0].dtype)
        return out.view(B, T, C)

    @staticmethod
    def backward(ctx, dout):
        x2, flat, xn1, qkv, att, lse, mid, xn2, pre, hid, stats = ctx.saved_tensors
        B, T, C, H, named, sizes, dtype = ctx.meta
        M, F, dev = B * T, 4 * C, x2.device
        need = ctx.needs_input_grad[5:]
        dy = dout.reshape(M, C)
        dy = (dy if dy.dtype == torch.bfloat16 else dy.bfloat16()).contiguous()
        if dy.data_ptr() % 16:
            dy = dy.clone()

        def buf(*shape, dtype=torch.bfloat16):
            return torch.empty(*shape, device=dev, dtype=dtype)

        # fp32 gradients, zeroed together; each a tensor of its own, because they become the parameters' `.grad`: as
        # views of one buffer any of them would keep, and a saved one would contain, those of the whole block
        new, f32, g = flat.new_empty, torch.float32, dict.fromkeys(_ORDER)
        for n, size in zip(named, sizes):
            g[n] = new((_SHAPES[n][0] * C, _SHAPES[n][1] * C) if n in _SHAPES else size, dtype=f32)
        g_qkv = new((3 * C, C), dtype=f32)
        torch._foreach_zero_([g_qkv, *(g[n] for n in named)])
        w, w_qkv = _split(flat, named, sizes, C)
        needs = dict(zip(_ORDER, need))

        d4, dc, dmid = buf(M, F), buf(M, C), buf(M, C)
        scratch = buf(N.layernorm_bwd_num_partials(M) * 3 * C, dtype=torch.float32)
        # MLP
        if needs["w_fc2"]:
            _wgrad(dy, hid, g["w_fc2"])
        if g["b_fc2"] is not None:
            N.colsum_bf16(dy, g["b_fc2"])
        # One pass for the activation's derivative and the bias gradient. The GEMM's own GELU epilogue would save it,
        # but takes tanh from tanh.approx, whose 11 bits leave errors of 20 % where the derivative is small, and with an
        # exact derivative it is no faster: 8192 x 3072 x 768 68 us so, 71 us as an epilogue; 2331 rows 23 and 29.
        dh = buf(M, F)
        G.gemm(dy, w["w_fc2"], dh, b_mn=True)
        if pre is not None:
            N.gelu_bwd(dh, pre, d4, g["b_fc"])
        else:
            N.relu_bwd(dh, hid, d4, g["b_fc"])
        if needs["w_fc"]:
            _wgrad(d4, xn2, g["w_fc"])
        G.gemm(d4, w["w_fc"], dc, b_mn=True)
        N.layernorm_bwd(dc, mid, w["ln2_w"], stats[2], stats[3], dy, dmid, g["ln2_w"], g["ln2_b"], scratch,
                        dxsum=g["b_proj"])
        # attention
        if needs["w_proj"]:
            _wgrad(dmid, att, g["w_proj"])
        G.gemm(dmid, w["w_proj"], dc, b_mn=True)
        dqkv = buf(M, 3 * C)
        dq = buf(N.flash_bwd_dq_elems(B, T, H), dtype=torch.float32)
        fstats = buf(N.flash_bwd_stats_elems(B, T, H), dtype=torch.float32)
        N.flash_bwd(qkv, att, dc, lse, dqkv, dq, fstats, B, T, H, dbias=g["b_qkv"])
        if any(need[len(_ORDER):]):
            _wgrad(dqkv, xn1, g_qkv)
        G.gemm(dqkv, w_qkv, dc, b_mn=True)
        dx = buf(M, C)
        N.layernorm_bwd(dc, x2, w["ln1_w"], stats[0], stats[1], dmid, dx, g["ln1_w"], g["ln1_b"], scratch)
        parts = len(sizes) - len(named)
        blocks = (g_qkv,) if parts == 1 else g_qkv.view(parts, 3 * C // parts, C).unbind(0)
        out = [*(g[n] for n in _ORDER), *blocks]
        out = [t if t is None or dtype == torch.float32 else t.to(dtype) for t in out]
        out = [t if n else None for t, n in zip(out, need)]
        return (dx.view(B, T, C), None, None, None, None, *out)


def block(x, num_heads, act, eps1, eps2, ln1, b_qkv, proj, ln2, fc, fc2, qkv_weights):
    """`ln1`, `ln2`, `proj`, `fc`, `fc2`: (weight, bias or None); `qkv_weights`: one [3C, C] weight or its row
    blocks in order; act: "gelu_tanh" or "relu"."""
    return _Block.apply(x, num_heads, act, eps1, eps2, *ln1, b_qkv, *proj, *ln2, *fc, *fc2, *qkv_weights)
