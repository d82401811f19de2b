"""Raw Python entry points of the sm_100a kernels (one function per C symbol).

Every function takes torch CUDA tensors, launches on the current stream and returns
immediately; nothing here allocates, so all of it can be captured into a CUDA graph. The
autograd-aware, module-level API lives in `zero_to_hero_b200.ops.functional`.
"""
from __future__ import annotations

import contextlib
import ctypes
import itertools
from ctypes import c_int, c_longlong, c_float, c_void_p

import torch

from . import _lib
from ._lib import address as ptr, raw_stream as stream_ptr

_sigs = {
    "z2h_layernorm_fwd": [c_void_p] * 6 + [c_int, c_int, c_float, c_void_p],
    "z2h_layernorm_bwd_num_partials": [c_int],
    "z2h_layernorm_bwd": [c_void_p] * 10 + [c_int, c_int, c_int, c_void_p],
    "z2h_layernorm_bwd_dxsum": [c_void_p] * 11 + [c_int, c_int, c_int, c_void_p],
    "z2h_embed_fwd": [c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int,
                      c_void_p, c_void_p],
    "z2h_embed_bwd": [c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int,
                      c_void_p],
    "z2h_embed_bwd_ordered": [c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int,
                              c_int, c_void_p],
    "z2h_colsum_bf16_ordered": [c_void_p, c_int, c_int, c_longlong, c_void_p, c_int, c_int, c_void_p, c_void_p],
    "z2h_flash_bwd_ex": [c_void_p] * 7 + [c_int, c_int, c_int, c_float, c_void_p, ctypes.c_uint,
                         c_void_p, c_int, c_void_p, c_void_p],
    "z2h_flash_bwd_sliced": [c_void_p] * 7 + [c_int, c_int, c_int, c_float, c_void_p, ctypes.c_uint,
                             c_void_p, c_int, c_int, c_void_p, c_void_p],
    "z2h_ce_fwd_bwd": [c_void_p, c_void_p, c_int, c_void_p, c_int, c_int, c_int, c_longlong,
                       c_float, c_int, c_int, c_void_p],
    "z2h_ce_fwd_save": [c_void_p, c_longlong, c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_int,
                        c_int, c_int, c_int, c_void_p, c_void_p],
    "z2h_ce_bwd": [c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_float, c_void_p, c_longlong, c_int, c_int, c_int,
                   c_int, c_int, c_void_p],
    "z2h_compact_rows": [c_void_p, c_longlong, c_void_p, c_int, c_int, c_void_p],
    "z2h_pdl_scope": [c_int],
    "z2h_relu": [c_void_p, c_longlong, c_void_p],
    "z2h_relu_bwd": [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_void_p],
    "z2h_pack_bf16": [c_void_p, c_void_p, c_void_p, c_int, c_int, c_void_p, c_void_p],
    "z2h_gelu_bwd": [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_void_p],
    "z2h_reduce_sum": [c_void_p, c_int, c_float, c_void_p, c_int, c_void_p],
    "z2h_gradnorm_partials": [c_void_p, c_longlong, c_void_p, c_void_p],
    "z2h_adamw_step": [c_void_p] * 5 + [c_longlong, c_longlong, c_void_p, c_void_p, c_int,
                                        c_void_p, c_int, c_void_p],
    "z2h_colsum_bf16": [c_void_p, c_int, c_int, c_longlong, c_void_p, c_int, c_void_p],
    "z2h_cast_f32_to_bf16": [c_void_p, c_void_p, c_longlong, c_void_p],
    "z2h_flash_fwd": [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p],
    "z2h_flash_bwd": [c_void_p] * 7 + [c_int, c_int, c_int, c_void_p, c_void_p],
    "z2h_flash_fwd_dropout": [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_float, c_void_p,
                              ctypes.c_uint, c_void_p, c_void_p],
    "z2h_flash_bwd_dbias": [c_void_p] * 7 + [c_int, c_int, c_int, c_float, c_void_p, ctypes.c_uint,
                            c_void_p, c_void_p, c_void_p],
    "z2h_flash_bwd_dropout": [c_void_p] * 7 + [c_int, c_int, c_int, c_float, c_void_p, ctypes.c_uint,
                                               c_void_p, c_void_p],
    "z2h_dropout_colsum": [c_void_p, c_void_p, c_void_p, c_int, c_int, c_float, c_void_p, ctypes.c_uint, c_void_p],
    "z2h_dropout_apply": [c_void_p, c_void_p, c_void_p, c_longlong, c_float, c_void_p, ctypes.c_uint,
                          c_void_p],
}
_fns: dict[str, ctypes._CFuncPtr] = {}


def _f(name: str):
    fn = _fns.get(name)
    if fn is None:
        fn = getattr(_lib.cuda_lib(), name)
        fn.restype = c_int
        fn.argtypes = _sigs[name]
        _fns[name] = fn
    return fn


def _check(rc: int, name: str) -> None:
    if rc != 0:
        raise RuntimeError(f"{name} failed with code {rc} (1 bad argument, 2 tensor map, 3 launch)")


@contextlib.contextmanager
def pdl_scope(on: bool):
    """Launches of this thread inside the block use programmatic dependent launch (csrc/common/launch.cuh)."""
    before = _f("z2h_pdl_scope")(int(on))
    try:
        yield
    finally:
        _f("z2h_pdl_scope")(before)


def _is64(t: torch.Tensor) -> int:
    assert t.dtype in (torch.int64, torch.int32)
    return int(t.dtype == torch.int64)


def layernorm_fwd(x, w, b, y, mean, rstd, eps=1e-5):
    M, C = x.numel() // x.shape[-1], x.shape[-1]
    _check(_f("z2h_layernorm_fwd")(ptr(x), ptr(w), ptr(b), ptr(y), ptr(mean), ptr(rstd), M, C,
                                   eps, stream_ptr()), "layernorm_fwd")


def layernorm_bwd_num_partials(M: int) -> int:
    return _f("z2h_layernorm_bwd_num_partials")(M)


def layernorm_bwd(dy, x, w, mean, rstd, dresid, dx, dw, db, scratch, accumulate=True, dxsum=None):
    """`dxsum` (fp32 [C], optional): += column sums of the output dx, i.e. the bias gradient of the
    projection whose output this residual-stream gradient is; scratch then needs 3 * C floats per
    partial row instead of 2 * C."""
    M, C = x.numel() // x.shape[-1], x.shape[-1]
    if dxsum is None:
        assert scratch.numel() >= layernorm_bwd_num_partials(M) * 2 * C
        _check(_f("z2h_layernorm_bwd")(ptr(dy), ptr(x), ptr(w), ptr(mean), ptr(rstd), ptr(dresid),
                                       ptr(dx), ptr(dw), ptr(db), ptr(scratch), M, C, int(accumulate),
                                       stream_ptr()), "layernorm_bwd")
        return
    assert scratch.numel() >= layernorm_bwd_num_partials(M) * 3 * C and dxsum.dtype == torch.float32
    _check(_f("z2h_layernorm_bwd_dxsum")(ptr(dy), ptr(x), ptr(w), ptr(mean), ptr(rstd), ptr(dresid),
                                         ptr(dx), ptr(dw), ptr(db), ptr(dxsum), ptr(scratch), M, C,
                                         int(accumulate), stream_ptr()), "layernorm_bwd_dxsum")


def embed_fwd(idx, wte, wpe, out, T):
    M, C = idx.numel(), wte.shape[1]
    _check(_f("z2h_embed_fwd")(ptr(idx), _is64(idx), ptr(wte), ptr(wpe), ptr(out), M, T, C,
                               wte.shape[0], ptr(_lib.status_word(out.device)), stream_ptr()),
           "embed_fwd")


def embed_bwd(idx, dx, dwte, dwpe, B, T, ordered: bool = False):
    """`ordered`: the token-embedding gradient is summed in ascending position by one writer per
    vocabulary row instead of with atomics (bitwise reproducible, slower)."""
    C = dx.shape[-1]
    _check(_f("z2h_embed_bwd_ordered")(ptr(idx), _is64(idx), ptr(dx), ptr(dwte), ptr(dwpe), B, T, C,
                                       dwte.shape[0], int(ordered), stream_ptr()), "embed_bwd")


def ce_fwd_bwd(logits, targets, losses, v_real, grad_scale, write_grad=True, ignore_index=-100):
    M, Vp = logits.shape
    _check(_f("z2h_ce_fwd_bwd")(ptr(logits), ptr(targets), _is64(targets), ptr(losses), M, v_real,
                                Vp, logits.stride(0), grad_scale, int(write_grad), ignore_index,
                                stream_ptr()), "ce_fwd_bwd")


CE_SAVE_MAX_COLUMNS = 57_300  # a row of logits lies in shared memory, two rows to an SM


def ce_fwd_save(logits, targets, losses, stats, copy, v_real, ignore_index=-100, strict=False):
    """Losses of the rows of `logits` [M, V] (bf16, unit inner stride, any pitch) and their maxima and
    logarithms of the sums of exp(x - maximum) (`stats`, fp32 [M, 2]); `copy` ([M, >= V] on a pitch of a
    multiple of 8, or None) receives the logits for `ce_bwd`. `strict`: a label that is neither a class nor
    `ignore_index` gives NaN and "bad argument" in the status word instead of counting as ignored."""
    M, V = logits.shape
    assert stats.shape == (M, 2) and stats.dtype == torch.float32 and stats.is_contiguous()
    _check(_f("z2h_ce_fwd_save")(ptr(logits), max(logits.stride(0), V) if M == 1 else logits.stride(0), ptr(targets),
                                 _is64(targets), ptr(losses), ptr(stats), ptr(copy),
                                 0 if copy is None else copy.stride(0), M, V, v_real, ignore_index, int(strict),
                                 ptr(_lib.status_word(logits.device)), stream_ptr()), "ce_fwd_save")


def ce_bwd(copy, targets, stats, upstream, scale, grad, V, v_real, ignore_index=-100, strict=False):
    """grad = (softmax - onehot) * scale * upstream[0]; `copy` and `grad` share one pitch."""
    assert copy.stride(0) == grad.stride(0) and upstream.dtype == torch.float32
    _check(_f("z2h_ce_bwd")(ptr(copy), ptr(targets), _is64(targets), ptr(stats), ptr(upstream), scale, ptr(grad),
                            copy.stride(0), copy.shape[0], V, v_real, ignore_index, int(strict), stream_ptr()), "ce_bwd")


def compact_rows(src, dst):
    """Tight dst [M, N] = src [M, N] on a wider pitch (bf16)."""
    _check(_f("z2h_compact_rows")(ptr(src), src.stride(0), ptr(dst), dst.shape[0], dst.shape[1], stream_ptr()),
           "compact_rows")


def gelu_bwd(dy, pre, dx, db=None):
    """dx = dy * gelu_tanh'(pre) over tight bf16 [M, N]; `db` (fp32 [N]) += column sums of dx."""
    M, N = pre.shape
    _check(_f("z2h_gelu_bwd")(ptr(dy), ptr(pre), ptr(dx), ptr(db), M, N, stream_ptr()), "gelu_bwd")


def relu_(x):
    """In place over a contiguous bf16 tensor whose size is a multiple of 8."""
    _check(_f("z2h_relu")(ptr(x), x.numel(), stream_ptr()), "relu")


def relu_bwd(dy, out, dx, db=None):
    """dx = 0 where out <= 0, else dy (at a NaN too), over tight bf16 [M, N]; `db` (fp32 [N]) += column sums of dx."""
    M, N = out.shape
    _check(_f("z2h_relu_bwd")(ptr(dy), ptr(out), ptr(dx), ptr(db), M, N, stream_ptr()), "relu_bwd")


def pack_bf16(tensors, sizes):
    """bf16 copies of contiguous, 16-byte aligned tensors of one type (fp32 or bf16), whose sizes are multiples
    of 64, one after the other in one buffer, by one launch (per 128 tensors)."""
    n = len(tensors)
    at = list(itertools.accumulate(sizes, initial=0))
    flat = torch.empty(at[-1], device=tensors[0].device, dtype=torch.bfloat16)
    _check(_f("z2h_pack_bf16")((c_void_p * n)(*[t.data_ptr() for t in tensors]), (c_longlong * n)(*at[:n]),
                               (c_longlong * n)(*sizes), n, int(tensors[0].dtype == torch.float32), ptr(flat),
                               stream_ptr()), "pack_bf16")
    return flat


def reduce_sum(x, out, scale=1.0, accumulate=False):
    _check(_f("z2h_reduce_sum")(ptr(x), x.numel(), scale, ptr(out), int(accumulate), stream_ptr()),
           "reduce_sum")


def gradnorm_partials(g, partials) -> int:
    n = _f("z2h_gradnorm_partials")(ptr(g), g.numel(), ptr(partials), stream_ptr())
    if n < 0:
        raise RuntimeError(f"gradnorm_partials failed with code {n}")
    return n


def adamw_step(p32, g, m, v, p16, n_decay, hyper, partials, num_partials, norm_out, zero_grad=True):
    _check(_f("z2h_adamw_step")(ptr(p32), ptr(g), ptr(m), ptr(v), ptr(p16), p32.numel(), n_decay,
                                ptr(hyper), ptr(partials), num_partials, ptr(norm_out),
                                int(zero_grad), stream_ptr()), "adamw_step")


def colsum_scratch_elems(M: int, N: int) -> int:
    """fp32 elements of scratch the ordered column sum of an M x N matrix uses (up to 128 partial rows)."""
    return min(128, max(1, (M + 127) // 128)) * N


def colsum_bf16(dy, db, accumulate=True, ordered: bool = False, scratch=None):
    """db (+)= column sums of dy. By default up to 128 row slabs are summed by CTAs of their own and
    meet in atomics. `ordered`: bitwise reproducible; with `scratch` (fp32, colsum_scratch_elems) the
    slabs store their partial sums there and a second kernel adds them in slab order, without it one CTA
    sums a whole column block (slow)."""
    M, N = dy.shape
    if scratch is not None:
        assert scratch.dtype == torch.float32 and scratch.numel() >= colsum_scratch_elems(M, N)
    _check(_f("z2h_colsum_bf16_ordered")(ptr(dy), M, N, dy.stride(0), ptr(db), int(accumulate), int(ordered),
                                         ptr(scratch), stream_ptr()), "colsum_bf16")


def cast_f32_to_bf16(src, dst):
    _check(_f("z2h_cast_f32_to_bf16")(ptr(src), ptr(dst), src.numel(), stream_ptr()), "cast")


def flash_fwd(qkv, out, lse, B, T, H, drop_p: float = 0.0, seed=None, site: int = 0):
    """Causal attention forward. With `drop_p` > 0 the attention probabilities are dropped with
    the mask of (`seed` [int64 device tensor of one element], `site`); see ops/dropout.py."""
    if drop_p > 0.0:
        assert seed is not None and seed.dtype == torch.int64 and seed.is_cuda
        _check(_f("z2h_flash_fwd_dropout")(ptr(qkv), ptr(out), ptr(lse), B, T, H, drop_p, ptr(seed), site,
                                           ptr(_lib.status_word(out.device)), stream_ptr()),
               "flash_fwd_dropout")
        return
    _check(_f("z2h_flash_fwd")(ptr(qkv), ptr(out), ptr(lse), B, T, H,
                               ptr(_lib.status_word(out.device)), stream_ptr()), "flash_fwd")


def flash_bwd_stats_elems(B: int, T: int, H: int) -> int:
    """Number of fp32 scratch elements `flash_bwd` needs for its per-row statistics."""
    return 2 * B * H * ((T + 127) // 128 * 128)


def flash_bwd_dq_elems(B: int, T: int, H: int) -> int:
    """Number of fp32 scratch elements `flash_bwd` needs for its dQ accumulation (rows rounded up
    to a multiple of 32: the kernels keep dQ there in a blocked layout)."""
    return (B * T + 31) // 32 * 32 * H * 64


def flash_bwd_copies(B: int, T: int, H: int, limit_mb: float = 512.0) -> int:
    """dq_accum copies worth having for the ordered form: one per 128-key tile, or 1 where they would take
    more than `limit_mb` (long contexts: their number and their size both grow with T)."""
    n = (T + 127) // 128
    return n if n * flash_bwd_dq_elems(B, T, H) * 4 <= limit_mb * 2 ** 20 else 1


def flash_bwd(qkv, out, dout, lse, dqkv, dq_accum, stats, B, T, H, drop_p: float = 0.0, seed=None,
              site: int = 0, dbias=None, ordered: bool = False):
    """`dbias` (fp32 [3*H*64]): the column sums of `dqkv` as stored are ADDED to it, i.e. the gradient
    of the QKV projection's bias comes out of the attention backward kernels.
    `ordered`: the fp32 accumulation of dQ happens in KV-tile order (bitwise reproducible; not together with
    `dbias`). With `flash_bwd_copies` times the dq_accum scratch every KV tile stores to a copy of its own;
    with less the KV tiles are launched one after the other (about 1.5x slower, the same bits)."""
    assert stats.numel() >= flash_bwd_stats_elems(B, T, H)
    assert dq_accum.numel() >= flash_bwd_dq_elems(B, T, H) and dq_accum.dtype == torch.float32
    if ordered:
        assert dbias is None, "the bias by-product is accumulated with atomics"
        if drop_p > 0.0:
            assert seed is not None and seed.dtype == torch.int64 and seed.is_cuda
        _check(_f("z2h_flash_bwd_sliced")(ptr(qkv), ptr(out), ptr(dout), ptr(lse), ptr(dqkv), ptr(dq_accum),
                                          ptr(stats), B, T, H, drop_p, ptr(seed) if drop_p > 0.0 else None, site,
                                          None, 1, dq_accum.numel() // flash_bwd_dq_elems(B, T, H),
                                          ptr(_lib.status_word(out.device)), stream_ptr()),
               "flash_bwd_sliced")
        return
    if dbias is not None:
        assert dbias.dtype == torch.float32 and dbias.numel() == 3 * H * 64 and dbias.is_contiguous()
        if drop_p > 0.0:
            assert seed is not None and seed.dtype == torch.int64 and seed.is_cuda
        _check(_f("z2h_flash_bwd_dbias")(ptr(qkv), ptr(out), ptr(dout), ptr(lse), ptr(dqkv),
                                         ptr(dq_accum), ptr(stats), B, T, H, drop_p,
                                         ptr(seed) if drop_p > 0.0 else None, site, ptr(dbias),
                                         ptr(_lib.status_word(out.device)), stream_ptr()),
               "flash_bwd_dbias")
        return
    if drop_p > 0.0:
        assert seed is not None and seed.dtype == torch.int64 and seed.is_cuda
        _check(_f("z2h_flash_bwd_dropout")(ptr(qkv), ptr(out), ptr(dout), ptr(lse), ptr(dqkv),
                                           ptr(dq_accum), ptr(stats), B, T, H, drop_p, ptr(seed), site,
                                           ptr(_lib.status_word(out.device)), stream_ptr()),
               "flash_bwd_dropout")
        return
    _check(_f("z2h_flash_bwd")(ptr(qkv), ptr(out), ptr(dout), ptr(lse), ptr(dqkv), ptr(dq_accum),
                               ptr(stats), B, T, H, ptr(_lib.status_word(out.device)),
                               stream_ptr()), "flash_bwd")


def dropout_apply(x, out, drop_p: float, seed, site: int, residual=None):
    """out = dropout(x) (+ residual) over contiguous bf16 tensors; `out` may be `x`. The mask is a
    function of (seed[0], site, element index): applying the call to a gradient with the same seed
    and site is the backward of the forward call (ops/dropout.py restates the mask on the host)."""
    assert x.is_contiguous() and out.is_contiguous() and x.dtype == torch.bfloat16
    assert seed.dtype == torch.int64 and seed.is_cuda
    if residual is not None:
        assert residual.is_contiguous() and residual.numel() == x.numel()
    _check(_f("z2h_dropout_apply")(ptr(x), ptr(residual), ptr(out), x.numel(), drop_p, ptr(seed), site,
                                   stream_ptr()), "dropout_apply")


def dropout_colsum(x, out, db, drop_p: float, seed, site: int):
    """out = dropout(x) over a contiguous bf16 [M, N] with the mask `dropout_apply` uses; `db` (fp32 [N])
    += column sums of out."""
    assert x.is_contiguous() and out.is_contiguous() and x.dtype == torch.bfloat16 and db.dtype == torch.float32
    M, N = x.shape
    _check(_f("z2h_dropout_colsum")(ptr(x), ptr(out), ptr(db), M, N, drop_p, ptr(seed), site, stream_ptr()),
           "dropout_colsum")
