"""Backward kernels at the sizes where their pipelines can go wrong."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = 2.0 ** -8


def _rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


# a warp with no row, one row, its ring's two rows, more; rows of one vector up to the widest; with and
# without a bias, a residual gradient and the column sums
@pytest.mark.parametrize("M", (1, 9, 2369, 7105))
@pytest.mark.parametrize("C,bias,extra", [(8, True, False), (768, False, True), (776, True, True), (2048, False, False),
                                          (2048, True, True)])
def test_layernorm_backward(M, C, bias, extra):
    from zero_to_hero_b200.ops import native as N

    g = torch.Generator().manual_seed(M + C)
    x, dy, res = (torch.randn(M, C, generator=g).bfloat16().cuda() for _ in range(3))
    w = torch.randn(C, generator=g).bfloat16().cuda()
    y, mean, rstd = torch.empty_like(x), torch.empty(M, device="cuda"), torch.empty(M, device="cuda")
    N.layernorm_fwd(x, w, None, y, mean, rstd)
    dx, dw = torch.empty_like(x), torch.ones(C, device="cuda")
    db = torch.ones(C, device="cuda") if bias else None
    dxsum = torch.ones(C, device="cuda") if extra else None
    scratch = torch.empty(N.layernorm_bwd_num_partials(M) * 3 * C, device="cuda")
    N.layernorm_bwd(dy, x, w, mean, rstd, res if extra else None, dx, dw, db, scratch, dxsum=dxsum)
    xd = x.double().requires_grad_()
    wd, bd = w.double().requires_grad_(), torch.zeros(C, dtype=torch.float64, device="cuda", requires_grad=True)
    torch.nn.functional.layer_norm(xd, (C,), wd, bd).backward(dy.double())
    want = xd.grad + res.double() if extra else xd.grad
    assert _rel(dx, want) < BF16 and _rel(dw, 1 + wd.grad) < 1e-4
    assert db is None or _rel(db, 1 + bd.grad) < 1e-4
    if extra:  # sums of what was computed, in fp32, before it was rounded for storage
        assert float((dxsum.double() - 1 - want.sum(0)).abs().max()) < 1e-4 * M ** 0.5 * float(want.abs().max())
    again = torch.empty_like(x)
    N.layernorm_bwd(dy, x, w, mean, rstd, res if extra else None, again, dw, db, scratch, dxsum=dxsum)
    assert torch.equal(again, dx)


# one tile, a second one of one row, several tiles and sequences whose rows share 32-row blocks
@pytest.mark.parametrize("B,T,H,p", [(1, 128, 1, 0.0), (2, 129, 2, 0.0), (3, 509, 2, 0.0), (2, 1024, 1, 0.2)])
def test_ordered_attention_backward_in_one_launch(B, T, H, p):
    from zero_to_hero_b200.ops import native as N

    C = 64 * H
    g = torch.Generator().manual_seed(T)
    qkv = (0.7 * torch.randn(B * T, 3 * C, generator=g)).bfloat16().cuda()
    out, dout = torch.empty(B * T, C, device="cuda", dtype=torch.bfloat16), torch.randn(B * T, C, generator=g).bfloat16().cuda()
    lse = torch.empty(B, H, T, device="cuda")
    seed = torch.tensor([3], device="cuda")
    N.flash_fwd(qkv, out, lse, B, T, H, p, seed, 1)
    elems, results = N.flash_bwd_dq_elems(B, T, H), []
    copies = N.flash_bwd_copies(B, T, H)
    assert copies == (T + 127) // 128
    for n in (1, copies, copies):  # a launch per KV tile, then one launch, twice
        dqkv = torch.zeros_like(qkv)
        dq = torch.full((n * elems,), float("nan"), device="cuda")
        N.flash_bwd(qkv, out, dout, lse, dqkv, dq, torch.empty(N.flash_bwd_stats_elems(B, T, H), device="cuda"), B, T, H,
                    p, seed, 1, ordered=True)
        results.append(dqkv)
    assert torch.equal(results[0], results[1]) and torch.equal(results[1], results[2])


def test_long_contexts_keep_one_copy():
    from zero_to_hero_b200.ops import native as N

    assert N.flash_bwd_copies(16, 1024, 12) == 8 and N.flash_bwd_copies(1, 65536, 16) == 1
    assert N.flash_bwd_copies(16, 1024, 12, 384) == 8 and N.flash_bwd_copies(16, 1024, 12, 383) == 1
    assert N.flash_bwd_copies(1, 128, 1, 0) == N.flash_bwd_copies(1, 129, 1, 0) == 1


# fewer positions than vocabulary rows (a warp per position) and as many (a warp per row); more than one
# chunk of ids and of columns; tokens that occur often, once, never and out of range
@pytest.mark.parametrize("B,T,C,V", [(1, 1, 8, 2), (3, 70, 264, 1000), (5, 509, 384, 50257), (2, 3000, 264, 6000)])
def test_ordered_embedding_gradient(B, T, C, V):
    from zero_to_hero_b200.ops import native as N

    g = torch.Generator().manual_seed(T)
    idx = torch.randint(0, V, (B, T), generator=g)
    idx[:, ::3] = idx[0, 0]
    idx[-1, -1] = V + 5  # clamped into the table
    dx = torch.randn(B * T, C, generator=g).bfloat16()
    want = torch.zeros(V, C).index_add_(0, idx.clamp(0, V - 1).flatten(), dx.float())  # ascending, fp32
    for dtype in (torch.int64, torch.int32):
        dwte, dwpe = torch.zeros(V, C, device="cuda"), torch.zeros(T, C, device="cuda")
        N.embed_bwd(idx.to(dtype).cuda(), dx.cuda(), dwte, dwpe, B, T, ordered=True)
        assert torch.equal(dwte.cpu(), want)


@pytest.mark.parametrize("M,N", [(1, 8), (33, 264), (4099, 768)])
def test_dropout_with_column_sums(M, N):
    from zero_to_hero_b200.ops import native

    x = torch.randn(M, N, generator=torch.Generator().manual_seed(M)).bfloat16().cuda()
    seed = torch.tensor([7], device="cuda")
    want, out = torch.empty_like(x), torch.empty_like(x)
    native.dropout_apply(x, want, 0.2, seed, 5)
    db = torch.ones(N, device="cuda")
    native.dropout_colsum(x, out, db, 0.2, seed, 5)
    assert torch.equal(out, want)
    assert torch.allclose(db.double(), 1 + want.double().sum(0), rtol=1e-4, atol=1e-4 * M ** 0.5)
