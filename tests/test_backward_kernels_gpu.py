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
