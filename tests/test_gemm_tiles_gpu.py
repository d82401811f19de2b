"""GEMMs of outputs with few tiles against fp64."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
BF16 = 2.0 ** -8  # a rounding to bf16 is off by at most this share of the value


def _rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


# every tile width on outputs of few tiles, every operand layout and epilogue, with remainders in every
# direction; the last one is a wave of pairs and a few tiles, which the rule gives to single SMs
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K", [(8, 8, 8), (136, 72, 64), (1000, 776, 200), (512, 1536, 384), (2304, 136, 768), (808, 4800, 192)])
@pytest.mark.parametrize("width", (64, 128, 2))
def test_gemm_narrow_tiles(M, N, K, a_mn, b_mn, width, request):
    from zero_to_hero_b200.ops import gemm as G

    G.set_algo(width)  # 2: the rule
    request.addfinalizer(lambda: G.set_algo(2))

    g = torch.Generator().manual_seed(M + N + K)
    a = torch.randn(K if a_mn else M, M if a_mn else K, generator=g).bfloat16().cuda()
    b = torch.randn(K if b_mn else N, N if b_mn else K, generator=g).bfloat16().cuda()
    bias, res = torch.randn(N, generator=g).bfloat16().cuda(), torch.randn(M, N, generator=g).bfloat16().cuda()
    ref = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    assert _rel(G.gemm(a, b, out, a_mn=a_mn, b_mn=b_mn, bias=bias), ref + bias.double()) < BF16
    assert _rel(G.gemm(a, b, out, a_mn=a_mn, b_mn=b_mn, bias=bias, residual=res, epi=G.EPI_RESIDUAL),
                ref + bias.double() + res.double()) < BF16
    pre = torch.empty_like(out)
    G.gemm(a, b, out, a_mn=a_mn, b_mn=b_mn, aux_out=pre, epi=G.EPI_GELU)
    assert _rel(pre, ref) < BF16 and _rel(out, F.gelu(ref, approximate="tanh")) < 2 * BF16
    G.gemm(a, b, out, a_mn=a_mn, b_mn=b_mn, aux_in=res, epi=G.EPI_MUL_AUX)
    assert _rel(out, ref * res.double()) < BF16
    acc = torch.ones(M, N, device="cuda")
    G.gemm(a, b, acc, a_mn=a_mn, b_mn=b_mn, epi=G.EPI_ACCUMULATE)
    assert _rel(acc, ref + 1) < 1e-5


# the remaining epilogues on the same tiles: both GELU derivatives, the column sums, atomic addition and K-slices
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K", [(8, 8, 8), (136, 72, 64), (160, 96, 72), (1000, 776, 200), (2304, 160, 768)])
@pytest.mark.parametrize("width", (64, 128, 2))
def test_gemm_narrow_tiles_other_epilogues(M, N, K, a_mn, b_mn, width, request):
    from zero_to_hero_b200.ops import gemm as G

    G.set_algo(width)  # 2: the rule
    request.addfinalizer(lambda: G.set_algo(2))
    g = torch.Generator().manual_seed(M + N + K)
    a = (torch.randn(K if a_mn else M, M if a_mn else K, generator=g) / K ** 0.5).bfloat16().cuda()
    b = torch.randn(K if b_mn else N, N if b_mn else K, generator=g).bfloat16().cuda()
    bias, x = torch.randn(N, generator=g).bfloat16().cuda(), (2 * torch.randn(M, N, generator=g)).bfloat16().cuda()
    ref = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())

    def derivative(v):
        v = v.double().requires_grad_()
        F.gelu(v, approximate="tanh").sum().backward()
        return v.grad

    kw = dict(a_mn=a_mn, b_mn=b_mn)
    whole = M % 32 == 0 and N % 32 == 0  # what the column sums need
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    db = torch.ones(N, device="cuda") if whole else None
    G.gemm(a, b, out, aux_in=x, epi=G.EPI_GELU_GRAD, colsum=db, **kw)
    assert _rel(out, ref * derivative(x)) < 2 * BF16  # tanh.approx: up to 3e-3 of a derivative around 0.6
    if whole:
        assert torch.allclose(db.double(), 1 + out.double().sum(0), rtol=1e-4, atol=1e-4 * M ** 0.5)
    grad = torch.empty_like(out)
    db = torch.ones(N, device="cuda") if whole else None
    G.gemm(a, b, out, bias=bias, aux_out=grad, epi=G.EPI_GELU_SAVE_GRAD, colsum=db, **kw)
    act = ref + bias.double()
    assert _rel(out, F.gelu(act, approximate="tanh")) < 2 * BF16 and _rel(grad, derivative(act)) < 2 * BF16
    if whole:
        assert torch.allclose(db.double(), 1 + out.double().sum(0), rtol=1e-4, atol=1e-4 * M ** 0.5)
    acc = torch.ones(M, N, device="cuda")
    G.gemm(a, b, acc, epi=G.EPI_ATOMIC_ADD, split_k=1, **kw)
    assert _rel(acc, ref + 1) < 1e-5
    G.gemm(a, b, acc.fill_(torch.nan), epi=G.EPI_SLICE_STORE, split_k=1, slice_stride=M * N, **kw)
    assert _rel(acc, ref) < 1e-5
