"""Autograd ops against fp64 PyTorch: cross-entropy of any vocabulary, linear layers of any output width
and the GELU backward."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
BF16 = 2.0 ** -8  # a rounding to bf16 is off by at most this share of the value


def _rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


# one row, rows of one vector, an odd start of every row, the usual vocabularies, the widest row that fits
@pytest.mark.parametrize("M,V", [(1, 8), (3, 65), (5, 1001), (129, 50257), (64, 50304), (7, 57297), (2, 57296)])
def test_cross_entropy(M, V):
    from zero_to_hero_b200.ops import functional as Z

    g = torch.Generator().manual_seed(M + V)
    x = (4 * torch.randn(M, V, generator=g)).bfloat16().cuda().requires_grad_()
    t = torch.randint(0, V, (M,), generator=g).cuda()
    if M > 2:
        t[1] = -100
    ref = x.detach().double().requires_grad_()
    losses = F.cross_entropy(ref, t, reduction="none")  # zero for an ignored row
    (losses.sum() / ((t != -100).sum() if V % 8 else M) * 3.0).backward()
    logits = x * 1.0
    loss = Z.cross_entropy(logits, t)
    with torch.no_grad():
        logits.zero_()  # the caller's logits are free once the loss is there
    (loss * 3.0).backward(retain_graph=True)
    first, x.grad = x.grad, None
    (loss * 3.0).backward()
    assert torch.equal(first, x.grad)
    value = float(loss.detach())
    assert abs(value - float(losses.detach().sum() / ((t != -100).sum() if V % 8 else M))) < 1e-4 * value
    assert _rel(x.grad, ref.grad) < BF16
    if M > 2:
        assert not x.grad[1].any()
    with torch.no_grad():
        assert torch.equal(Z.cross_entropy(x * 1.0, t), loss)


def test_cross_entropy_other_forms_keep_their_results():
    from zero_to_hero_b200.ops import functional as Z

    g = torch.Generator().manual_seed(0)
    x = torch.randn(6, 40, generator=g).bfloat16().cuda()
    t = torch.randint(0, 33, (6,), generator=g).cuda()
    ref = F.cross_entropy(x[:, :33].double(), t)
    for form in (x, x.float(), torch.cat((x, x), 1)[:, :40], torch.stack((x, x), 2)[:, :, 0]):
        assert abs(float(Z.cross_entropy(form, t, 33)) - float(ref)) < 1e-4
        assert abs(float(Z.cross_entropy(form, t.int(), 33)) - float(ref)) < 1e-4
    y = x[:, :33].contiguous().requires_grad_()  # an odd vocabulary can be differentiated twice
    d = y.detach().double().requires_grad_()
    for v in (y, d):
        loss = Z.cross_entropy(v, t) if v is y else F.cross_entropy(v, t)
        (grad,) = torch.autograd.grad(loss, v, create_graph=True)
        grad.square().sum().backward()
    assert _rel(y.grad, d.grad) < 4 * BF16
    lowest = torch.full((2, 33), torch.finfo(torch.bfloat16).min, dtype=torch.bfloat16, device="cuda")
    lowest[:, 5] = 1.0
    lowest[:, 6] = -torch.inf
    assert float(Z.cross_entropy(lowest, torch.tensor([5, 5], device="cuda"))) == 0.0


# rows of one value, so large that its multiple by log2(e) leaves fp32: the loss is log V whatever the value is;
# widths of both routes, and one where the rows start anywhere
@pytest.mark.parametrize("V", (33, 40, 50257))
def test_cross_entropy_of_the_largest_values(V):
    from zero_to_hero_b200.ops import functional as Z

    top = torch.finfo(torch.bfloat16).max
    for value in (-top, top, -1e5, 1e5):
        x = torch.full((3, V), value).bfloat16().cuda()
        x[1, 5:] = 0.0  # beside another row: one class, or all but five, take everything
        t = torch.tensor([1, 2, V - 1], device="cuda")
        ref = x.double().requires_grad_()
        F.cross_entropy(ref[[0, 2]], t[[0, 2]]).backward()
        x.requires_grad_()
        loss = Z.cross_entropy(x, t)
        rows = torch.stack([Z.cross_entropy(x[i:i + 1].detach(), t[i:i + 1]) for i in range(3)])
        want = F.cross_entropy(x.detach().float(), t, reduction="none")
        assert torch.allclose(rows, want, rtol=1e-6, atol=1e-6), (value, rows, want)
        loss.backward()
        assert x.grad.isfinite().all()
        assert _rel(x.grad[[0, 2]] * 1.5, ref.grad[[0, 2]]) < BF16


def test_cross_entropy_shows_a_label_out_of_range():
    from zero_to_hero_b200.ops import _lib, functional as Z

    _lib.check_status("cuda")
    x = torch.randn(4, 33).bfloat16().cuda().requires_grad_()
    for bad in (33, -1, 1 << 40):
        t = torch.tensor([1, bad, 2, -100], device="cuda")
        loss = Z.cross_entropy(x, t)
        (grad,) = torch.autograd.grad(loss, x, retain_graph=True)
        (again,) = torch.autograd.grad(loss, x, create_graph=True)
        assert loss.isnan() and grad[1].isnan().all() and again[1].isnan().all()
        with pytest.raises(RuntimeError, match="bad argument"):
            _lib.check_status("cuda")
    t = torch.tensor([1, 32, 0, -100], device="cuda")
    assert torch.allclose(Z.cross_entropy(x, t), F.cross_entropy(x.float(), t), rtol=1e-5)
    wide = torch.randn(4, 40).bfloat16().cuda()  # multiples of 8: such a row has always counted as ignored
    assert Z.cross_entropy(wide, torch.tensor([1, 40, 2, -1], device="cuda")).isfinite()
    _lib.check_status("cuda")


# what the graph keeps: freed by the backward even while the loss lives on, seen by saved-tensor hooks, and right
# for a second derivative after the caller has changed its logits
@pytest.mark.parametrize("V", (1001, 1008))
def test_cross_entropy_keeps_its_logits_in_the_graph(V):
    import weakref

    from zero_to_hero_b200.ops import functional as Z

    g = torch.Generator().manual_seed(V)
    x = torch.randn(64, V, generator=g).bfloat16().cuda().requires_grad_()
    t = torch.randint(0, V, (64,), generator=g).cuda()
    before = torch.cuda.memory_allocated()
    logits = x * 1.0
    inner, packed = weakref.ref(logits), []
    with torch.autograd.graph.saved_tensors_hooks(lambda s: packed.append(s.numel()) or s, lambda s: s):
        loss = Z.cross_entropy(logits, t)
    assert sum(n >= 64 * V for n in packed) == 1
    del logits
    assert inner() is None  # the graph holds its own copy only
    loss.backward()
    x.grad = None
    assert torch.cuda.memory_allocated() - before < 64 * V  # `loss` is alive, the copy (two bytes each) is not
    d = x.detach().double().requires_grad_()
    logits = x * 1.0
    loss, ref = Z.cross_entropy(logits, t), F.cross_entropy(d, t)
    with torch.no_grad():
        logits.zero_()
    scale = torch.ones((), device="cuda", requires_grad=True)  # a graph of the backward for both kinds of width
    (first,) = torch.autograd.grad(loss * scale, x, create_graph=True)
    first.float().square().sum().backward()
    (want,) = torch.autograd.grad(ref, d, create_graph=True)
    want.square().sum().backward()
    assert _rel(first, want) < BF16 and _rel(x.grad, d.grad) < 4 * BF16


@pytest.mark.parametrize("M,K,N,bias", [(1, 8, 1, True), (300, 384, 65, True), (130, 64, 127, False),
                                        (2048, 64, 257, True), (33, 768, 50257, False)])
def test_linear_of_any_width(M, K, N, bias):
    from zero_to_hero_b200.ops import functional as Z

    Z.FALLBACK_COUNTS.clear()
    g = torch.Generator().manual_seed(M + N)
    x = torch.randn(M, K, generator=g).cuda().requires_grad_()
    w = (torch.randn(N, K, generator=g) / K ** 0.5).cuda().requires_grad_()
    b = torch.randn(N, generator=g).cuda().requires_grad_() if bias else None
    dy = torch.randn(M, N, generator=g).cuda()
    y = Z.linear(x, w, b)
    y.backward(dy.bfloat16())
    assert not Z.FALLBACK_COUNTS and y.is_contiguous() and y.dtype == torch.bfloat16
    rx, rw = x.detach().bfloat16().double().requires_grad_(), w.detach().bfloat16().double().requires_grad_()
    rb = b.detach().bfloat16().double().requires_grad_() if bias else None
    r = F.linear(rx, rw, rb)
    r.backward(dy.bfloat16().double())
    assert _rel(y, r) < BF16 and _rel(x.grad, rx.grad) < BF16 and _rel(w.grad, rw.grad) < BF16
    assert not bias or _rel(b.grad, rb.grad) < BF16


# an upstream gradient that starts between two 16-byte boundaries, for every epilogue of the forward and with
# the bias alone wanted
@pytest.mark.parametrize("act,residual,frozen", [("gelu_tanh", False, False), (None, False, False), (None, True, False),
                                                 (None, False, True)])
def test_linear_takes_a_gradient_of_any_alignment(act, residual, frozen):
    from zero_to_hero_b200.ops import functional as Z, native

    g = torch.Generator().manual_seed(3)
    x, w, b, r = (torch.randn(*s, generator=g).bfloat16().cuda() for s in ((24, 64), (72, 64), (72,), (24, 72)))
    for t in (x, w):
        t.requires_grad_(not frozen)
    b.requires_grad_()
    up = torch.randn(24 * 72 + 1, generator=g).bfloat16().cuda()[1:].view(24, 72)
    assert up.data_ptr() % 16
    Z.linear(x, w, b, act, r if residual else None).backward(up)
    got = [t.grad for t in (x, w, b)]
    for t in (x, w, b):
        t.grad = None
    Z.linear(x, w, b, act, r if residual else None).backward(up.clone())
    assert all((p is None and t.grad is None) or torch.equal(p, t.grad) for p, t in zip(got, (x, w, b)))
    assert frozen == (x.grad is None) and b.grad is not None
    with pytest.raises(RuntimeError):  # refused by the host, nothing is launched
        native.colsum_bf16(up, torch.zeros(72, device="cuda"))


@pytest.mark.parametrize("M,N", [(1, 8), (33, 264), (1000, 256), (4099, 3072)])
def test_gelu_backward(M, N):
    from zero_to_hero_b200.ops import native

    g = torch.Generator().manual_seed(M)
    pre = (3 * torch.randn(M, N, generator=g)).bfloat16().cuda()
    pre[0, :4] = torch.tensor([0.0, 40.0, -40.0, 1e30])
    dy = torch.randn(M, N, generator=g).bfloat16().cuda()
    ref = pre.double().requires_grad_()
    F.gelu(ref, approximate="tanh").backward(dy.double())
    dx, db = torch.empty_like(dy), torch.ones(N, device="cuda")
    native.gelu_bwd(dy, pre, dx, db)
    ok = torch.isfinite(ref.grad)  # fp64's own x^3 stays finite where fp32's overflows: both end at 0 or dy
    assert _rel(dx[ok], ref.grad[ok]) < BF16 and torch.isfinite(dx).all()
    assert torch.allclose(db.double(), 1 + dx.double().sum(0), rtol=1e-4, atol=1e-4 * M ** 0.5)


def test_odd_widths_that_the_kernels_do_not_compute_keep_the_library():
    from zero_to_hero_b200.ops import functional as Z

    x, w = torch.randn(5, 64).cuda(), torch.randn(7, 64).cuda()
    for b in (torch.full((1,), 2.0).cuda(), torch.full((1, 7), 2.0).cuda()):  # broadcast
        assert torch.equal(Z.linear(x, w, b), F.linear(x.bfloat16(), w.bfloat16(), b.bfloat16()))
    for bad in ((x, w[:, :32]), (x, w.cpu()), (x, w, torch.zeros(6).cuda()), (x, w, torch.zeros(7))):
        with pytest.raises(RuntimeError):  # F.linear's own refusal, on the host
            Z.linear(*bad)


@pytest.mark.parametrize("M,N", [(1, 8), (70, 264)])
def test_relu_and_its_backward(M, N):
    from zero_to_hero_b200.ops import native

    x = torch.randn(M, N, generator=torch.Generator().manual_seed(M)).bfloat16().cuda()
    x[0, :6] = torch.tensor([0.0, -0.0, torch.nan, torch.inf, -torch.inf, 1e-40])
    dy = torch.randn(M, N, generator=torch.Generator().manual_seed(N)).bfloat16().cuda()
    ref = x.clone().requires_grad_()
    y = F.relu(ref)
    y.backward(dy)
    out = x.clone()
    native.relu_(out)
    dx, db = torch.empty_like(dy), torch.zeros(N, device="cuda")
    native.relu_bwd(dy, out, dx, db)
    assert torch.equal(out.nan_to_num(), y.detach().nan_to_num()) and torch.equal(out.isnan(), y.isnan())
    assert torch.equal(dx, ref.grad)
    assert torch.allclose(db.double(), ref.grad.double().sum(0), rtol=1e-5, atol=1e-5 * M ** 0.5)
