"""Which calls of the autograd ops take the kernels for unpadded widths (rules only, on the CPU)."""
import torch

from zero_to_hero_b200.ops import functional as Z


def test_odd_widths_take_the_kernels_only_for_what_they_compute():
    def ok(x, w, b=None):
        return Z._any_width_ok(x, w, b)

    x, w = torch.zeros(2, 3, 16), torch.zeros(7, 16)
    assert ok(x, w) and ok(x, w, torch.zeros(7)) and ok(x[0, 0], w) and ok(x.bfloat16(), w.double())
    for b in (torch.zeros(1), torch.zeros(()), torch.zeros(1, 7), torch.zeros(6)):  # broadcast or refused by F.linear
        assert not ok(x, w, b)
    assert not ok(x, torch.zeros(7, 8)) and not ok(x, torch.zeros(16)) and not ok(x[:0], w) and not ok(x, w[:0])
    elsewhere = torch.zeros(7, 16, device="meta")
    assert not ok(x, elsewhere) and not ok(x, w, elsewhere[:, 0])
    with torch.autocast("cpu", dtype=torch.bfloat16):
        assert ok(x, w)
    with torch.autocast("cpu", dtype=torch.float16):
        assert not ok(x, w)
    torch.use_deterministic_algorithms(True)
    try:
        assert not ok(x, w)
    finally:
        torch.use_deterministic_algorithms(False)


def test_traces_and_transforms_are_seen():
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.fx.experimental.proxy_tensor import make_fx

    seen = []

    def look(x):
        seen.append(Z._transformed())
        return x * 2.0

    x = torch.ones(3)
    look(x)
    assert seen == [False]
    torch.func.vmap(look)(x)
    torch.func.jvp(look, (x,), (x,))
    torch.func.grad(lambda v: look(v).sum())(x)
    torch.jit.trace(look, (x,), check_trace=False)
    make_fx(look)(x)
    with FakeTensorMode():
        look(torch.ones(3))
    assert len(seen) == 7 and all(seen[1:])
    look(x)
    assert not seen[-1]


def test_tensors_of_another_device_than_the_current_one(monkeypatch):
    class On:
        def __init__(self, device):
            self.device = torch.device(device)

    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    assert Z._here(On("cuda:1")) and not Z._here(On("cuda:0")) and not Z._here(On("cuda:2"))
    # as on a GPU, on another device: the library's operations
    monkeypatch.setattr(Z, "_native", lambda t: True)
    monkeypatch.setattr(Z, "_here", lambda t: False)
    g = torch.Generator().manual_seed(1)
    x, w = torch.randn(4, 16, generator=g).bfloat16(), torch.randn(7, 16, generator=g).bfloat16()
    logits, targets = Z.linear(x, w), torch.tensor([0, 6, -100, 3])
    assert torch.equal(logits, torch.nn.functional.linear(x, w))
    assert torch.equal(Z.cross_entropy(logits, targets), torch.nn.functional.cross_entropy(logits.float(), targets))
