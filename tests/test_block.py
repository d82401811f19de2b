"""The transformer block as one autograd node: which blocks take it (CPU) and its results (GPU)."""
import copy

import pytest
import torch
import torch.nn as nn

from zero_to_hero_b200.config import ModelConfig
from zero_to_hero_b200.models.gpt import GPTLM
from zero_to_hero_b200.models.gpt2 import GPT2


def _gpt2(heads=2, layers=2, vocab=96, block=64, ln_bias=True, dropout=0.0):
    torch.manual_seed(0)
    return GPT2(ModelConfig(vocab_size=vocab, block_size=block, emb_dim=64 * heads, num_heads=heads, num_layers=layers,
                            dropout=dropout, ln_bias=ln_bias))


def _char(heads=2, layers=2, vocab=65, block=64, dropout=0.0):
    torch.manual_seed(0)
    return GPTLM(vocab, block, 64 * heads, layers, heads, dropout)


def test_only_plain_blocks_are_fused():
    def gpt2(edit, **kw):
        m = _gpt2(**kw)
        edit(m.transformer.h[0])
        return m.transformer.h[0]._parts() is not None

    def char(edit, **kw):
        m = _char(**kw)
        edit(m.blocks[0])
        return m.blocks[0]._parts() is not None

    class Own(nn.Linear):
        pass

    for case, inner in ((gpt2, lambda b: b.mlp), (char, lambda b: b.ff)):
        assert case(lambda b: None) and case(lambda b: b.eval(), dropout=0.1) and not case(lambda b: None, dropout=0.1)
        assert case(lambda b: b.register_forward_hook(lambda *a: None))  # the block is still called as a module
        assert not case(lambda b: inner(b).register_forward_hook(lambda *a: None))
        assert not case(lambda b: inner(b).register_full_backward_hook(lambda *a: None))
        assert not case(lambda b: b.attn.register_forward_pre_hook(lambda *a: None))
        assert not case(lambda b: setattr(b.attn, "forward", lambda x: x))
    assert not gpt2(lambda b: setattr(b.attn, "c_attn", Own(128, 384)))
    assert not char(lambda b: setattr(b.attn.heads[1], "key", Own(128, 64, bias=False)))
    assert not char(lambda b: setattr(b.ff.ff, "1", nn.GELU()))
    from zero_to_hero_b200.ops import block as FB
    assert not FB.usable(torch.zeros(1, 2, 128, dtype=torch.bfloat16), 2, [torch.zeros(128)])  # not on a GPU
    whole = [torch.zeros(3)] * 12
    shapes = ((3,),) * 12
    assert FB.shaped(whole, shapes) and not FB.shaped(whole, shapes[:11]) and not FB.shaped(whole, shapes[:11] + ((3, 3),))
    for i in range(12):  # in the order of the node's parameters: only biases may be absent
        assert FB.shaped([None if j == i else t for j, t in enumerate(whole)], shapes) == (i in (1, 2, 4, 6, 8, 10))


def test_blocks_with_replaced_parts_are_not_touched():
    class Odd(nn.Module):  # none of the attributes of what it stands for
        def forward(self, *args):
            return args[0]

    def gone(make, path):
        m = make()
        b = m.transformer.h[0] if make is _gpt2 else m.blocks[0]
        *way, last = path.split(".")
        owner = b
        for name in way:
            owner = getattr(owner, name)
        setattr(owner, last, Odd())
        return b._parts()

    for path in ("ln_1", "ln_2", "attn", "mlp", "attn.c_attn", "attn.c_proj", "mlp.c_fc", "mlp.c_proj"):
        assert gone(_gpt2, path) is None, path
    for path in ("ln1", "ln2", "attn", "ff", "attn.proj", "attn.heads", "ff.ff", "attn.heads.0", "attn.heads.1.key",
                 "ff.ff.0", "ff.ff.1", "ff.ff.2", "ff.ff.4"):
        assert gone(_char, path) is None, path


# the same on a GPU: such a block runs through its parts
@pytest.mark.gpu
@pytest.mark.parametrize("make", (_gpt2, _char))
def test_block_with_another_attention_runs(make):
    class Own(nn.Module):
        def forward(self, x, residual=None, cdrop=None):
            return x if residual is None else residual + x

    m = make()
    (m.transformer.h[0] if make is _gpt2 else m.blocks[0]).attn = Own()
    m = m.cuda()
    X = torch.randint(0, 60, (2, 9)).cuda()
    m(X, X)[1].backward()
    assert all(p.grad.isfinite().all() for p in m.parameters())


def _grads(model, X, Y):
    model.zero_grad(set_to_none=True)
    logits, loss = model(X, Y)
    loss.backward()
    return logits.detach().double().cpu(), [p.grad.double().cpu() for p in model.parameters()], float(loss.detach())


# one token, a whole and a part of a 32-row group, several tiles; one head up to a wide block; tied and untied
# vocabularies of both kinds; fp32 and bf16 parameters; LayerNorm with and without bias
@pytest.mark.gpu
@pytest.mark.parametrize("make,B,T,kw,bf16", [
    (_gpt2, 1, 1, {"heads": 1}, False), (_gpt2, 2, 64, {"ln_bias": False}, False), (_gpt2, 3, 41, {"vocab": 97}, False),
    (_gpt2, 4, 300, {"heads": 12, "block": 512}, False), (_gpt2, 2, 50, {"heads": 3}, True),
    (_char, 1, 3, {"heads": 1}, False), (_char, 5, 63, {}, False), (_char, 8, 256, {"heads": 6, "block": 256}, False)])
def test_block_matches_the_single_ops(make, B, T, kw, bf16):
    m = make(**kw)
    vocab = m.config.vocab_size if make is _gpt2 else 65
    g = torch.Generator().manual_seed(B * T)
    X, Y = (torch.randint(0, vocab, (B, T), generator=g) for _ in range(2))
    m = m.bfloat16() if bf16 else m
    oracle = copy.deepcopy(m).double()
    m = m.cuda()
    blocks = m.transformer.h if make is _gpt2 else m.blocks
    assert all(b._parts() is not None for b in blocks)
    ref = _grads(oracle, X, Y)
    got = _grads(m, X.cuda(), Y.cuda())
    handles = [b.attn.register_forward_hook(lambda *a: None) for b in blocks]  # the single ops
    single = _grads(m, X.cuda(), Y.cuda())
    for h in handles:
        h.remove()

    def off(r):
        scale = torch.sqrt(sum(v.square().sum() for v in ref[1]))
        return (float((r[0] - ref[0]).norm() / ref[0].norm()),
                float(torch.sqrt(sum((a - b).square().sum() for a, b in zip(r[1], ref[1]))) / scale))

    # the same rounding points, so two draws of one error; 2e-3 is a single bf16 rounding
    for a, b in zip(off(got), off(single)):
        assert a <= 1.3 * b + 2e-3, (off(got), off(single))
    # each parameter by itself, as errors in a bias or LayerNorm gradient do not show beside the matrices (the two
    # are within 1.2 of each other; what is a thousandth of all gradients together is noise)
    whole = torch.sqrt(sum(v.square().sum() for v in ref[1]))
    for (n, _), r, a, b in zip(m.named_parameters(), ref[1], got[1], single[1]):
        assert (a - r).norm() <= 1.3 * (b - r).norm() + 2e-3 * max(r.norm(), 1e-3 * whole), n
    # the loss: that of the logits beside it, and off from the exact one by the mean of the tokens' errors, which
    # is their size over sqrt(tokens), and by the second-order term of the logits' errors
    def per_token(logits):
        return nn.functional.cross_entropy(logits.flatten(0, 1), Y.flatten(), reduction="none")

    for r in (got, single):
        assert abs(r[2] - float(per_token(r[0]).mean())) < 1e-5 * abs(r[2])
        d = per_token(r[0]) - per_token(ref[0])
        assert abs(r[2] - ref[2]) <= 4 * float(d.square().mean().sqrt()) / d.numel() ** 0.5 + \
            float((r[0] - ref[0]).square().mean())
    frozen = [p for b in blocks for p in b.parameters() if p.dim() >= 2][:2]
    for p in frozen:
        p.requires_grad_(False)
    m.zero_grad(set_to_none=True)
    m(X.cuda(), Y.cuda())[1].backward()
    assert all(p.grad is None for p in frozen)
    assert all(p.grad is not None for p in m.parameters() if p.requires_grad)


# The derivative of the activation by itself: a hidden unit's input is its bias alone, every unit gets the
# gradient 16, and the bias gradient adds the same number once per token.
@pytest.mark.gpu
@pytest.mark.parametrize("T", (32, 31))
def test_block_gelu_derivative_is_exact(T):
    block = _gpt2(layers=1).transformer.h[0]
    with torch.no_grad():
        block.mlp.c_fc.weight.zero_()
        block.mlp.c_fc.bias.copy_(torch.linspace(-5, 5, 512).bfloat16())
        block.mlp.c_proj.weight.fill_(0.125)
    block = block.cuda()
    out = block(torch.randn(1, T, 128).bfloat16().cuda())
    assert "_Block" in type(out.grad_fn).__name__
    out.backward(torch.ones_like(out))
    b = block.mlp.c_fc.bias.detach().double().requires_grad_()
    nn.functional.gelu(b, approximate="tanh").sum().backward()
    want = 16 * T * b.grad
    # 512 numbers rounded to 8 bits each, and an error of 1e-6 in the derivative
    assert ((block.mlp.c_fc.bias.grad.double() - want).abs() <= 2.0 ** -8 * want.abs() + 16 * T * 2e-6).all()


@pytest.mark.gpu
@pytest.mark.parametrize("make", (_gpt2, _char))
def test_block_gradients_do_not_share_memory(make):
    m = make().cuda()
    X = torch.randint(0, 60, (2, 33)).cuda()
    m(X, X)[1].backward()
    for b in m.transformer.h if make is _gpt2 else m.blocks:
        for n, p in b.named_parameters():
            size = p.grad.untyped_storage().nbytes()
            if ".heads." in n:  # row blocks of one matrix, whose gradient is one product
                assert size == 3 * p.shape[1] ** 2 * 4
            else:
                assert size == p.numel() * 4
