"""Cached decoding: the rules that send a call there (CPU) and its results (GPU)."""
import copy

import pytest
import torch
import torch.nn as nn

from zero_to_hero_b200.config import ModelConfig
from zero_to_hero_b200.models.gpt2 import GPT2
from zero_to_hero_b200.ops import decode


def _model(heads=2, layers=2, vocab=101, block=40, ln_bias=False, dropout=0.0, seed=0):
    torch.manual_seed(seed)
    cfg = ModelConfig(vocab_size=vocab, block_size=block, emb_dim=64 * heads, num_heads=heads, num_layers=layers,
                      dropout=dropout, ln_bias=ln_bias)
    m = GPT2(cfg)
    with torch.no_grad():  # biases and norm weights that matter, logits that spread
        for n, p in m.named_parameters():
            if p.dim() < 2:
                p.add_(0.1 * torch.randn_like(p))
        m.transformer.wte.weight.normal_(0.0, 0.3)
        m.transformer.wpe.weight.normal_(0.0, 0.3)
    return m.eval()


@pytest.mark.parametrize("ln_bias", (False, True))
def test_packed_layout_holds_every_parameter_once(ln_bias):
    m = _model(heads=3, layers=3, vocab=77, ln_bias=ln_bias)
    off, numbers, total = decode.packed_layout(m.config)
    spans = sorted((off[n], off[n] + p.numel()) for n, p in m.named_parameters())
    assert len(spans) == len(off) and all(a % 64 == 0 for a, _ in spans) and spans[-1][1] <= total
    assert all(e <= s for (_, e), (s, _) in zip(spans, spans[1:]))
    names = ("attn.c_attn.weight", "attn.c_proj.weight", "mlp.c_fc.weight", "mlp.c_proj.weight", "ln_1.weight",
             "ln_1.bias", "attn.c_attn.bias", "attn.c_proj.bias", "ln_2.weight", "ln_2.bias", "mlp.c_fc.bias",
             "mlp.c_proj.bias")
    assert len(numbers) == 18
    for i in range(3):
        for n, o in zip(names, numbers[6:]):
            key = f"transformer.h.{i}.{n}"
            assert (o == -1) == (key not in off)
            if o >= 0:
                assert numbers[2] + i * numbers[3] + o == off[key]


def test_only_plain_models_take_the_decode_kernel():
    plain = _model()
    assert decode.plain_model(plain) and decode.plain_model(plain.bfloat16())
    assert not decode.supports(plain, torch.zeros(1, 3, dtype=torch.int64))  # not on a GPU

    def changed(edit, **kw):
        m = _model(**kw)
        edit(m)
        return decode.plain_model(m)

    class Own(nn.Linear):
        pass

    assert not changed(lambda m: m.register_forward_hook(lambda *a: None))
    assert not changed(lambda m: m.transformer.h[1].mlp.register_forward_pre_hook(lambda *a: None))
    assert not changed(lambda m: setattr(m.transformer.h[0].attn, "c_proj", Own(128, 128)))
    assert not changed(lambda m: setattr(m.lm_head, "weight", nn.Parameter(m.lm_head.weight.detach().clone())))
    assert not changed(lambda m: setattr(m.transformer.ln_f, "eps", 1e-6))
    assert not changed(lambda m: setattr(m.transformer.h[0].attn, "num_heads", 1))
    assert not changed(lambda m: m.transformer.h[0].double())
    assert not changed(lambda m: m.half())
    assert not changed(lambda m: m.transformer.wpe.__setattr__("weight", nn.Parameter(torch.zeros(41, 128))))
    assert not changed(lambda m: setattr(m.transformer.h[0].mlp.c_fc, "bias", None))
    assert not changed(lambda m: setattr(m.transformer.h[0].mlp.c_fc, "weight",
                                         nn.Parameter(torch.zeros(128, 512).t())))
    assert not changed(lambda m: m.train(), dropout=0.1)
    assert changed(lambda m: m.train()) and changed(lambda m: None, dropout=0.1)


def test_shapes_that_the_kernel_refuses_keep_the_general_path(monkeypatch):
    asked = []

    def epochs(n, C, layers):  # a device where eight wide sequences do not fit
        asked.append((n, C, layers))
        return 0 if n * C > 8 * 1024 else 5 * layers

    monkeypatch.setattr(decode, "_f", lambda name: {"z2h_decode_epochs": epochs}[name])
    assert decode.group_sizes(1) == [1] and decode.group_sizes(8) == [8] and decode.group_sizes(19) == [8, 8, 3]
    assert decode.kernel_takes(19, 1024, 2) and sorted(asked) == [(3, 1024, 2), (8, 1024, 2)]
    assert decode.kernel_takes(3, 2048, 2) and not decode.kernel_takes(8, 2048, 2) and not decode.kernel_takes(11, 2048, 2)


# widths below one row per SM up to the widest, batches of one launch and of several, every kind of
# remainder in vocabulary and length; several key ranges per head (one sequence, long context)
@pytest.mark.gpu
@pytest.mark.parametrize("heads,layers,vocab,block,B,T,ln_bias,bf16", [
    (1, 1, 5, 9, 1, 9, True, False), (2, 2, 101, 40, 3, 12, False, False), (12, 2, 50257, 64, 8, 5, False, False),
    (12, 2, 1000, 700, 1, 650, True, False), (25, 2, 50304, 300, 4, 270, False, True),
    (32, 1, 777, 1024, 8, 530, True, False), (6, 3, 65, 128, 11, 100, True, True)])
def test_decode_matches_the_forward_pass(heads, layers, vocab, block, B, T, ln_bias, bf16):
    m = _model(heads, layers, vocab, block, ln_bias)
    X = torch.randint(0, vocab, (B, T), generator=torch.Generator().manual_seed(1))
    oracle = copy.deepcopy(m).double()
    m = m.cuda().bfloat16() if bf16 else m.cuda()
    if bf16:
        oracle = copy.deepcopy(m).cpu().double()
    n = min(T, 6)  # positions compared: the last six (the first ones of short prompts)
    Xc = X.cuda()
    with torch.inference_mode():
        assert decode.supports(m, Xc)
        s = decode.DecodeSession(m, B, T)
        s.prefill(Xc[:, :T - n])
        got = torch.stack([s.step(Xc[:, t], t).clone() for t in range(T - n, T)], 1).cpu().double()
        mod = torch.stack([m(Xc[:, :t + 1])[0][:, -1].float() for t in range(T - n, T)], 1).cpu().double()
        ref = torch.stack([oracle(X[:, :t + 1])[0][:, -1] for t in range(T - n, T)], 1)
    scale = ref.norm()
    e_got, e_mod = (got - ref).norm() / scale, (mod - ref).norm() / scale
    # both round activations to bf16 at the same places, so their errors are two draws of one size
    assert e_got <= 1.3 * e_mod + 1e-3, (float(e_got), float(e_mod))


# NaN keys reach the result, wherever they lie: one among others, all keys of a warp (it takes four neighbours and
# those 60 further on), a whole key range, the step's own. The sequence beside them stays clean.
@pytest.mark.gpu
@pytest.mark.parametrize("T,first,count", [(1, 0, 1), (3, 0, 1), (5, 4, 1), (9, 4, 4), (64, 0, 1), (60, 8, 4), (61, 60, 1),
                                           (900, 301, 1), (900, 100, 250), (900, 0, 899), (897, 780, 117)])
def test_decode_keeps_nan(T, first, count):
    m = _model(heads=2, layers=1, vocab=101, block=900).cuda()
    X = torch.randint(0, 101, (2, T), generator=torch.Generator().manual_seed(T)).cuda()
    with torch.inference_mode():
        s = decode.DecodeSession(m, 2, T)
        s.prefill(X[:, :T - 1])
        clean = s.step(X[:, T - 1], T - 1).clone()
        s.groups[0]["kv"][0, 0, 0, first:first + count, 70] = torch.nan  # a column of head 1
        if first + count == T:  # the step's own key: a bias reaches it, and the other sequence's too
            s.view("transformer.h.0.attn.c_attn.bias")[128 + 70] = torch.nan
        got = s.step(X[:, T - 1], T - 1)
    assert clean.isfinite().all() and got[0].isnan().all()
    assert got[1].isnan().all() if first + count == T else torch.equal(got[1], clean[1])


# Sequences that outgrow the context: from there on every token moves the window. The logits that each token is
# taken from against the module's forward and fp64 over the same window, and the greedy choice from them.
@pytest.mark.gpu
@pytest.mark.parametrize("block,T0,new,layers", [(24, 20, 12, 2), (24, 24, 3, 2), (24, 31, 5, 2), (8, 1, 20, 1), (1, 3, 4, 1)])
def test_generate_past_the_context_window(block, T0, new, layers, monkeypatch):
    from zero_to_hero_b200.ops import sampling

    m = _model(heads=2, layers=layers, vocab=101, block=block)
    oracle = copy.deepcopy(m).double()
    m = m.cuda()
    X = torch.randint(0, 101, (2, T0), generator=torch.Generator().manual_seed(2))
    seen, real = [], sampling.sample_next

    def spy(logits, *args, **kw):
        seen.append(logits.clone())
        return real(logits, *args, **kw)

    monkeypatch.setattr(sampling, "sample_next", spy)
    out = m.generate(X.cuda(), new, top_k=1)
    assert len(seen) == new and out.shape == (2, T0 + new) and torch.equal(out[:, :T0].cpu(), X)
    got = torch.stack(seen, 1)
    # a tie of bf16 logits goes to any of the largest
    assert torch.equal(got.gather(2, out[:, T0:, None]).squeeze(2), got.amax(2))
    windows = [out[:, max(0, t - block):t] for t in range(T0, T0 + new)]
    with torch.inference_mode():
        mod = torch.stack([m(w)[0][:, -1].float() for w in windows], 1).cpu().double()
        ref = torch.stack([oracle(w.cpu())[0][:, -1] for w in windows], 1)
    errors = [(v - ref).norm(dim=(0, 2)) / ref.norm(dim=(0, 2)) for v in (got.cpu().double(), mod)]
    assert (errors[0] <= 1.3 * errors[1].max() + 1e-3).all(), errors  # at each step


@pytest.mark.gpu
def test_generate_sampling_seeds_and_types():
    m = _model(heads=2, layers=2, vocab=101, block=24).cuda()
    X = torch.randint(0, 101, (2, 20), generator=torch.Generator().manual_seed(2)).cuda()
    torch.manual_seed(3)
    out = m.generate(X, 12, temperature=0.9, top_k=7)
    torch.manual_seed(3)
    again = m.generate(X, 12, temperature=0.9, top_k=7)
    assert out.shape == (2, 32) and out.dtype == torch.int64 and torch.equal(out, again)
    handle = m.register_forward_hook(lambda *a: None)  # the general path draws the same numbers
    torch.manual_seed(3)
    want = m.generate(X, 12, temperature=0.9, top_k=7)
    handle.remove()
    # the same until a near-tie falls the other way after rounding, and no two tokens agree by chance (1 in 7)
    assert (out[:, 20:24] == want[:, 20:24]).float().mean() >= 0.5 and want.dtype == out.dtype
    g = torch.Generator("cuda").manual_seed(4)
    assert m.generate(X.int(), 2, generator=g).shape == (2, 22) and m.generate(X, 0) is X


@pytest.mark.gpu
def test_generate_where_the_kernel_does_not_fit(monkeypatch):
    m = _model().cuda()
    X = torch.zeros(2, 3, dtype=torch.int64, device="cuda")
    assert decode.supports(m, X)
    want = m.generate(X, 4, top_k=1)
    monkeypatch.setattr(decode, "_fns", {**decode._fns, "z2h_decode_epochs": lambda n, C, layers: 0})
    assert not decode.supports(m, X)
    assert torch.equal(m.generate(X, 4, top_k=1), want)


@pytest.mark.gpu
def test_status_word_made_by_generate_can_be_reset_outside(monkeypatch):
    from zero_to_hero_b200.ops import _lib

    monkeypatch.setattr(_lib, "_status", {})
    _model().cuda().generate(torch.zeros(1, 1, dtype=torch.int64, device="cuda"), 1)
    _lib.status_word("cuda").fill_(6)
    with pytest.raises(RuntimeError, match="timeout in an intra-CTA wait"):
        _lib.check_status("cuda")
    _lib.check_status("cuda")


@pytest.mark.gpu
def test_generate_raises_what_a_kernel_reported():
    from zero_to_hero_b200.ops import _lib

    m = _model().cuda()
    X = torch.zeros(2, 3, dtype=torch.int64, device="cuda")
    _lib.check_status("cuda")
    want = m.generate(X, 4, top_k=1)
    _lib.status_word("cuda").fill_(6)  # what an expired wait leaves
    with pytest.raises(RuntimeError, match="timeout in an intra-CTA wait"):
        m.generate(X, 4, top_k=1)
    assert torch.equal(m.generate(X, 4, top_k=1), want)
    with pytest.raises(RuntimeError, match="bad argument"):
        m.generate(X + 101, 4, top_k=1)  # one past the vocabulary: clamped, and reported
    _lib.check_status("cuda")


# the top-k select: values that crowd into one first digit, ties, both signs of zero, -inf, one row in
# shared memory and one too long for it
@pytest.mark.gpu
@pytest.mark.parametrize("V", (1, 33, 1000, 50257, 56320, 56321))
def test_top_k_keeps_what_the_sort_keeps(V):
    from zero_to_hero_b200.ops.sampling import sample_next, sample_topk_native

    g = torch.Generator().manual_seed(V)
    rows = torch.stack((torch.randn(V, generator=g), 3 + 0.01 * torch.randn(V, generator=g), -100 - torch.rand(V, generator=g),
                        torch.randint(-2, 3, (V,), generator=g) * 1.0, torch.full((V,), -torch.inf)))
    rows[3][rows[3] == 0] *= torch.randint(0, 2, (int((rows[3] == 0).sum()),), generator=g) * 2.0 - 1.0  # +-0.0
    rows[4, V // 2] = -3.0
    positive = int((rows[3] > 0).sum())  # the next one is a zero
    for k in (1, 2, 7, positive, positive + 1, V - 1, V, None):
        if k is not None and not 0 < k <= V:
            continue
        n = 256
        many = rows.cuda().repeat(n, 1)
        column = torch.zeros(many.shape[0], 3, dtype=torch.int64, device="cuda")
        ids = sample_topk_native(many, 1.0, k, seed=5, out=column[:, 1])
        assert torch.equal(ids[:, 0], column[:, 1]) and not column[:, (0, 2)].any()
        assert torch.equal(ids, sample_topk_native(many, 1.0, k, seed=5))
        low = rows.topk(k if k else V).values[:, -1].repeat(n)
        picked = many.gather(1, ids).squeeze(1).cpu()
        assert (picked >= low).all() and (picked > -torch.inf).all()
        if k == 1:
            assert torch.equal(picked, low)
        # At a temperature that makes all kept logits alike, many draws meet every value that is kept (a value among
        # n of them is missed with (1 - 1/n)^draws, 1e-13 at most here), and both zeros once zero is.
        ids = sample_topk_native(many, 1e6, k, seed=6).view(n, 5).cpu()
        for r, row in enumerate(rows):
            drawn = row[ids[:, r]]
            kept = row[(row >= row.topk(k if k else V).values[-1]) & (row > -torch.inf)].unique()
            assert drawn.min() >= kept.min()
            if len(kept) <= 8:
                assert torch.equal(drawn.unique(), kept), (k, r)
            if V >= 1000 and r == 3 and (drawn == 0).any():
                assert len(torch.signbit(drawn[drawn == 0]).unique()) == 2
    assert sample_next(rows[:2].cuda(), out=column[:2, 0]).shape == (2, 1)
