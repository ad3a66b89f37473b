"""The calls that run a stack of layers as one kernel (host/chain.cpp): the operations that it lists for encoders, decoder-only models and
decoders with context attention, against plain PyTorch in fp64 and against the layers called one by one, on both sides of the rule that
chooses the route. Widths start where the route does, at 512. Tolerances: whole fp16 models lie within 1.5e-3 of fp64 (2-norm over
2-norm: activations are rounded to 2^-11 some five times a layer); twice that is allowed, and a wrong operand gives 1e-1 and more.
"""
import math

import pytest
import torch

import turbotransformers_b200 as tt
from turbotransformers_b200._cxx import cxx
from turbotransformers_b200.graphs import CapturedForward

pytestmark = pytest.mark.gpu
torch.set_grad_enabled(False)
DEV = torch.device("cuda:0")
TOL = 3e-3


def weights(module, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    module = module.to(DEV).requires_grad_(False).eval().half()
    for name, p in module.named_parameters():
        scale = "norm" in name.lower() or "ln_" in name
        p.normal_(1.0 if scale and name.endswith("weight") else 0.0, 0.1 if scale else 0.03, generator=g)
    return module


def err(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def launches(fn):
    before = cxx.launch_count(0)
    out = fn()
    return out, cxx.launch_count(0) - before


def ids_of(vocab, *shape, seed=0):
    return torch.randint(2, vocab, shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)


# ---- encoders ------------------------------------------------------------------------------------------------------------
def bert(hidden, inner, layers, seed=1):
    from transformers.models.bert.modeling_bert import BertConfig, BertModel
    cfg = BertConfig(vocab_size=500, hidden_size=hidden, num_hidden_layers=layers, num_attention_heads=hidden // 64, intermediate_size=inner, hidden_act="gelu_new",
                     max_position_embeddings=128, hidden_dropout_prob=0.0, attention_probs_dropout_prob=0.0, layer_norm_eps=1e-12)
    hf = weights(BertModel(cfg), seed)
    return hf, tt.BertModel.from_torch(hf, DEV), weights(BertModel(cfg), seed).double()


@pytest.mark.parametrize("hidden,inner", [(512, 2048), (768, 3072), (1024, 4096)])
def test_encoder_on_both_sides_of_the_rule(hidden, inner):
    layers = 3
    hf, model, exact = bert(hidden, inner, layers)
    model(ids_of(500, 1, 4))  # weights are laid out in the first pass
    for B, L, masked in [(1, 1, 0), (1, 17, 0), (1, 24, 1), (3, 8, 1), (12, 2, 1), (2, 7, 0), (1, 25, 0), (5, 5, 1)]:
        ids = ids_of(500, B, L, seed=B * L)
        mask = None
        if masked:
            kept = torch.randint(1, L + 1, (B, ), generator=torch.Generator(device=DEV).manual_seed(L), device=DEV)
            mask = (torch.arange(L, device=DEV)[None] < kept[:, None]).long()
        (got, pooled), n = launches(lambda: model(ids, mask)[:2])
        assert (n < 10) if B * L <= 24 else (n >= 6 * layers), (B, L, n)
        want = exact(ids, mask)
        assert err(got, want[0]) < TOL and err(pooled, want[1]) < TOL
        if B * L <= 24:
            by_layer, n = launches(lambda: model(ids, mask, output_hidden_states=True)[0])
            assert n >= 6 * layers and err(got, by_layer) < TOL
    assert cxx.device_status(0) == 0


class LayerOfACaller(tt.BertLayer):
    calls = 0

    def __call__(self, *args, **kwargs):
        self.calls += 1
        return super().__call__(*args, **kwargs)


def test_encoder_with_a_layer_of_a_callers_class():
    hf, model, exact = bert(768, 3072, 2)
    ids = ids_of(500, 1, 9)
    want = model(ids)[0]
    model.bertmodel_nopooler.encoder.layer[1] = LayerOfACaller(model.bertmodel_nopooler.encoder.layer[1].attention, model.bertmodel_nopooler.encoder.layer[1].intermediate, model.bertmodel_nopooler.encoder.layer[1].output)
    got, n = launches(lambda: model(ids)[0])
    assert model.bertmodel_nopooler.encoder.layer[1].calls == 1 and n >= 12 and err(got, want) < TOL


def test_encoder_in_a_captured_graph_and_on_another_stream():
    hf, model, exact = bert(768, 3072, 3)
    ids = [ids_of(500, 1, 17, seed=s) for s in range(3)]
    eager = [model(i)[0].clone() for i in ids]
    replay = CapturedForward(lambda x: model(x)[0], ids[0].clone())
    for i, e in zip(ids + ids[:1], eager + eager[:1]):
        out = replay(i)
        torch.cuda.synchronize()
        assert torch.equal(out, e)
    replay.close()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for i, e in zip(ids, eager):
            assert torch.equal(model(i)[0], e)
    side.synchronize()
    assert torch.equal(model(ids[1])[0], eager[1]) and cxx.device_status(0) == 0


# ---- decoder-only models -------------------------------------------------------------------------------------------------
def gpt2(hidden, layers, seed=2, positions=256):
    from transformers import GPT2Config, GPT2Model
    cfg = GPT2Config(vocab_size=1003, n_positions=positions, n_embd=hidden, n_layer=layers, n_head=hidden // 64, resid_pdrop=0., embd_pdrop=0., attn_pdrop=0.)
    return tt.GPT2Model.from_torch(weights(GPT2Model(cfg), seed), DEV), weights(GPT2Model(cfg), seed).double()


@pytest.mark.parametrize("hidden", [512, 768, 1024])
@pytest.mark.parametrize("B,prompt", [(1, 3), (3, 7), (2, 12), (4, 30), (24, 1), (8, 15)])
def test_generation_across_both_routes_and_over_pages(hidden, B, prompt):
    """A prompt (by one kernel up to 24 rows), single tokens by one kernel past two page boundaries, three tokens at once layer by layer, single
    tokens again; logits contiguous, padded and none."""
    layers = 2
    model, exact = gpt2(hidden, layers)
    n_steps = 20
    ids = ids_of(1003, B, prompt + 2 * n_steps + 3, seed=B)
    want = exact(ids).last_hidden_state
    logits = want @ exact.wte.weight.T
    model(ids[:, :1].contiguous())  # weights are laid out in the first pass
    past, at = model.new_cache(), 0

    def feed(n, **kw):
        nonlocal at
        (hidden_states, lg), count = launches(lambda: model(ids[:, at:at + n].contiguous(), past=past, **kw))
        assert err(hidden_states, want[:, at:at + n]) < TOL, at
        if kw.get("return_logits", True):
            assert tuple(lg.shape) == (B, n, 1003) and err(lg, logits[:, at:at + n]) < TOL, at
        else:
            assert lg is None
        at += n
        assert model.cached_length(past) == at
        return count

    n = feed(prompt)
    assert (n <= 3) if B * prompt <= 24 else (n >= 6 * layers)
    for s in range(n_steps):
        assert feed(1, **({}, {"contiguous_logits": False}, {"return_logits": False})[s % 3]) <= 3
    assert feed(3) >= 6 * layers
    for s in range(n_steps):
        assert feed(1) <= 3
    if B * prompt <= 24:  # without a cache
        (hidden_states, lg), n = launches(lambda: model(ids[:, :prompt].contiguous()))
        assert n <= 3 and err(hidden_states, want[:, :prompt]) < TOL and err(lg, logits[:, :prompt]) < TOL
    assert cxx.device_status(0) == 0


def test_a_step_of_more_rows_goes_layer_by_layer_over_the_same_cache():
    model, exact = gpt2(768, 2)
    ids = ids_of(1003, 25, 6)
    want = exact(ids).last_hidden_state
    past = model.new_cache()
    for t in range(6):
        (got, _), n = launches(lambda: model(ids[:, t:t + 1].contiguous(), past=past))
        assert n >= 12 and err(got, want[:, t:t + 1]) < TOL


# ---- decoders with context attention ---------------------------------------------------------------------------------------
class Attention(torch.nn.Module):
    max_relative_positions = 0

    def __init__(self, H):
        super().__init__()
        self.head_count = H // 64
        self.linear_keys, self.linear_values, self.linear_query, self.final_linear = (torch.nn.Linear(H, H) for _ in range(4))


class FeedForward(torch.nn.Module):
    def __init__(self, H, F):
        super().__init__()
        self.w_1, self.w_2, self.layer_norm = torch.nn.Linear(H, F), torch.nn.Linear(F, H), torch.nn.LayerNorm(H, eps=1e-6)


class Layer(torch.nn.Module):
    def __init__(self, H, F):
        super().__init__()
        self.self_attn, self.context_attn, self.feed_forward = Attention(H), Attention(H), FeedForward(H, F)
        self.layer_norm_1, self.layer_norm_2 = torch.nn.LayerNorm(H, eps=1e-6), torch.nn.LayerNorm(H, eps=1e-6)


class Embeddings(torch.nn.Module):
    word_padding_idx = 1

    def __init__(self, H):
        super().__init__()
        self.table = torch.nn.Embedding(300, H)

    def forward(self, tgt, step=None):
        return self.table(tgt[:, :, 0])


class Stack(torch.nn.Module):
    def __init__(self, H, F, layers):
        super().__init__()
        self.embeddings, self.layer_norm = Embeddings(H), torch.nn.LayerNorm(H, eps=1e-6)
        self.transformer_layers = torch.nn.ModuleList([Layer(H, F) for _ in range(layers)])


def attend(a, q, k, v, seen):
    q, k, v = (t.unflatten(-1, (a.head_count, 64)).transpose(1, 2) for t in (a.linear_query(q), a.linear_keys(k), a.linear_values(v)))
    p = (q @ k.transpose(-1, -2) / 8.0).masked_fill(~seen, -math.inf).softmax(-1)
    return a.final_linear((p @ v).transpose(1, 2).flatten(2)), p[:, 0]


def decoded(m, targets, memory, lengths):
    """All steps at once in fp64: hidden [B, T, H] and the last layer's attention of head 0 [B, T, S]."""
    x, memory = m.embeddings(targets).transpose(0, 1), memory.double().transpose(0, 1)
    T, S = x.shape[1], memory.shape[1]
    before = torch.ones(T, T, dtype=torch.bool, device=DEV).tril()
    real = (torch.arange(S, device=DEV)[None] < lengths[:, None])[:, None, None]
    for l in m.transformer_layers:
        y = l.layer_norm_1(x)
        x = x + attend(l.self_attn, y, y, y, before)[0]
        c, p = attend(l.context_attn, l.layer_norm_2(x), memory, memory, real)
        x = x + c
        x = x + l.feed_forward.w_2(torch.relu(l.feed_forward.w_1(l.feed_forward.layer_norm(x))))
    return m.layer_norm(x), p


@pytest.mark.parametrize("H,F,B,S,chained", [(512, 2048, 1, 1, 1), (512, 2048, 20, 45, 1), (512, 2048, 64, 37, 1), (512, 1024, 65, 9, 0), (768, 3072, 17, 200, 1),
                                             (1024, 4096, 32, 20, 1), (1024, 4096, 33, 20, 0)])
def test_translation_steps(H, F, B, S, chained):
    layers, T = 2, 19
    dec, exact = tt.TransformerDecoder.from_onmt(weights(Stack(H, F, layers), 3), DEV), weights(Stack(H, F, layers), 3).double()
    g = torch.Generator(device=DEV).manual_seed(B)
    memory, targets = torch.randn(S, B, H, generator=g, device=DEV).half(), ids_of(300, T, B, 1, seed=B)
    lengths = torch.randint(1, S + 1, (B, ), generator=g, device=DEV)
    hidden, attention = decoded(exact, targets, memory, lengths)
    dec.init_state(torch.zeros(S, B, 1), memory, None)
    dec(targets[:1], memory, step=0, memory_lengths=lengths)  # weights are laid out in the first pass; step 0 starts anew
    for t in range(T):
        if t == 5:  # a half-filled memory cache is replaced as a pair
            cache = dec.state["cache"]["layer_1"]
            cache["memory_keys"], kept = None, cache["memory_values"].clone()
            cache["memory_values"] = torch.zeros_like(kept)
        (out, attns), n = launches(lambda: dec(targets[t:t + 1], memory, step=t, memory_lengths=lengths))
        projected = 2 * layers if t == 0 else (2 if t == 5 else 0)  # products of the memory, a transpose behind each
        assert (n == 1 + 2 * projected) if chained else (n >= 10 * layers), (t, n)
        assert tuple(out.shape) == (1, B, H) and err(out[0], hidden[:, t]) < TOL, t
        assert tuple(attns["std"].shape) == (1, B, S) and err(attns["std"][0], attention[:, t]) < TOL, t
        if t == 5:
            assert torch.equal(dec.state["cache"]["layer_1"]["memory_values"], kept)
    assert dec.state["cache"]["layer_0"]["self_keys"].shape(0) == T
    assert cxx.device_status(0) == 0


def test_translation_step_on_another_stream_and_by_layers_of_a_callers_class():
    H, F, B, S = 512, 2048, 5, 12
    modules = weights(Stack(H, F, 2), 3)
    memory, targets, lengths = torch.randn(S, B, H, device=DEV).half(), ids_of(300, 6, B, 1), torch.tensor([12, 3, 7, 1, 9], device=DEV)
    runs = []
    for how in ("here", "side", "caller"):
        dec = tt.TransformerDecoder.from_onmt(modules, DEV)
        if how == "caller":
            class Caller(tt.TransformerDecoderLayer):
                def __call__(self, *args, **kwargs):
                    return super().__call__(*args, **kwargs)
            dec.transformer_layers = [Caller(l.self_attn, l.context_attn, l.feed_forward) for l in dec.transformer_layers]
        dec.init_state(torch.zeros(S, B, 1), memory, None)
        stream = torch.cuda.Stream() if how == "side" else torch.cuda.current_stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            runs.append([dec(targets[t:t + 1], memory, step=t, memory_lengths=lengths) for t in range(6)])
        stream.synchronize()
    for here, side, caller in zip(*runs):
        assert torch.equal(here[0], side[0]) and torch.equal(here[1]["std"], side[1]["std"])
        assert err(here[0], caller[0]) < TOL and err(here[1]["std"], caller[1]["std"]) < TOL


# ---- calls that the route does not take ------------------------------------------------------------------------------------
@pytest.mark.parametrize("H,F,B,S", [(1024, 4096, 33, 20), (512, 2048, 65, 9), (512, 2048, 64, 700)])
def test_a_step_outside_the_rule_costs_no_list_of_operations(monkeypatch, H, F, B, S):
    """The rule is asked before parts and caches of every layer are gathered and converted (65 us a step of six layers)."""
    dec = tt.TransformerDecoder.from_onmt(weights(Stack(H, F, 2), 3), DEV)
    memory, lengths = torch.randn(S, B, H, device=DEV).half(), torch.full((B, ), S, device=DEV)
    dec.init_state(torch.zeros(S, B, 1), memory, None)
    monkeypatch.setattr(cxx, "decoder_chain", lambda *a: pytest.fail("gathered"))
    for t in range(2):
        out, n = launches(lambda: dec(ids_of(300, 1, B, 1), memory, step=t, memory_lengths=lengths))
        assert n >= 20 and torch.isfinite(out[0]).all()


def test_a_call_of_more_rows_costs_no_list_of_operations(monkeypatch):
    monkeypatch.setattr(cxx, "decoder_chain", lambda *a: pytest.fail("gathered"))
    monkeypatch.setattr(cxx, "encoder_chain", lambda *a: pytest.fail("gathered"))
    hf, model, exact = bert(768, 3072, 2)
    assert torch.isfinite(model(ids_of(500, 1, 25))[0]).all()
    model, exact = gpt2(768, 2)
    assert torch.isfinite(model(ids_of(1003, 1, 25))[0]).all()


def test_a_long_history_goes_layer_by_layer():
    model, exact = gpt2(512, 2, positions=1400)
    ids = ids_of(1003, 20, 1201, seed=4)
    past = model.new_cache()
    model(ids[:, :1180].contiguous(), return_logits=False, past=past)
    for t in range(1180, 1201):  # twenty rows of eight heads are two to a CTA: up to 1190 tokens in the cache
        (got, _), n = launches(lambda: model(ids[:, t:t + 1].contiguous(), past=past))
        assert (n <= 3) if t <= 1190 else (n >= 12), t
    assert err(got, exact(ids).last_hidden_state[:, -1:]) < TOL


# ---- calls that the route does not take ------------------------------------------------------------------------------------
@pytest.mark.parametrize("H,F,B,S", [(1024, 4096, 33, 20), (512, 2048, 65, 9), (512, 2048, 64, 700)])
def test_a_step_outside_the_rule_costs_no_list_of_operations(monkeypatch, H, F, B, S):
    """The rule is asked before parts and caches of every layer are gathered and converted (65 us a step of six layers)."""
    dec = tt.TransformerDecoder.from_onmt(weights(Stack(H, F, 2), 3), DEV)
    memory, lengths = torch.randn(S, B, H, device=DEV).half(), torch.full((B, ), S, device=DEV)
    dec.init_state(torch.zeros(S, B, 1), memory, None)
    monkeypatch.setattr(cxx, "decoder_chain", lambda *a: pytest.fail("gathered"))
    for t in range(2):
        out, n = launches(lambda: dec(ids_of(300, 1, B, 1), memory, step=t, memory_lengths=lengths))
        assert n >= 20 and torch.isfinite(out[0]).all()


def test_a_call_of_more_rows_costs_no_list_of_operations(monkeypatch):
    monkeypatch.setattr(cxx, "decoder_chain", lambda *a: pytest.fail("gathered"))
    monkeypatch.setattr(cxx, "encoder_chain", lambda *a: pytest.fail("gathered"))
    hf, model, exact = bert(768, 3072, 2)
    assert torch.isfinite(model(ids_of(500, 1, 25))[0]).all()
    model, exact = gpt2(768, 2)
    assert torch.isfinite(model(ids_of(1003, 1, 25))[0]).all()


def test_a_long_history_goes_layer_by_layer():
    model, exact = gpt2(512, 2, positions=1400)
    ids = ids_of(1003, 20, 1201, seed=4)
    past = model.new_cache()
    model(ids[:, :1180].contiguous(), return_logits=False, past=past)
    for t in range(1180, 1201):  # twenty rows of eight heads are two to a CTA: up to 1190 tokens in the cache
        (got, _), n = launches(lambda: model(ids[:, t:t + 1].contiguous(), past=past))
        assert (n <= 3) if t <= 1190 else (n >= 12), t
    assert err(got, exact(ids).last_hidden_state[:, -1:]) < TOL
