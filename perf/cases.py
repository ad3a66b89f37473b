"""The work that users of this framework have it do, as cases that a timing harness can run: encoder requests from one short
sentence to full batches, packed variable-length batches, causal language model forward passes, token-by-token generation
over a key/value cache and stepwise translation decoding, in the data types that the models are served in.

    listed()             the cases by name
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  the model and the inputs, on the GPU, from the seed
    run(state)           one pass through the public entry points
    exact(case, seed)    what that pass computes, in 64 bits and plain torch
    work(case)           the bytes and floating-point operations that one pass cannot do without
    tolerance(case)      how far two correct implementations at the case's precision may differ
"""
import copy
import functools
import math
import random

import torch

import turbotransformers_b200 as tt
from turbotransformers_b200 import synthetic

DEVICE = torch.device("cuda:0")
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "int8": torch.float16}

# The decoder of the usual translation model ("transformer base" sizes).
NMT = {"layers": 6, "hidden": 512, "heads": 8, "ffn": 2048, "vocab": 32000}


def listed():
    return [
        # One short query, the smallest call that a service sees: latency, all launches.
        {"name": "bert_f16_b1_s17", "kind": "bert", "model": "bert-base", "dtype": "f16", "batch": 1, "seq": 17, "masked": False},
        # One request of the usual benchmark length in the data type that a HuggingFace model comes in.
        {"name": "bert_f32_b1_s128", "kind": "bert", "model": "bert-base", "dtype": "f32", "batch": 1, "seq": 128, "masked": False},
        # A handful of requests padded to the longest (an odd length) with an attention mask.
        {"name": "bert_f16_b8_s99_mask", "kind": "bert", "model": "bert-base", "dtype": "f16", "batch": 8, "seq": 99, "masked": True},
        # A masked batch of a bfloat16 model.
        {"name": "bert_bf16_b16_s200_mask", "kind": "bert", "model": "bert-base", "dtype": "bf16", "batch": 16, "seq": 200, "masked": True},
        # The int8 model at its middle benchmark point.
        {"name": "bert_int8_b16_s128", "kind": "bert", "model": "bert-base", "dtype": "int8", "batch": 16, "seq": 128, "masked": False},
        # Serving throughput: 64 requests of 8 to 512 tokens, packed without padding (the headline benchmark).
        {"name": "packed_f16_b64_8to512", "kind": "packed", "model": "bert-base", "dtype": "f16", "batch": 64, "low": 8, "high": 512},
        # A small ragged batch in fp32.
        {"name": "packed_f32_b8_10to120", "kind": "packed", "model": "bert-base", "dtype": "f32", "batch": 8, "low": 10, "high": 120},
        # The largest encoder batch: one GPU's share of 256 sequences of 512.
        {"name": "large_f16_b32_s512", "kind": "bert", "model": "bert-large", "dtype": "f16", "batch": 32, "seq": 512, "masked": False},
        # Language model scoring: hidden states and logits of whole sequences.
        {"name": "gpt2_f16_b8_s1024", "kind": "gpt2", "model": "gpt2-small", "dtype": "f16", "batch": 8, "seq": 1024},
        # Generation for one user: a short prompt, then token by token.
        {"name": "generate_f16_b1_p64_n24", "kind": "generate", "model": "gpt2-small", "dtype": "f16", "batch": 1, "prompt": 64, "steps": 24},
        # Generation for a full batch with a longer history.
        {"name": "generate_f16_b32_p300_n16", "kind": "generate", "model": "gpt2-small", "dtype": "f16", "batch": 32, "prompt": 300, "steps": 16},
        # Translation: target tokens one after the other over an encoder memory, a batch of beams.
        {"name": "nmt_f16_b20_src45_n10", "kind": "nmt", "dtype": "f16", "batch": 20, "source": 45, "steps": 10},
    ]


def _spread(rng, low, high):
    """A whole number from [low, high], uniform over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


# The most tokens of a drawn encoder batch: what the largest listed cases cost, in each data type's time per token.
MOST_TOKENS = {"f16": 16384, "int8": 16384, "bf16": 10240, "f32": 3072}


def draw(rng):
    kind = rng.choice(["bert", "bert", "bert", "packed", "packed", "gpt2", "generate", "generate", "nmt"])
    if kind == "bert":
        dtype = rng.choice(["f16", "f16", "f32", "bf16", "int8"])
        model = "bert-large" if dtype == "f16" and rng.random() < 0.25 else "bert-base"
        seq = _spread(rng, 8, 512)
        most = MOST_TOKENS[dtype] // seq
        return {"kind": kind, "model": model, "dtype": dtype, "batch": _spread(rng, 1, max(1, min(64, most))), "seq": seq,
                "masked": rng.random() < 0.5}
    if kind == "packed":
        dtype = rng.choice(["f16", "f16", "f32", "bf16"])
        low, high = sorted((_spread(rng, 4, 512), _spread(rng, 4, 512)))
        most = MOST_TOKENS[dtype] * 2 // (low + high)
        return {"kind": kind, "model": "bert-base", "dtype": dtype, "batch": _spread(rng, 1, max(1, min(64, most))), "low": low, "high": high}
    if kind == "gpt2":
        seq = _spread(rng, 16, 1024)
        return {"kind": kind, "model": "gpt2-small", "dtype": rng.choice(["f16", "f16", "bf16"]), "batch": _spread(rng, 1, max(1, min(32, 6144 // seq))), "seq": seq}
    if kind == "generate":
        prompt = _spread(rng, 8, 600)
        return {"kind": kind, "model": "gpt2-small", "dtype": "f16", "batch": _spread(rng, 1, max(1, min(64, 8192 // prompt))), "prompt": prompt,
                "steps": rng.randint(4, 16)}
    return {"kind": kind, "dtype": "f16", "batch": _spread(rng, 1, 64), "source": _spread(rng, 6, 200), "steps": rng.randint(3, 10)}


# ---------------------------------------------------------------------------------------------------
# models: the modules that the framework's from_torch / from_onmt loaders take, with weights from the seed
# ---------------------------------------------------------------------------------------------------
@functools.cache
def _skeleton(name):
    """The torch module of a named configuration, without storage."""
    make = synthetic.make_hf_gpt2 if name.startswith("gpt2") else synthetic.make_hf_bert
    return make(name).to("meta")


class _Attention(torch.nn.Module):
    max_relative_positions = 0

    def __init__(self):
        super().__init__()
        self.head_count, H = NMT["heads"], NMT["hidden"]
        self.linear_keys, self.linear_values = torch.nn.Linear(H, H), torch.nn.Linear(H, H)
        self.linear_query, self.final_linear = torch.nn.Linear(H, H), torch.nn.Linear(H, H)


class _FeedForward(torch.nn.Module):
    def __init__(self):
        super().__init__()
        self.w_1, self.w_2 = torch.nn.Linear(NMT["hidden"], NMT["ffn"]), torch.nn.Linear(NMT["ffn"], NMT["hidden"])
        self.layer_norm = torch.nn.LayerNorm(NMT["hidden"], eps=1e-6)


class _DecoderLayer(torch.nn.Module):
    def __init__(self):
        super().__init__()
        self.self_attn, self.context_attn, self.feed_forward = _Attention(), _Attention(), _FeedForward()
        self.layer_norm_1 = torch.nn.LayerNorm(NMT["hidden"], eps=1e-6)
        self.layer_norm_2 = torch.nn.LayerNorm(NMT["hidden"], eps=1e-6)


class _Embeddings(torch.nn.Module):
    word_padding_idx = 1

    def __init__(self):
        super().__init__()
        self.table = torch.nn.Embedding(NMT["vocab"], NMT["hidden"])

    def forward(self, tgt, step=None):
        return self.table(tgt[:, :, 0])


class _DecoderStack(torch.nn.Module):
    """Laid out like OpenNMT-py's transformer decoder."""

    def __init__(self):
        super().__init__()
        self.embeddings = _Embeddings()
        self.transformer_layers = torch.nn.ModuleList([_DecoderLayer() for _ in range(NMT["layers"])])
        self.layer_norm = torch.nn.LayerNorm(NMT["hidden"], eps=1e-6)


def _weights(module, generator, dtype):
    """`module` on the GPU: matrices, embeddings and biases ~ N(0, 0.02), layer norms near (1, 0)."""
    module = module.to_empty(device=DEVICE).to(dtype).requires_grad_(False).eval()
    for name, p in module.named_parameters():
        norm = "norm" in name.lower() or "ln_" in name
        p.normal_(1.0 if norm and name.endswith("weight") else 0.0, 0.02, generator=generator)
    return module


def _lengths(count, low, high, seed):
    """`count` lengths spread evenly over [low, high], in an order that depends on the seed."""
    lens = [low + (high - low) * i // max(1, count - 1) for i in range(count)]
    random.Random(seed).shuffle(lens)
    return lens


def _mask_lengths(case, seed):
    """Kept lengths of a padded batch: a quarter of the longest up to the longest."""
    return _lengths(case["batch"], max(1, case["seq"] // 4), case["seq"], seed) if case["batch"] > 1 else [max(1, case["seq"] * 3 // 4)]


def _inputs(case, seed):
    """The torch module and the inputs of one pass."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    dtype, kind, B = DTYPES[case["dtype"]], case["kind"], case["batch"]
    if kind == "nmt":
        with torch.device("meta"):
            stack = _DecoderStack()
        S = case["source"]
        lens = torch.tensor(_lengths(B, max(1, S // 2), S, seed) if B > 1 else [S], device=DEVICE)
        return {"kind": kind, "torch_model": _weights(stack, g, dtype),
                "memory": torch.randn(S, B, NMT["hidden"], generator=g, device=DEVICE, dtype=dtype), "lengths": lens,
                "source": torch.randint(2, NMT["vocab"], (S, B, 1), generator=g, device=DEVICE),
                "targets": [torch.randint(2, NMT["vocab"], (1, B, 1), generator=g, device=DEVICE) for _ in range(case["steps"])]}
    torch_model = _weights(copy.deepcopy(_skeleton(case["model"])), g, dtype)
    vocab = torch_model.config.vocab_size
    # the torch module stays with the state: the framework's layers alias some of its tensors
    state = {"kind": kind, "torch_model": torch_model}
    if kind == "bert":
        state["mask"] = None
        if case["masked"]:
            kept = torch.tensor(_mask_lengths(case, seed), device=DEVICE)
            state["mask"] = (torch.arange(case["seq"], device=DEVICE)[None] < kept[:, None]).to(torch.int64)
        state["ids"] = torch.randint(0, vocab, (B, case["seq"]), generator=g, device=DEVICE)
    elif kind == "packed":
        state["lengths"] = _lengths(B, case["low"], case["high"], seed)
        state["ids"] = [torch.randint(0, vocab, (n,), generator=g, device=DEVICE) for n in state["lengths"]]
    elif kind == "gpt2":
        state["ids"] = torch.randint(0, vocab, (B, case["seq"]), generator=g, device=DEVICE)
    else:
        state["prompt"] = torch.randint(0, vocab, (B, case["prompt"]), generator=g, device=DEVICE)
        state["tokens"] = [torch.randint(0, vocab, (B, 1), generator=g, device=DEVICE) for _ in range(case["steps"])]
    return state


def prepare(case, seed):
    state = _inputs(case, seed)
    if state["kind"] == "nmt":
        state["model"] = tt.TransformerDecoder.from_onmt(state["torch_model"], DEVICE)
    else:
        loader = {"bert": tt.QBertModel if case["dtype"] == "int8" else tt.BertModel, "packed": tt.BertModelSmartBatch}.get(state["kind"], tt.GPT2Model)
        state["model"] = loader.from_torch(state["torch_model"], DEVICE)
    return state


def run(state):
    kind, model = state["kind"], state["model"]
    with torch.no_grad():
        if kind == "bert":
            sequence, pooled = model(state["ids"], state["mask"])[:2]
            return [sequence, pooled]
        if kind == "packed":
            sequence, pooled = model(state["ids"], state["lengths"])[:2]
            return [sequence, pooled]
        if kind == "gpt2":
            hidden, logits = model(state["ids"])
            return [hidden, logits]
        if kind == "generate":
            # The continuation is given (a scored or replayed one), so that the outputs do not hang on ties of an argmax.
            past = model.new_cache()
            model(state["prompt"], return_logits=False, past=past)
            return [model(token, past=past)[1] for token in state["tokens"]]
        outs = []
        model.init_state(state["source"], state["memory"], None)
        for step, token in enumerate(state["targets"]):
            hidden, attention = model(token, state["memory"], step=step, memory_lengths=state["lengths"])
            outs += [hidden, attention["std"]]
        return outs


# ---------------------------------------------------------------------------------------------------
# the same passes in 64 bits
# ---------------------------------------------------------------------------------------------------
def _norm(x, ln):
    return torch.nn.functional.layer_norm(x, ln.normalized_shape, ln.weight, ln.bias, ln.eps)


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")  # the form that the framework documents for every model


def _attend(q, k, v, heads, keep=None):
    """Rows [B, L, H] and keys and values [B, S, H] -> context [B, L, H] and probabilities [B, heads, L, S]; keep: what is seen."""
    q, k, v = (t.unflatten(-1, (heads, -1)).transpose(1, 2) for t in (q, k, v))
    scores = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    probs = (scores if keep is None else scores.masked_fill(~keep, -math.inf)).softmax(-1)
    return (probs @ v).transpose(1, 2).flatten(2), probs


def _bert(m, ids, mask):
    e, keep = m.embeddings, None if mask is None else mask.bool()[:, None, None]
    x = e.word_embeddings(ids) + e.position_embeddings.weight[: ids.shape[1]] + e.token_type_embeddings.weight[0]
    x = _norm(x, e.LayerNorm)
    for layer in m.encoder.layer:
        a = layer.attention
        context, _ = _attend(a.self.query(x), a.self.key(x), a.self.value(x), m.config.num_attention_heads, keep)
        x = _norm(x + a.output.dense(context), a.output.LayerNorm)
        x = _norm(x + layer.output.dense(_gelu(layer.intermediate.dense(x))), layer.output.LayerNorm)
    return x, torch.tanh(m.pooler.dense(x[:, 0]))


def _gpt2(m, ids):
    L = ids.shape[1]
    x = m.wte(ids) + m.wpe.weight[:L]
    seen = torch.ones(L, L, dtype=torch.bool, device=DEVICE).tril()
    for b in m.h:
        q, k, v = (_norm(x, b.ln_1) @ b.attn.c_attn.weight + b.attn.c_attn.bias).chunk(3, -1)
        x = x + _attend(q, k, v, m.config.n_head, seen)[0] @ b.attn.c_proj.weight + b.attn.c_proj.bias
        x = x + _gelu(_norm(x, b.ln_2) @ b.mlp.c_fc.weight + b.mlp.c_fc.bias) @ b.mlp.c_proj.weight + b.mlp.c_proj.bias
    return _norm(x, m.ln_f)


def exact(case, seed):
    """The int8 models are compared with their unquantised weights: what is left is then mostly the quantisation."""
    s = _inputs(case, seed)
    kind, m = s["kind"], s["torch_model"].double()
    with torch.no_grad():
        if kind == "bert":
            return list(_bert(m, s["ids"], s["mask"]))
        if kind == "packed":
            each = [_bert(m, ids[None], None) for ids in s["ids"]]
            return [torch.cat([x for x, _ in each], 1), torch.cat([p for _, p in each], 0)]
        if kind == "gpt2":
            hidden = _gpt2(m, s["ids"])
            return [hidden, hidden @ m.wte.weight.T]
        if kind == "generate":
            hidden = _gpt2(m, torch.cat([s["prompt"]] + s["tokens"], 1))[:, case["prompt"]:]
            return [hidden[:, t: t + 1] @ m.wte.weight.T for t in range(case["steps"])]
        # All steps at once, each row seeing the steps before it.
        memory, T = s["memory"].double().transpose(0, 1), case["steps"]
        x = m.embeddings(torch.cat(s["targets"])).transpose(0, 1)
        seen = torch.ones(T, T, dtype=torch.bool, device=DEVICE).tril()
        real = (torch.arange(case["source"], device=DEVICE)[None] < s["lengths"][:, None])[:, None, None]
        for layer in m.transformer_layers:
            a, f, y = layer.self_attn, layer.feed_forward, _norm(x, layer.layer_norm_1)
            x = x + a.final_linear(_attend(a.linear_query(y), a.linear_keys(y), a.linear_values(y), a.head_count, seen)[0])
            a, y = layer.context_attn, _norm(x, layer.layer_norm_2)
            context, probs = _attend(a.linear_query(y), a.linear_keys(memory), a.linear_values(memory), a.head_count, real)
            x = x + a.final_linear(context)
            x = x + f.w_2(torch.relu(f.w_1(_norm(x, f.layer_norm))))
        hidden = _norm(x, m.layer_norm)
        return [out for t in range(T) for out in (hidden[:, t][None], probs[:, 0, t][None])]


# ---------------------------------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------------------------------
def work(case):
    kind, B = case["kind"], case["batch"]
    act = 4 if case["dtype"] == "f32" else 2
    weight = 1 if case["dtype"] == "int8" else act
    if kind == "nmt":
        # A step reads the layers' weights (the key and value projections of the memory only once), the cached keys and values
        # and the memory's, and writes a hidden row and the attention over the source.
        L, H, F, S, n = NMT["layers"], NMT["hidden"], NMT["ffn"], case["source"], case["steps"]
        step_w = L * (6 * H * H + 2 * H * F)
        flops = 2.0 * B * (n * step_w + L * 2 * H * H * S) + 4.0 * H * B * L * (n * S + n * (n + 1) / 2)
        moved = act * (n * step_w + L * 2 * H * H + S * B * H + n * L * 2 * B * S * H + L * 2 * B * H * n * (n + 1) / 2 + n * B * (2 * H + S))
        return {"bytes": moved, "flops": flops}
    if kind in ("gpt2", "generate"):
        L, H, _, V, _ = synthetic.GPT2_CONFIGS[case["model"]]
        body = L * 12 * H * H
        if kind == "gpt2":
            n = B * case["seq"]
            return {"bytes": act * (body + V * H + n * (2 * H + V)) + 8 * n,
                    "flops": 2.0 * n * (body + V * H) + 2.0 * B * L * H * case["seq"] * (case["seq"] + 1)}
        # Every step depends on the one before it and reads the weights and the cache anew.
        P, n = case["prompt"], case["steps"]
        seen = sum(P + t + 1 for t in range(n))
        flops = 2.0 * B * P * body + 2.0 * B * L * H * P * (P + 1) + 2.0 * B * n * (body + V * H) + 4.0 * B * L * H * seen
        moved = act * ((n + 1) * body + n * V * H + B * P * H + L * 2 * B * H * (P + seen) + n * B * (H + V))
        return {"bytes": moved, "flops": flops}
    L, H, _, F, _, _, _ = synthetic.CONFIGS[case["model"]]
    if kind == "packed":
        lens = _lengths(B, case["low"], case["high"], 0)
    else:
        lens = _mask_lengths(case, 0) if case["masked"] else [case["seq"]] * B
    n = B * case["seq"] if kind == "bert" else sum(lens)
    # a padded batch's hidden states are returned for the padding too; its keys beyond the kept length take no part
    attention = 4.0 * H * L * (sum(m * case["seq"] for m in lens) if kind == "bert" else sum(m * m for m in lens))
    body = L * (4 * H * H + 2 * H * F)
    return {"bytes": weight * body + act * (n * 2 * H + H * H + B * H) + 8 * n, "flops": 2.0 * n * body + 2.0 * B * H * H + attention}


def tolerance(case):
    """Relative differences of whole models. Each figure is about twice what the data type itself costs on these models against the
    same weights in fp32 (two correct implementations may each be that far off): fp16 rounds its activations to 2^-11 between some
    60 kernels, 1.3e-3; bf16 models keep two planes between layers and round their outputs to 2^-9, 2.6e-3; fp32 sums of up to
    3072 terms in another order, or as products of three tf32 pairs, 5e-5. int8: about one activation in a hundred lies within an
    fp16 rounding of the border between two quantisation steps (1/127 of its row's largest value) and may fall to either side,
    which is half the effect of the quantisation itself, 3e-2."""
    return {"rel": {"f32": 1e-4, "f16": 3e-3, "bf16": 6e-3, "int8": 1.5e-2}[case["dtype"]]}
