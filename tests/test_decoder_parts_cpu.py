"""CPU: which route TransformerDecoder takes through its layers, with parts that record what they are given. No kernel runs."""
import pytest
import torch

import turbotransformers_b200 as tt
from turbotransformers_b200.layers import modeling_decoder
from turbotransformers_b200.layers.return_type import ReturnType, convert_returns_as_type
from turbotransformers_b200.layers.utils import convert2tt_tensor

B, T, S, H, HEADS = 2, 3, 4, 8, 2


class Embeddings:
    word_padding_idx = 1

    def __call__(self, tgt, step=None):
        return torch.ones(tgt.shape[0], tgt.shape[1], H)


class OwnAttention(tt.MultiHeadedAttention):
    """A caller's attention: a torch user's code, which gets what it always got."""

    def __call__(self, key, value, query, mask=None, layer_cache=None, attn_type=None, return_type=None, **_):
        self.seen.append((attn_type, key, query, mask))
        q = query if isinstance(query, torch.Tensor) else convert_returns_as_type(query, ReturnType.TORCH)
        return convert2tt_tensor(q.clone()), convert2tt_tensor(torch.ones(B, HEADS, T, S))


class OwnFeedForward(tt.PositionwiseFeedForward):
    def __call__(self, x, return_type=None, is_trans_weight=True, output=None):
        self.seen.append(("ffn", x))
        return convert_returns_as_type(x, return_type)


def own(cls, seen):
    part = cls.__new__(cls)  # no weights: the framework's side of it is never called
    part.seen = seen
    return part


def make_layer(**parts):
    """A layer of the framework's class; parts that are not given are the framework's (and never run)."""
    layer = tt.TransformerDecoderLayer.__new__(tt.TransformerDecoderLayer)
    for name, cls in (("self_attn", tt.MultiHeadedAttention), ("context_attn", tt.MultiHeadedAttention), ("feed_forward", tt.PositionwiseFeedForward)):
        setattr(layer, name, parts.get(name) or cls.__new__(cls))
    return layer


def decode(layers, norm=None):
    dec = tt.TransformerDecoder(Embeddings(), layers, norm or torch.nn.LayerNorm(H))
    dec.init_state(torch.zeros(S, B, 1), None, None)
    return dec(torch.zeros(T, B, 1, dtype=torch.int64), torch.ones(S, B, H), memory_lengths=torch.tensor([S, S - 1]))


def test_a_callers_own_parts_get_torch_tensors():
    seen = []
    out, attns = decode([make_layer(self_attn=own(OwnAttention, seen), context_attn=own(OwnAttention, seen), feed_forward=own(OwnFeedForward, seen))
                         for _ in range(2)])
    assert tuple(out.shape) == (T, B, H) and tuple(attns["std"].shape) == (T, B, S)
    calls = [s for s in seen if s[0] in ("self", "context")]
    assert [s[0] for s in calls] == ["self", "context"] * 2
    for kind, key, query, mask in calls:
        assert isinstance(key, torch.Tensor) and isinstance(mask, torch.Tensor)
        assert kind == "context" or isinstance(query, torch.Tensor)  # the context attention's query always was the runtime's tensor


@pytest.mark.parametrize("part,cls", [("self_attn", OwnAttention), ("context_attn", OwnAttention), ("feed_forward", OwnFeedForward)])
def test_one_part_of_the_callers_is_enough(part, cls):
    assert modeling_decoder._unmodified(make_layer())
    assert not modeling_decoder._unmodified(make_layer(**{part: own(cls, [])}))


def test_the_runtime_is_back_on_the_callers_stream_before_torch_reads_the_results(monkeypatch):
    # Another thread may point the device's kernel stream elsewhere between two layers; pointing it back orders the caller's
    # stream behind what was queued meanwhile.
    log = []

    def run(self, x, memory, src_mask, dec_mask, layer_cache, return_type, output=None):
        log.append("layer")
        return convert_returns_as_type(convert2tt_tensor(torch.ones(B, T, H)), return_type), convert2tt_tensor(torch.ones(B, HEADS, T, S))

    class Norm(torch.nn.LayerNorm):
        def forward(self, x):
            log.append("torch")
            return super().forward(x)

    monkeypatch.setattr(tt.TransformerDecoderLayer, "_run", run)
    monkeypatch.setattr(modeling_decoder, "use_current_stream", lambda t: log.append("stream"))
    decode([make_layer(), make_layer()], Norm(H))
    assert log == ["layer", "layer", "stream", "torch"]
