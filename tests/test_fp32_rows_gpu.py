"""fp32 layers: what a row of activations comes out as does not depend on how large or small other rows are, nor on how far a weight could take it at most.
Against plain PyTorch in fp64, with the tolerances that the layers have for rows by themselves.
"""
import copy

import pytest
import torch

import turbotransformers_b200 as tt
from turbotransformers_b200 import synthetic
from turbotransformers_b200._cxx import cxx
from turbotransformers_b200.layers.modeling_bert import feed_forward as feed_forward_of

pytestmark = pytest.mark.gpu
torch.set_grad_enabled(False)
DEV = torch.device("cuda:0")


def err(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def layer(bias=0.0):
    from transformers.models.bert.modeling_bert import BertLayer
    cfg = synthetic.bert_config("bert-mini", 1)
    cfg.hidden_act, cfg._attn_implementation = "gelu_new", "eager"
    layer = synthetic.reinit_(BertLayer(cfg).eval(), 1).to(DEV)
    for name, p in layer.named_parameters():
        if name.endswith("bias"):
            p.mul_(bias)
    return layer


def rows(L, seed=1):
    return torch.randn(1, L, 256, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)


def attention(block, x, mask=None):
    out = tt.BertAttention.from_torch(block.attention)(x, mask)[0]
    double = copy.deepcopy(block.attention).double()
    return out, double(x.double(), None if mask is None else mask.double())[0]


@pytest.mark.parametrize("size", [1.0, 1e-2, 1e-4])
@pytest.mark.parametrize("L", [2, 65, 300])
def test_a_row_of_zeros_among_small_ones(built, L, size):
    block, x = layer(), rows(L) * size
    x[0, L // 2] = 0
    out, want = attention(block, x)
    others = torch.arange(L, device=DEV) != L // 2
    assert err(out[:, others], want[:, others]) < 2e-6


@pytest.mark.parametrize("L", [9, 300])
def test_a_value_weight_that_meets_nothing(built, L):
    """The same as below of the attention's values and output."""
    block, x = layer(bias=1.0), rows(L)
    x[..., 7] = 0
    block.attention.self.value.weight[5] = 0
    block.attention.self.value.weight[5, 7] = 2.0 ** 24
    out, want = attention(block, x)
    assert err(out, want) < 2e-6


@pytest.mark.parametrize("size", [1e3, 1e9])
@pytest.mark.parametrize("L", [9, 300])
def test_a_row_that_no_other_sees(built, L, size):
    """Keys that the mask hides, as a batch's padding, however large what they hold."""
    block, x = layer(bias=1.0), rows(L)
    x[0, L // 2] *= size
    mask = torch.zeros(1, 1, 1, L, device=DEV)
    mask[..., L // 2] = -3e38
    out, want = attention(block, x, mask)
    others = torch.arange(L, device=DEV) != L // 2
    assert err(out[:, others], want[:, others]) < 2e-6


def feed_forward(block, x):
    """The layer's feed-forward behind its attention's output for x: as this framework runs it, and in 64 bits on the same attention output."""
    mine = tt.BertLayer.from_torch(block)
    y = mine.attention(x, return_type=tt.ReturnType.turbo_transformers)[0]
    exact = torch.from_numpy(cxx.tensor2nparrayf(y)).to(DEV).double().view(x.shape)
    double = copy.deepcopy(block).double()
    return feed_forward_of(mine.intermediate, mine.output, y, None), double.output(double.intermediate(exact), exact), mine


@pytest.mark.parametrize("L", [9, 300])
def test_a_weight_that_meets_nothing(built, L):
    """A weight of 2^24 whose activations are zeros could take the inner activation far, and takes it nowhere."""
    block = layer(bias=1.0)
    block.attention.output.LayerNorm.weight[7] = block.attention.output.LayerNorm.bias[7] = 0
    block.intermediate.dense.weight[5] = 0
    block.intermediate.dense.weight[5, 7] = 2.0 ** 24
    out, want, _ = feed_forward(block, rows(L))
    assert err(out, want) < 2e-6


def test_a_bias_that_is_changed_in_place(built):
    """The runtime reads the caller's bias where it is, at each pass."""
    block, x = layer(bias=1.0), rows(70)
    _, _, mine = feed_forward(block, x)
    block.intermediate.dense.bias.mul_(1e6)
    y = mine.attention(x, return_type=tt.ReturnType.turbo_transformers)[0]
    _, want, _ = feed_forward(block, x)
    assert err(feed_forward_of(mine.intermediate, mine.output, y, None), want) < 2e-6


@pytest.mark.parametrize("lens", [[17], [128], [513, 90]])
def test_attention_of_rows_and_dimensions_far_apart(ctx, lens):
    """Queries and keys whose dimensions are up to 2^16 apart and make up for one another, values whose rows and dimensions are. Every output is as close to its own
    terms as operands of 22 bits (of which scores of up to 5 make five times as much of a probability) and sums in fp32 leave it."""
    T, heads = sum(lens), 12
    H, g = heads * 64, torch.Generator(device=DEV).manual_seed(5)
    powers = lambda *shape: 2.0 ** torch.randint(-8, 9, shape, generator=g, device=DEV)
    qkv, dims = torch.randn(T, 3 * H, generator=g, device=DEV), powers(1, H)
    qkv[:, :H] *= dims
    qkv[:, H:2 * H] /= dims
    qkv[:, 2 * H:] *= powers(T, 1) * powers(1, H)
    cu, out = torch.tensor([0] + lens, device=DEV).cumsum(0).int(), torch.zeros(T, H, device=DEV)
    ctx.call("attention_f32", qkv, cu, len(lens), max(lens), heads, 64, None, 0, 0, 0, 0.125, out, None)
    for b, n in enumerate(lens):
        rows = slice(int(cu[b]), int(cu[b + 1]))
        q, k, v = (t.reshape(n, heads, 64).transpose(0, 1).double() for t in qkv[rows].split(H, 1))
        p = (q @ k.transpose(1, 2) / 8).softmax(-1)
        want, terms = ((p @ x).transpose(0, 1).reshape(n, H) for x in (v, v.abs()))
        assert float(((out[rows] - want).abs() / terms).max()) < 2e-6
