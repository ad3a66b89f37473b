"""The feed-forward of fp32 models, whatever planes the activations between its products have: widths that only one of its products takes as fp16 planes, and
inputs that bring none along, against plain PyTorch in fp64. The memory that the framework hands out again holds large values from a pass before.
"""
import copy

import pytest
import torch

import turbotransformers_b200 as tt
from turbotransformers_b200 import synthetic
from turbotransformers_b200.layers.utils import convert2tt_tensor

pytestmark = pytest.mark.gpu
torch.set_grad_enabled(False)
DEV = torch.device("cuda:0")


def err(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def bert(layers=2, **config):
    from transformers.models.bert.modeling_bert import BertModel
    cfg = synthetic.bert_config("bert-mini", layers)
    for k, v in dict(config, hidden_act="gelu_new", _attn_implementation="eager").items():
        setattr(cfg, k, v)
    return synthetic.reinit_(BertModel(cfg).eval(), 1).to(DEV)


# (tolerance: sums in fp32 of up to 1028 terms, 1e-8 of the result a term in the tensor cores' accumulator, through two layers)
TOLERANCE = 2e-5


@pytest.mark.parametrize("inner", [1024, 1028, 1026])
@pytest.mark.parametrize("batch,seq", [(1, 9), (3, 100)])
def test_inner_widths(built, inner, batch, seq):
    hf = bert(intermediate_size=inner)
    model = tt.BertModel.from_torch(hf, DEV)
    ids = torch.randint(0, hf.config.vocab_size, (batch, seq), generator=torch.Generator().manual_seed(1)).to(DEV)
    want = copy.deepcopy(hf).double()(ids)[0]
    loud = copy.deepcopy(hf)  # the same pass with activations of 1e8
    for layer in loud.encoder.layer:
        layer.attention.output.LayerNorm.weight.mul_(1e8)
        layer.output.LayerNorm.weight.mul_(1e8)
    loud = tt.BertModel.from_torch(loud, DEV)
    for _ in range(3):
        loud(ids)
        assert err(model(ids)[0], want) < TOLERANCE


def test_an_input_without_planes(built):
    """As after a caller's own attention class, which returns a tensor of its own making."""
    from turbotransformers_b200._cxx import cxx
    layer = bert(1).encoder.layer[0]
    inter, out = tt.BertIntermediate.from_torch(layer.intermediate), tt.BertOutput.from_torch(layer.output)
    x = torch.randn(2, 70, 256, generator=torch.Generator(device=DEV).manual_seed(3), device=DEV)
    double = copy.deepcopy(layer).double()
    want = double.output(double.intermediate(x.double()), x.double())
    for _ in range(3):
        results = []
        for y in (1e8 * x, x):
            y, inner = convert2tt_tensor(y), cxx.Tensor.create_empty()
            inter.for_output(y, inner)
            results.append(out(inner, y))
        assert err(results[1], want) < TOLERANCE
