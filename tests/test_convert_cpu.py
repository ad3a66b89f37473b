"""Runtime tensors made from torch tensors keep the memory and the shape that they were made with, whatever is done to the torch tensor afterwards."""
import gc

import pytest
import torch

from turbotransformers_b200._cxx import cxx
from turbotransformers_b200.layers.utils import convert2tt_tensor, lend, try_convert


def other_data(t):
    t.data = torch.zeros(40, 50)


@pytest.mark.parametrize("change", [lambda t: t.resize_(1, 2), lambda t: t.t_(), lambda t: t.unsqueeze_(0), lambda t: t.set_(torch.zeros(40, 50)), other_data],
                         ids=["resize_", "t_", "unsqueeze_", "set_", "data"])
@pytest.mark.parametrize("convert", [convert2tt_tensor, try_convert])
@pytest.mark.parametrize("grad", [False, True])
def test_keeps_its_shape_and_memory(change, convert, grad):
    want = torch.arange(6.0).reshape(2, 3)
    t = want.clone().requires_grad_(grad)
    kept = convert(t)
    if grad:
        t = t.detach()  # (a leaf that needs a gradient is changed in place through another object, which shares its memory)
    change(t)
    del t
    gc.collect()
    fill = [torch.full((2, 3), 7.0) for _ in range(64)]  # takes freed memory again
    assert [kept.shape(i) for i in range(kept.n_dim())] == [2, 3]
    assert (cxx.tensor2nparrayf(kept) == want.numpy()).all() and len(fill) == 64


def test_keeps_its_shape_where_the_memory_grows():
    """(The storage itself is another one then, which torch's own views of it see too.)"""
    t = torch.zeros(2, 3)
    kept = convert2tt_tensor(t)
    t.resize_(40, 50)
    assert [kept.shape(i) for i in range(kept.n_dim())] == [2, 3] and kept.numel() == 6


def test_lent_for_a_call():
    """For as long as the tensor is left alone the alias is that of try_convert, and what is no plain tensor goes the usual way."""
    t = torch.arange(6.0).reshape(2, 3)
    for given in (t, t.clone().requires_grad_(), torch.nn.Parameter(t.clone())):
        lent = lend(given)
        assert [lent.shape(i) for i in range(lent.n_dim())] == [2, 3] and (cxx.tensor2nparrayf(lent) == t.numpy()).all()
    assert lend(None) is None and lend(lent) is lent
