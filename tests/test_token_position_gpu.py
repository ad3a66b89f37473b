"""Token plus position embedding in one kernel: bit for bit the two lookups that it takes the place of, ids outside the table included."""
import pytest
import torch

from turbotransformers_b200 import _capi

pytestmark = pytest.mark.gpu
torch.set_grad_enabled(False)
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("dt,code", [(torch.float16, _capi.F16), (torch.bfloat16, _capi.BF16), (torch.float32, _capi.F32)])
@pytest.mark.parametrize("B,L,H,offset", [(1, 1, 768, 0), (3, 17, 768, 5), (64, 1, 512, 40), (2, 300, 72, 0), (5, 7, 67, 3)])
def test_equals_two_lookups(ctx, dt, code, B, L, H, offset):
    g = torch.Generator(device=DEV).manual_seed(B * L)
    vocab = 97
    token, position = (torch.randn(n, H, generator=g, device=DEV).to(dt) for n in (vocab, offset + L))
    ids = torch.randint(0, vocab, (B, L), generator=g, device=DEV)
    ids[-1, -1] = vocab  # clamped and flagged
    places = torch.arange(offset, offset + L, device=DEV).repeat(B)
    want, got = torch.empty(B * L, H, device=DEV, dtype=dt), torch.empty(B * L, H, device=DEV, dtype=dt)
    ctx.call("lookup_embedding", code, want, token, ids, B * L, H, vocab, 0)
    ctx.call("lookup_embedding", code, want, position, places, B * L, H, offset + L, 1)
    assert ctx.device_status() == _capi.ERR_BAD_INDEX
    ctx.call("token_position_embedding", code, got, token, position[offset:], ids, B, L, H, vocab)
    assert ctx.device_status() == _capi.ERR_BAD_INDEX
    assert torch.equal(got, want)
