"""Tokens to heads and back where the kernel's groups can go wrong: heads of no whole group, pointers off the 16-byte boundary, rows of
one group and of more than a warp's 32, packed tokens with padding. Every element is one addition in fp32, rounded once: exact."""
import pytest
import torch

from tests.helpers import TORCH_DT, code

pytestmark = pytest.mark.gpu


def _place(t: torch.Tensor, offset: int) -> torch.Tensor:
    """`t` in memory that starts `offset` elements after a 16-byte boundary."""
    room = torch.full((t.numel() + offset,), 7.0, dtype=t.dtype, device="cuda")[offset:]
    room.copy_(t.reshape(-1))
    return room.view(t.shape)


@pytest.mark.parametrize("dt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("lens,heads,d", [([1], 1, 1), ([5, 3], 3, 8), ([4, 7, 2], 2, 12), ([33, 1, 0, 17], 5, 20), ([9, 64], 12, 64), ([2, 3], 1, 260)])
@pytest.mark.parametrize("offset", [0, 1])
def test_transposes_are_exact(ctx, dt, lens, heads, d, offset):
    g = torch.Generator().manual_seed(len(lens) * 1000 + heads * d)
    t, B, L = TORCH_DT[dt], len(lens), max(lens)
    draw = lambda *shape: torch.randn(*shape, generator=g).to(t)
    for cu in (None, torch.tensor([sum(lens[:i]) for i in range(B + 1)], dtype=torch.int32)):
        rows = [(b, l) for b in range(B) for l in range(L if cu is None else lens[b])]
        at = torch.tensor([b * L + l for b, l in rows])
        for W in (1, 3):
            x, bias = draw(len(rows), W, heads, d), draw(W, heads, d)
            want = torch.zeros(B * L, W, heads, d, dtype=t)
            want[at] = (x.float() + bias.float()).to(t)
            want = want.view(B, L, W, heads, d).permute(2, 0, 3, 1, 4).contiguous()
            got = [_place(torch.full((B, heads, L, d), 7.0, dtype=t), offset) for _ in range(W)]
            packed = [] if cu is None else [cu.cuda()]
            name = "split_add_bias_transpose" if W == 3 else "add_bias_transpose_for_score"
            ctx.call(name + ("" if cu is None else "_pad"), code(dt), _place(x, offset), _place(bias, offset), *packed, B, L, heads, d, *got)
            for a, b in zip(got, want):
                assert torch.equal(a.cpu(), b)
        head = draw(B, heads, L, d)
        back = _place(torch.full((len(rows), heads, d), 7.0, dtype=t), offset)
        args = (_place(head, offset), B, heads, L, d, back) if cu is None else (_place(head, offset), cu.cuda(), B, L, heads, d, back)
        ctx.call("transpose_for_score" + ("" if cu is None else "_pad"), code(dt), *args)
        assert torch.equal(back.cpu(), head.permute(0, 2, 1, 3).reshape(B * L, heads, d)[at])
