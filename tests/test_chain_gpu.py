"""Stacks of layers over few rows as one kernel (ttb_chain_forward): each operation against plain PyTorch in fp64 at the edges of its
tiles (rows in sixteens, columns in eights, K in slots, keys in pages of sixteen, more pairs than warps), a longer chain through the
grid's barrier, and the calls that it refuses. Tolerances: fp16 outputs of sums in fp32, 2^-11 of the value and of the sums' terms.
"""
import math

import pytest
import torch

from turbotransformers_b200 import _capi

pytestmark = pytest.mark.gpu
torch.set_grad_enabled(False)
DEV = torch.device("cuda:0")


def half(*shape, seed, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).half()


def close(got, want, rel=2e-3, most=1e-3, extra=0.0):
    """2-norm over 2-norm, and every element by itself: a rounding to fp16 is 2^-11 = 4.9e-4 of the value at most; as much again, and as much of the
    row's root mean square, for the fp32 sums and what went into them. extra: what else an element may be off."""
    got, want = got.double(), want.double()
    assert torch.isfinite(got).all()
    err = (got - want).norm() / want.norm().clamp_min(1e-30)
    assert err < rel, float(err)
    bound = most * (want.abs() + want.square().mean(-1, keepdim=True).sqrt()) + extra
    assert ((got - want).abs() <= bound).all(), float(((got - want).abs() / bound).max())


def norm(x, g, b, eps):
    return torch.nn.functional.layer_norm(x.double(), x.shape[-1:], g.double(), b.double(), eps)


@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32, 33, 63, 64])
@pytest.mark.parametrize("N,K,normed", [(768, 768, True), (8, 256, True), (3072, 1024, True), (24, 320, True), (768, 3072, False), (1024, 4096, False),
                                        (2304, 512, False), (40, 2048, False), (4000, 1536, False)])
def test_linear(ctx, M, N, K, normed):
    x, w, bias, res = half(M, K, seed=1), half(N, K, seed=2, scale=K ** -0.5), half(N, seed=3), half(M, N, seed=4)
    g, b = half(K, seed=5, scale=0.1) + 1, half(K, seed=6)
    out, rows = torch.full((M, N), 7.0, device=DEV).half(), torch.zeros(M, K, device=DEV).half()
    op = dict(A=x, W=w, bias=bias, out=out, M=M, N=N, K=K, lda=K, ldo=N, act=1 if normed else 2, eps=1e-6)
    if normed:
        op.update(gamma=g, beta=b, normed=rows)
    else:
        op.update(residual=res, ldr=N)
    ctx.chain_forward([("linear", op)])
    if normed:
        close(rows, norm(x, g, b, 1e-6), 1e-3)
        inner = rows.double() @ w.double().T + bias.double()
        want = torch.nn.functional.gelu(inner, approximate="tanh")
        extra = 2.0 ** -11 * 0.51 * inner.abs()  # 0.5 x (1 + tanh): the hardware's tanh is good to 2^-10.99
    else:
        want, extra = torch.relu(x.double() @ w.double().T + bias.double()) + res.double(), 0.0
    close(out, want, extra=extra)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("M,N", [(1, 50257), (33, 50257), (64, 30522), (5, 1)])
def test_wide_ragged_product_behind_a_layer_norm(ctx, M, N):
    K = 768
    x, w, g, b = half(M, K, seed=1), half(N, K, seed=2, scale=0.05), half(K, seed=5, scale=0.1) + 1, half(K, seed=6)
    out, rows = torch.full((M, N + 3), 7.0, device=DEV).half(), torch.zeros(M, K, device=DEV).half()
    ctx.chain_forward([("linear", dict(A=x, W=w, out=out, M=M, N=N, K=K, lda=K, ldo=N + 3, eps=1e-5, gamma=g, beta=b, normed=rows))])
    want = rows.double() @ w.double().T
    close(out[:, :N], want)
    close(out[:, (N - 1) // 8 * 8:N], want[:, (N - 1) // 8 * 8:])  # the last, ragged unit by itself
    assert (out[:, N:] == 7.0).all()  # nothing beyond a row's own columns
    assert ctx.device_status() == 0


def attend(q, k, v, bias=None):
    """q [.., 64], k and v [n, 64] per leading index -> (context, probabilities)."""
    s = (q.double().unsqueeze(-2) @ k.double().transpose(-1, -2)).squeeze(-2) / 8.0
    p = (s if bias is None else s + bias.double()).softmax(-1)
    return (p.unsqueeze(-2) @ v.double()).squeeze(-2), p


@pytest.mark.parametrize("B,L,heads,causal", [(1, 1, 12, 1), (1, 17, 12, 0), (4, 16, 12, 1), (1, 64, 16, 0), (64, 1, 16, 1), (3, 21, 2, 0)])
def test_attention_over_rows(ctx, B, L, heads, causal):
    M, H = B * L, heads * 64
    qkv, out = half(M, 3 * H, seed=1), torch.zeros(M, H, device=DEV).half()
    mask = None if causal else torch.where(torch.rand(B, L, generator=torch.Generator(device=DEV).manual_seed(9), device=DEV) < 0.3, -10000.0, 0.0)
    pages = (L + 15) // 16
    kc, vc = (torch.zeros(pages, B, 16, H, device=DEV).half() for _ in range(2))
    op = dict(q=qkv, out=out, rows=M, heads=heads, length=L, ldq=3 * H, ldo=H, keys=_capi.CHAIN_KEYS_ROWS, causal=causal, scale=0.125)
    if causal:
        op.update(k_cache=kc, v_cache=vc)
    else:
        op.update(mask=mask, mask_pitch=L)
    ctx.chain_forward([("attention", op)])
    q, k, v = (t.reshape(B, L, heads, 64).transpose(1, 2) for t in qkv.split(H, 1))
    s = q.double() @ k.double().transpose(-1, -2) / 8.0
    if causal:
        s = s.masked_fill(~torch.ones(L, L, dtype=torch.bool, device=DEV).tril(), -math.inf)
        for cache, x in ((kc, k), (vc, v)):
            assert torch.equal(cache.permute(0, 2, 1, 3).reshape(pages * 16, B, H)[:L].transpose(0, 1), x.transpose(1, 2).reshape(B, L, H))
    else:
        s = s + mask[:, None, None].double()
    close(out.reshape(B, L, H), (s.softmax(-1) @ v.double()).transpose(1, 2).reshape(B, L, H))


@pytest.mark.parametrize("B,heads,past", [(1, 12, 1), (1, 12, 15), (1, 12, 16), (3, 8, 255), (1, 2, 1000), (32, 12, 316), (64, 16, 77)])
def test_attention_over_a_cache(ctx, B, heads, past):
    H = heads * 64
    qkv, out = half(B, 3 * H, seed=1), torch.zeros(B, H, device=DEV).half()
    pages = past // 16 + 1
    kc, vc = half(pages, B, 16, H, seed=2), half(pages, B, 16, H, seed=3)
    flat = lambda c: c.permute(1, 0, 2, 3).reshape(B, pages * 16, heads, 64).clone()
    k, v = flat(kc), flat(vc)
    ctx.chain_forward([("attention", dict(q=qkv, out=out, rows=B, heads=heads, past=past, ldq=3 * H, ldo=H, k_cache=kc, v_cache=vc,
                                          keys=_capi.CHAIN_KEYS_CACHE, scale=0.125))])
    q, kn, vn = (t.reshape(B, heads, 64) for t in qkv.split(H, 1))
    k[:, past], v[:, past] = kn, vn
    assert torch.equal(flat(kc), k) and torch.equal(flat(vc), v)  # filed, and nothing else touched
    want, _ = attend(q, k[:, :past + 1].transpose(1, 2), v[:, :past + 1].transpose(1, 2))
    close(out, want.reshape(B, H))


@pytest.mark.parametrize("B,heads,Lk", [(1, 8, 1), (20, 8, 45), (64, 8, 200), (2, 12, 17), (1, 4, 2000)])
def test_attention_over_a_memory(ctx, B, heads, Lk):
    H = heads * 64
    q, k, v = half(B, H, seed=1), half(B, heads, Lk, 64, seed=2), half(B, heads, Lk, 64, seed=3)
    lens = torch.randint(1, Lk + 1, (B,), generator=torch.Generator(device=DEV).manual_seed(4), device=DEV)
    mask = torch.where(torch.arange(Lk, device=DEV)[None] < lens[:, None], 0.0, -1e18)
    out, probs = torch.zeros(B, H, device=DEV).half(), torch.zeros(B, Lk, device=DEV).half()
    ctx.chain_forward([("attention", dict(q=q, k=k, v=v, out=out, rows=B, heads=heads, length=Lk, ldq=H, ldo=H, mask=mask, mask_pitch=Lk, probs=probs,
                                          scores=torch.empty(B, Lk, device=DEV), keys=_capi.CHAIN_KEYS_MEMORY, scale=0.125))])
    want, p = attend(q.reshape(B, heads, 64), k, v, mask[:, None])
    close(out, want.reshape(B, H))
    close(probs, p[:, 0])


@pytest.mark.parametrize("M", [1, 20, 64])
def test_long_chain(ctx, M):
    """Every operation reads what all CTAs wrote just before: 126 products around the ring and through the grid's barrier."""
    H, F, n = 512, 2048, 63
    w1, w2 = half(n, F, H, seed=1, scale=H ** -0.5), half(n, H, F, seed=2, scale=0.3 * F ** -0.5)
    g, b, bias1, bias2 = half(n, H, seed=3, scale=0.1) + 1, half(n, H, seed=4, scale=0.1), half(n, F, seed=5, scale=0.1), half(n, H, seed=6, scale=0.1)
    x = half(M, H, seed=7)
    start, inter = x.clone(), torch.zeros(M, F, device=DEV).half()
    ops = []
    for i in range(n):
        ops.append(("linear", dict(A=x, W=w1[i], bias=bias1[i], gamma=g[i], beta=b[i], out=inter, M=M, N=F, K=H, lda=H, ldo=F, act=2, eps=1e-5)))
        ops.append(("linear", dict(A=inter, W=w2[i], bias=bias2[i], residual=x, out=x, M=M, N=H, K=F, lda=F, ldo=H, ldr=H)))
    for repeat in range(3):
        x.copy_(start)
        ctx.chain_forward(ops)
        want = start.double()
        for i in range(n):
            want = want + torch.relu(norm(want, g[i], b[i], 1e-5) @ w1[i].double().T + bias1[i].double()) @ w2[i].double().T + bias2[i].double()
        close(x, want, 1e-2, n * 2.0 ** -11)  # 63 roundings of the stream to 2^-11
        if repeat:
            assert torch.equal(x, first)  # the order of sums does not depend on timing
        first = x.clone()
    assert ctx.device_status() == 0


def test_refusals(ctx):
    x, w, out = half(64, 768, seed=1), half(8, 768, seed=2), torch.zeros(64, 8, device=DEV).half()
    good = dict(A=x, W=w, out=out, M=64, N=8, K=768, lda=768, ldo=8)
    ctx.chain_forward([("linear", good)])
    for bad in (dict(M=65), dict(M=0), dict(K=100), dict(K=128), dict(lda=767), dict(ldo=7), dict(out=None), dict(A=x[:, 1:]), dict(act=9), dict(gamma=x[0])):
        with pytest.raises(_capi.TTBError):
            ctx.chain_forward([("linear", {**good, **bad})])
    with pytest.raises(_capi.TTBError):
        ctx.chain_forward([("linear", good)] * 129)
    with pytest.raises(_capi.TTBError):
        ctx.chain_forward([("attention", dict(q=x, out=out, rows=4, heads=1, length=3, ldq=192, ldo=64, keys=_capi.CHAIN_KEYS_ROWS))])


def test_rows_that_a_chain_takes(ctx):
    rows = _capi.lib().ttb_chain_rows
    assert [rows(512, 2048), rows(768, 3072), rows(1024, 4096), rows(768, 100), rows(100, 512), rows(2048, 8192)] == [64, 64, 32, 0, 0, 0]
    assert [rows(512, 8192), rows(1024, 8192)] == [32, 16]
    for hidden, inner in ((768, 3072), (1024, 4096), (512, 8192), (1024, 8192)):  # the kernel agrees, also where the ring is the limit
        for M in (rows(hidden, inner), rows(hidden, inner) + 1):
            x, h, w1, w2 = half(M, hidden, seed=1), half(M, inner, seed=2), half(8, hidden, seed=3), half(8, inner, seed=4)
            out, g = torch.zeros(M, 8, device=DEV).half(), half(hidden, seed=5)
            ops = [("linear", dict(A=x, W=w1, out=out, M=M, N=8, K=hidden, lda=hidden, ldo=8, gamma=g, beta=g)),
                   ("linear", dict(A=h, W=w2, out=out, M=M, N=8, K=inner, lda=inner, ldo=8))]
            if M > rows(hidden, inner):
                with pytest.raises(_capi.TTBError):
                    ctx.chain_forward(ops)
            else:
                ctx.chain_forward(ops)
