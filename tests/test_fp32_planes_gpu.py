"""fp32 models on the tensor cores: the one-kernel attention against plain PyTorch in fp64 at the edges of its tiles, and the second planes
that the kernels leave for the next product (what the tensor cores drop of a value). Tolerances: sums in fp32 of up to 512 terms.
"""
import math

import pytest
import torch

from turbotransformers_b200 import _capi

pytestmark = pytest.mark.gpu
torch.set_grad_enabled(False)
DEV = torch.device("cuda:0")


def rest(x):
    """What is left of x without its last 13 bits, to the 10 bits and the implicit one that tf32 has (rounded half away from zero)."""
    x = x.contiguous()
    r = x - (x.view(torch.int32) & -8192).view(torch.float32)
    return ((r.view(torch.int32) + 4096) & -8192).view(torch.float32)


def err(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("lens,heads,masked,causal", [([1], 12, 0, 0), ([128], 12, 0, 0), ([7, 64, 33, 120], 12, 0, 0), ([65, 65, 65], 2, 1, 0), ([130] * 4, 3, 1, 0),
                                                      ([50, 17, 513], 12, 0, 1), ([40, 40], 12, 2, 0)])
def test_attention(ctx, lens, heads, masked, causal):
    B, T, H, L = len(lens), sum(lens), heads * 64, max(lens)
    g = torch.Generator(device=DEV).manual_seed(sum(lens))
    qkv = torch.randn(T, 3 * H, generator=g, device=DEV)
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).int()
    mask = None
    if masked:
        mask = torch.where(torch.rand(B, L if masked == 2 else 1, L, generator=g, device=DEV) < 0.3, -10000.0, 0.0).contiguous()
    out, lo = torch.zeros(T, H, device=DEV), torch.zeros(T, H, device=DEV)
    ctx.call("attention_f32", qkv, cu, B, L, heads, 64, mask, 0 if mask is None else mask.shape[1] * L, L if masked == 2 else 0, causal, 0.125, out, lo)
    for b, n in enumerate(lens):
        rows = slice(int(cu[b]), int(cu[b + 1]))
        q, k, v = (t.reshape(n, heads, 64).transpose(0, 1).double() for t in qkv[rows].split(H, 1))
        s = q @ k.transpose(1, 2) / 8
        if mask is not None:
            s = s + mask[b][None].double()
        if causal:
            s = s.masked_fill(~torch.ones(n, n, dtype=torch.bool, device=DEV).tril(), -math.inf)
        assert err(out[rows], (s.softmax(-1) @ v).transpose(0, 1).reshape(n, H)) < 2e-6
    assert torch.equal(lo, rest(out))


@pytest.mark.parametrize("M,N,K", [(1, 768, 768), (128, 3072, 768), (200, 100, 768), (1100, 3072, 768), (3000, 3072, 768), (130, 770, 64)])
def test_product_of_rows_as_they_are(ctx, M, N, K):
    """A taken as it is with its rest, and the output's own rest from every tile of the product (few rows, wide, ragged)."""
    g = torch.Generator(device=DEV).manual_seed(M)
    x, w, bias = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV) * K ** -0.5, torch.randn(N, generator=g, device=DEV)
    planes = torch.zeros(2, N, K, device=DEV)
    ctx.call("split_tf32", w, N * K, planes[0], planes[1])
    out, lo, plain = (torch.zeros(M, N, device=DEV) for _ in range(3))
    ctx.linear_ex(_capi.F32, _capi.F32, x, planes[0], M, N, K, _capi.EPI_BIAS_GELU, out, A2=rest(x), W2=planes[1], bias=bias, out_lo=lo)
    want = torch.nn.functional.gelu(x.double() @ w.double().T + bias.double(), approximate="tanh")
    split = torch.zeros(2, M, K, device=DEV)
    ctx.call("split_tf32", x, M * K, split[0], split[1])
    ctx.linear_ex(_capi.F32, _capi.F32, split[0], planes[0], M, N, K, _capi.EPI_BIAS_GELU, plain, A2=split[1], W2=planes[1], bias=bias)
    # as close as the rounded split is (1e-8 a term of truncation in the accumulator, which both have)
    assert err(out, want) < 1.1 * err(plain, want) + 2e-7
    assert err(out, want) < 2e-5
    assert torch.equal(lo, rest(out))


@pytest.mark.parametrize("M,N", [(1, 768), (37, 1024), (1184, 768), (1185, 768), (3000, 768), (5, 770)])
def test_layer_norm(ctx, M, N):
    g = torch.Generator(device=DEV).manual_seed(N)
    x, y = torch.randn(M, N, generator=g, device=DEV), torch.randn(M, N, generator=g, device=DEV)
    bias, gamma, beta = (torch.randn(N, generator=g, device=DEV) for _ in range(3))
    want = torch.nn.functional.layer_norm((x + y + bias).double(), (N,), gamma.double(), beta.double(), 1e-12)
    out, lo = x.clone(), torch.zeros(M, N, device=DEV)
    ctx.call("add_bias_layernorm_f32", out, lo, y, bias, gamma, beta, M, N, 1e-12)
    assert err(out, want) < 1e-6
    assert torch.equal(lo, rest(out))
