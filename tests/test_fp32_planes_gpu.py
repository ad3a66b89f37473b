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


def split(ctx, x):
    hi, lo = torch.zeros_like(x), torch.zeros_like(x)
    ctx.call("split_tf32", x, x.numel(), hi, lo)
    return torch.stack([hi, lo])


@pytest.mark.parametrize("M,N", [(1, 768), (128, 3072), (200, 100), (1100, 3072), (3000, 3072), (130, 770), (77, 2316)])
def test_planes_of_a_product(ctx, M, N):
    """Every tile of the product (few rows, split along K, wide, pairs, ragged) leaves, in place of its output, what splitting that output gives."""
    K = 768 if M != 130 else 64
    g = torch.Generator(device=DEV).manual_seed(M)
    x, w, bias = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV) * K ** -0.5, torch.randn(N, generator=g, device=DEV)
    a, b = split(ctx, x), split(ctx, w)
    hi, lo, plain, rest_of_plain = (torch.full((M, N), 7.0, device=DEV) for _ in range(4))
    product = lambda epilogue, out, **kw: ctx.linear_ex(_capi.F32, _capi.F32, a[0], b[0], M, N, K, epilogue, out, A2=a[1], W2=b[1], bias=bias, **kw)
    product(_capi.EPI_BIAS_GELU | _capi.EPI_FLAG_TF32_PLANES, hi, out_lo=lo)
    product(_capi.EPI_BIAS_GELU, plain, out_lo=rest_of_plain)  # the same tile, and with it the same sums
    assert torch.equal(torch.stack([hi, lo]), split(ctx, plain))
    with pytest.raises(_capi.TTBError):
        product(_capi.EPI_BIAS_GELU | _capi.EPI_FLAG_TF32_PLANES, plain)


def test_planes_of_layer_norm_attention_and_embedding(ctx):
    g = torch.Generator(device=DEV).manual_seed(1)
    rand = lambda *shape: torch.randn(*shape, generator=g, device=DEV)
    for M, N in ((1, 768), (37, 1024), (148, 768), (149, 768), (297, 768), (1184, 768), (1185, 768), (5, 770), (600, 776), (600, 2048), (1500, 264), (900, 248)):
        out, hi, lo = rand(M, N), torch.zeros(M, N, device=DEV), torch.zeros(M, N, device=DEV)
        ctx.call("add_bias_layernorm_f32_planes", out, hi, lo, rand(M, N), rand(N), rand(N), rand(N), M, N, 1e-12)
        assert torch.equal(torch.stack([hi, lo]), split(ctx, out))
    for lens in ([1], [7, 64, 33, 120], [65] * 30):
        T, H = sum(lens), 768
        cu = torch.tensor([0] + lens, device=DEV).cumsum(0).int()
        qkv, out, hi, lo = rand(T, 3 * H), *(torch.zeros(T, H, device=DEV) for _ in range(3))
        ctx.call("attention_f32", qkv, cu, len(lens), max(lens), 12, 64, None, 0, 0, 0, 0.125, out, None)
        ctx.call("attention_f32_planes", qkv, cu, len(lens), max(lens), 12, 64, None, 0, 0, 0, 0.125, hi, lo)
        assert torch.equal(torch.stack([hi, lo]), split(ctx, out))
    ids, out, planes = torch.randint(0, 100, (3, 7), generator=g, device=DEV), torch.zeros(21, 768, device=DEV), torch.zeros(2, 21, 768, device=DEV)
    ctx.call("embedding_ln_planes", _capi.F32, ids, None, None, None, 3, 7, 21, rand(100, 768), rand(16, 768), rand(2, 768), rand(768), rand(768), 768, 100, 16, 2,
             1e-12, out, planes[1], planes[0])
    assert torch.equal(planes, split(ctx, out))


@pytest.mark.parametrize("B,L", [(1, 17), (3, 64), (9, 200)])
def test_planes_hold_an_activation_to_the_last_bit_that_splitting_it_would(B, L):
    """A layer gives the same bits for an activation that brings its planes along and for the same values without them."""
    import turbotransformers_b200 as tt
    from turbotransformers_b200 import synthetic
    from turbotransformers_b200._cxx import cxx
    hf = synthetic.make_hf_bert("bert-base", num_layers=1).to(DEV).encoder.layer[0]
    attention, inter, out = tt.BertAttention.from_torch(hf.attention), tt.BertIntermediate.from_torch(hf.intermediate), tt.BertOutput.from_torch(hf.output)
    turbo = tt.ReturnType.turbo_transformers
    bare = lambda t: torch.from_numpy(cxx.tensor2nparrayf(t)).to(DEV)
    x = torch.randn(B, L, 768, generator=torch.Generator(device=DEV).manual_seed(B), device=DEV)
    a = attention(x, return_type=turbo)[0]
    i = inter(a, return_type=turbo)
    assert torch.equal(bare(i), inter(bare(a)))
    y = out(i, a, return_type=turbo)
    assert torch.equal(bare(y), out(bare(i), bare(a)))
    assert torch.equal(attention(y)[0], attention(bare(y))[0])
    # a NaN or an infinity, from the largest values on, is not lost on the way
    for bad in (float("nan"), float("inf"), 3.4e38):
        z = bare(y).clone()
        z.view(-1, 768)[0, 5] = bad
        assert not torch.isfinite(out(inter(z, return_type=turbo), z).view(-1, 768)[0]).any()
        w = attention(z)[0].view(B, L, 768)
        assert not torch.isfinite(out(inter(w, return_type=turbo), w)[0, 0]).any() and torch.isfinite(w[1:]).all()
    # between the two products of a layer the activation is its planes
    planes = cxx.Tensor.create_empty()
    inter.for_output(a, planes)
    assert err(out(planes, a), bare(y)) < 2e-6  # (the tile of the first product, and with it the order of its sums, may be another)
    cxx.set_fp32_tensor_cores(False)
    try:  # and stays what it is when the switch is thrown in between
        assert err(out(planes, a), bare(y)) < 1e-4
    finally:
        cxx.set_fp32_tensor_cores(True)
