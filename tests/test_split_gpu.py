"""fp32 as two scaled fp16 planes: the planes against the values, products of planes against fp64 on every tile (few rows, split along K, wide, pairs, ragged) and
over the range of scales that fp32 has, and the kernels that leave planes for the next product. Tolerances: planes hold 22 bits of an element and 2^-39
of the row's largest; the tensor cores truncate their partial sums, 1e-8 of the result a term.
"""
import pytest
import torch

from turbotransformers_b200 import _capi

pytestmark = pytest.mark.gpu
torch.set_grad_enabled(False)
DEV = torch.device("cuda:0")


def randn(*shape, seed=1, scale=1.0):
    return torch.randn(*shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV) * scale


def err(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def split(ctx, x):
    """Planes [2, rows, K] and their scale."""
    planes, scale = torch.zeros(2, *x.shape, device=DEV).half(), torch.zeros(x.shape[0], device=DEV)
    ctx.call("split_f16", x, x.shape[0], x.shape[1], planes[0], planes[1], scale)
    return planes, scale


def value(planes, scale):
    return (planes[0].double() + planes[1].double()) * scale.double()[:, None]


def held(planes, scale, want, bound):
    """Whether planes hold `want` to what they have bits for; bound: a row's largest magnitude."""
    off = (value(planes, scale) - want.double()).abs()
    return bool((off <= 2.0 ** -22 * want.double().abs() + 2.0 ** -39 * bound.double()[:, None]).all())


@pytest.mark.parametrize("M,K", [(1, 1), (3, 77), (8, 768), (9, 3072), (1000, 40), (1, 8), (2, 264), (5, 8192), (3, 8200), (5000, 768)])
def test_planes(ctx, M, K):
    x = randn(M, K) * 2.0 ** torch.randint(-90, 90, (M, 1), generator=torch.Generator(device=DEV).manual_seed(2), device=DEV)
    x[0, 0] = 0
    planes, scale = split(ctx, x)
    assert held(planes, scale, x, x.abs().amax(1))
    assert torch.equal(torch.frexp(scale).mantissa, torch.full_like(scale, 0.5))  # powers of two
    for odd in (float("nan"), float("inf"), 3.4e38):
        y = x.clone()
        y[-1, -1] = odd
        planes, scale = split(ctx, y)
        assert bool(torch.isfinite(value(planes, scale)[-1, -1])) == (odd == 3.4e38) and held(planes[:, :-1], scale[:-1], x[:-1], x[:-1].abs().amax(1))
    planes, scale = split(ctx, torch.zeros(M, K, device=DEV))
    assert not value(planes, scale).any()


def product(ctx, a, w, N, K, epilogue, **more):
    M = a[1].numel()
    out = torch.full((M, N), 7.0, device=DEV)
    ctx.linear_split(M, N, K, epilogue, out=out, A=a[0][0], A2=a[0][1], row_scale=a[1], W=w[0][0], W2=w[0][1], col_scale=w[1], **more)
    return out


@pytest.mark.parametrize("M,N,K", [(1, 768, 768), (31, 2304, 768), (128, 768, 3072), (129, 3072, 768), (527, 100, 1024), (200, 65, 64), (1100, 3072, 768), (3000, 768, 768),
                                   (5000, 2304, 768), (77, 770, 8)])
def test_product(ctx, M, N, K):
    x, w, bias, res = randn(M, K), randn(N, K, seed=2, scale=K ** -0.5), randn(N, seed=3), randn(M, N, seed=4)
    a, b = split(ctx, x), split(ctx, w)
    exact = x.double() @ w.double().T
    gelu = torch.nn.functional.gelu(exact + bias.double(), approximate="tanh")
    tol = 1e-8 * K + 2e-6  # (tanh in fp32 for the second term)
    assert err(product(ctx, a, b, N, K, _capi.EPI_NONE), exact) < 1e-8 * K + 3e-7
    assert err(product(ctx, a, b, N, K, _capi.EPI_BIAS_RESIDUAL, bias=bias, residual=res), exact + bias.double() + res.double()) < tol
    assert err(product(ctx, a, b, N, K, _capi.EPI_BIAS_GELU, bias=bias), gelu) < tol
    assert ctx.device_status() == 0


@pytest.mark.parametrize("M,N,K", [(1, 768, 768), (128, 768, 768), (17, 512, 512), (128, 384, 384), (250, 512, 512), (128, 1024, 1024), (100, 768, 3072), (300, 2304, 768)])
def test_no_further_off_than_tf32_planes(ctx, M, N, K):
    """Few rows, whose products are split along K: an accumulator adds up no more than with tf32 planes."""
    x, w, tf32 = randn(M, K), randn(N, K, seed=2, scale=K ** -0.5), torch.zeros(M, N, device=DEV)
    exact = x.double() @ w.double().T
    xp, wp = torch.zeros(2, M, K, device=DEV), torch.zeros(2, N, K, device=DEV)
    ctx.call("split_tf32", x, M * K, xp[0], xp[1])
    ctx.call("split_tf32", w, N * K, wp[0], wp[1])
    ctx.linear_ex(_capi.F32, _capi.F32, xp[0], wp[0], M, N, K, _capi.EPI_NONE, tf32, A2=xp[1], W2=wp[1])
    # (both are mostly what the accumulators cut off, which is the same but for the inputs' noise where as much is added up)
    assert err(product(ctx, split(ctx, x), split(ctx, w), N, K, _capi.EPI_NONE), exact) < 1.1 * err(tf32, exact)


@pytest.mark.parametrize("M", [5, 300])
def test_product_over_the_range_of_scales(ctx, M):
    """Rows and columns many powers of two apart, and a row's own elements too: every element is as close to its own terms as in tf32 planes, whose exponent is fp32's."""
    N, K = 96, 256
    powers = lambda n, most, seed: 2.0 ** torch.randint(-most, most, (n, 1), generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)
    x, w = randn(M, K) * powers(M, 50, 5), randn(N, K, seed=2) * powers(N, 50, 6)
    x, w = x * powers(K, 4, 7).T, w * powers(K, 4, 8).T
    out = product(ctx, split(ctx, x), split(ctx, w), N, K, _capi.EPI_NONE)
    terms = x.double().abs() @ w.double().abs().T
    # of every term: both operands' planes, the product of the two second ones that is left out, and the accumulator
    assert float(((out.double() - x.double() @ w.double().T).abs() / terms).max()) < 3 * 2.0 ** -22 + 1e-8 * K


@pytest.mark.parametrize("M,N", [(1, 768), (37, 1024), (149, 768), (1184, 768), (1185, 768), (600, 776), (600, 2048), (1500, 264), (900, 8)])
def test_layer_norm_leaves_the_planes_of_its_output(ctx, M, N):
    out, y, bias, gamma, beta = randn(M, N), randn(M, N, seed=2), randn(N, seed=3), randn(N, seed=4), randn(N, seed=5)
    want = torch.nn.functional.layer_norm((out + y + bias).double(), (N,), gamma.double(), beta.double(), 1e-12)
    planes, scale = torch.zeros(2, M, N, device=DEV).half(), torch.zeros(M, device=DEV)
    ctx.call("add_bias_layernorm_split", out, planes[0], planes[1], scale, y, bias, gamma, beta, M, N, 1e-12)
    assert err(out, want) < 1e-6
    again, s = split(ctx, out)
    assert torch.equal(planes, again) and torch.equal(scale, s)


def test_embedding_leaves_the_planes_of_its_output(ctx):
    for hidden in (768, 128, 1000, 8, 264, 520, 1024, 1032, 2048, 2056):
        ids, out = torch.randint(0, 100, (3, 7), generator=torch.Generator(device=DEV).manual_seed(1), device=DEV), torch.zeros(21, hidden, device=DEV)
        planes, scale, plain = torch.zeros(2, 21, hidden, device=DEV).half(), torch.zeros(21, device=DEV), torch.zeros(21, hidden, device=DEV)
        tables = (randn(100, hidden), randn(16, hidden, seed=2), randn(2, hidden, seed=3), randn(hidden, seed=4), randn(hidden, seed=5))
        ctx.call("embedding_ln_split", ids, None, None, None, 3, 7, 21, *tables, hidden, 100, 16, 2, 1e-12, out, planes[0], planes[1], scale)
        ctx.call("embedding_ln", _capi.F32, ids, None, None, None, 3, 7, 21, *tables, hidden, 100, 16, 2, 1e-12, plain)
        again, s = split(ctx, out)
        assert torch.equal(out, plain) and torch.equal(planes, again) and torch.equal(scale, s)


def test_what_is_refused(ctx):
    x = randn(16, 64)
    a, w = split(ctx, x), split(ctx, randn(32, 64, seed=2))
    out = torch.zeros(16, 32, device=DEV)
    for bad in (dict(A2=None), dict(row_scale=None), dict(col_scale=None), dict(lda=68), dict(K=60), dict(W2=w[0][1].view(-1)[4:])):
        fields = dict(dict(A=a[0][0], A2=a[0][1], row_scale=a[1], W=w[0][0], W2=w[0][1], col_scale=w[1], out=out), **bad)
        with pytest.raises(_capi.TTBError):
            ctx.linear_split(16, 32, fields.pop("K", 64), _capi.EPI_NONE, **fields)
    with pytest.raises(_capi.TTBError):
        ctx.call("add_bias_layernorm_split", x, a[0][0], a[0][1], a[1], x, x, x, x, 16, 60, 1e-12)
    assert ctx.device_status() == 0
