"""Layer norms where the launch changes: a warp a row over one round of the grid and over two, one or two rows a warp before the
int8 form of the output. A row's result depends on that row alone: bit for bit that of a launch of a few rows."""
import pytest
import torch

from turbotransformers_b200 import _capi

pytestmark = pytest.mark.gpu
torch.set_grad_enabled(False)
DEV = torch.device("cuda:0")


def _rows(M, N, dtype):
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x = torch.randn(M, N, generator=g, device=DEV) * 3 + 1
    return x, *(torch.randn(N, generator=g, device=DEV).to(dtype) for _ in range(2))


@pytest.mark.parametrize("N", [8, 256, 776, 1024, 1032])
@pytest.mark.parametrize("waves,more", [(0, 1), (0, 3), (5, 1), (8, 0), (30, 0), (30, 1), (64, 0), (64, 1)])
def test_planes_of_many_rows_are_those_of_few(ctx, N, waves, more):
    M = waves * torch.cuda.get_device_properties(0).multi_processor_count + more
    x, gamma, beta = _rows(M, N, torch.bfloat16)
    out, lo, f = torch.zeros(M, N, device=DEV).bfloat16(), torch.zeros(M, N, device=DEV).bfloat16(), torch.zeros(M, N, device=DEV)
    ctx.call("layernorm_planes", _capi.F32, _capi.BF16, x, out, lo, f, gamma, beta, M, N, 1e-12)
    want = torch.nn.functional.layer_norm(x.double(), (N,), gamma.double(), beta.double(), 1e-12)
    # sums of N fp32 terms in chains of at most N / 32 + 5; values to 2^-24 of numbers up to |gamma| sqrt(N) + |beta|
    assert float((f - want).abs().max()) <= (N / 32 + 16) * 2.0 ** -23 * float(want.abs().max())
    assert torch.equal(out, f.bfloat16()) and torch.equal(lo, (f - out.float()).bfloat16())
    last = x[-2:].contiguous() if M > 1 else x
    o2, l2, f2 = torch.zeros_like(out[-2:]), torch.zeros_like(lo[-2:]), torch.zeros_like(f[-2:])
    ctx.call("layernorm_planes", _capi.F32, _capi.BF16, last, o2, l2, f2, gamma, beta, last.shape[0], N, 1e-12)
    assert torch.equal(f2, f[-2:]) and torch.equal(l2, lo[-2:])


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N", [8, 264, 768, 1024])
@pytest.mark.parametrize("waves,more", [(0, 1), (8, 1), (56, 0), (56, 1)])
def test_int8_form_is_that_of_the_two_kernels(ctx, dtype, N, waves, more):
    M = waves * torch.cuda.get_device_properties(0).multi_processor_count + more
    x, gamma, beta = _rows(M, N, dtype)
    x, code = x.to(dtype), _capi.F16 if dtype == torch.float16 else _capi.BF16
    out, q, s = torch.zeros_like(x), torch.zeros(M, N, dtype=torch.int8, device=DEV), torch.zeros(M, device=DEV)
    ctx.call("layernorm_quant_int8", code, x, out, q, s, gamma, beta, M, N, 1e-12)
    out2, q2, s2 = torch.zeros_like(x), torch.zeros_like(q), torch.zeros_like(s)
    ctx.call("layernorm", code, x, out2, gamma, beta, M, N, 1e-12)
    ctx.call("quantize_rows_int8", code, out2, M, N, q2, s2)
    assert torch.equal(out, out2) and torch.equal(q, q2) and torch.equal(s, s2)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("N", [8, 256, 264, 1024])
@pytest.mark.parametrize("waves,more", [(5, 1), (8, 0), (30, 1), (30, 2), (56, 0), (56, 1)])
def test_sums_of_many_rows_are_those_of_few(ctx, dtype, N, waves, more):
    M = waves * torch.cuda.get_device_properties(0).multi_processor_count + more
    y, gamma, beta = _rows(M, N, dtype)
    y, bias, out, code = y.to(dtype), beta * 3, (y * 0.5 + 1).to(dtype), _capi.dtype_code(dtype)
    last = out[-3:].clone()
    want = torch.nn.functional.layer_norm(out.double() + y.double() + bias.double(), (N,), gamma.double(), beta.double(), 1e-12)
    ctx.call("add_bias_layernorm", code, out, y, bias, gamma, beta, M, N, 1e-12)
    tolerance = (N / 32 + 16) * 2.0 ** -23 if dtype == torch.float32 else 2.0 ** -10
    assert float((out.double() - want).abs().max()) <= tolerance * float(want.abs().max())
    ctx.call("add_bias_layernorm", code, last, y[-3:].contiguous(), bias, gamma, beta, 3, N, 1e-12)
    assert torch.equal(last, out[-3:])
