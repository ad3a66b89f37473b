"""Chains whose operations hand their results on through a flow (ttb_chain_forward_flow) against the same operations with a barrier over the grid between
them (ttb_chain_forward, which the other tests hold against fp64): the same kernel, so that every bit has to be the same. Row counts
at the edges of the kernels (tiles of eight rows), widths that are a whole number of a kernel's steps of K and widths that are not, deep products whose
rows are fetched in several pieces.
"""
import pytest
import torch

from turbotransformers_b200 import _capi

pytestmark = pytest.mark.gpu
torch.set_grad_enabled(False)
DEV = torch.device("cuda:0")
DEVICE_WAIT = 5  # TTB_ERR_DEVICE_WAIT


def half(*shape, seed, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).half()


class Flow:
    def __init__(self, n):
        self.memory, self.at = torch.empty(n, dtype=torch.uint8, device=DEV), 0

    def next(self, rows, columns):
        t = self.memory[self.at:self.at + rows * columns * 2].view(torch.float16).view(rows, columns)
        self.at += (rows * columns * 2 + 255) // 256 * 256
        return t


def stack(x, heads, F, weights, flow, keys, past=37, length=19, layers=2):
    """Pre-LN layers (the second product of each with a normalised copy that is the residual of a later one), as a decoder's and as an encoder's."""
    M, H = x.shape
    ops, into = [], x
    for layer in range(layers):
        w = weights[layer]
        rows, qkv, context, total, inter, out = flow.next(M, H), flow.next(M, 3 * H), flow.next(M, H), flow.next(M, H), flow.next(M, F), flow.next(M, H)
        ops.append(("linear", dict(A=into, W=w["qkv"], bias=w["b"], gamma=w["g"], beta=w["g"], normed=rows, out=qkv, M=M, N=3 * H, K=H, lda=H, ldo=3 * H, eps=1e-5)))
        at = dict(q=qkv, out=context, rows=M, heads=heads, ldq=3 * H, ldo=H, keys=keys, scale=0.125)
        if keys == _capi.CHAIN_KEYS_ROWS:
            at.update(length=M, causal=1)
        elif keys == _capi.CHAIN_KEYS_CACHE:
            at.update(past=past, k_cache=w["k"], v_cache=w["v"])
        else:
            at.update(length=length, k=w["k"], v=w["v"])
        ops.append(("attention", at))
        ops.append(("linear", dict(A=context, W=w["o"], bias=w["b"], residual=rows, out=total, M=M, N=H, K=H, lda=H, ldo=H, ldr=H)))
        ops.append(("linear", dict(A=total, W=w["up"], bias=w["b"], gamma=w["g"], beta=w["g"], out=inter, M=M, N=F, K=H, lda=H, ldo=F, eps=1e-5, act=1)))
        ops.append(("linear", dict(A=inter, W=w["down"], bias=w["b"], residual=total, out=out, M=M, N=H, K=F, lda=F, ldo=H, ldr=H)))
        into = out
    return ops, into


def weights_of(M, H, F, seed, past=37):
    return [dict(qkv=half(3 * H, H, seed=seed + i, scale=H ** -0.5), o=half(H, H, seed=seed + i + 10, scale=H ** -0.5), up=half(F, H, seed=seed + i + 20, scale=H ** -0.5),
                 down=half(H, F, seed=seed + i + 30, scale=F ** -0.5), b=half(max(F, 3 * H), seed=seed + i + 40), g=half(H, seed=seed + i + 50, scale=0.1) + 1,
                 k=half(past // 16 + 1, M, 16, H, seed=seed + i + 60), v=half(past // 16 + 1, M, 16, H, seed=seed + i + 70)) for i in range(2)]


@pytest.mark.parametrize("H,F,V", [(512, 2048, 1003), (768, 3072, 50257), (1024, 4096, 8), (320, 640, 24), (960, 6720, 40)])
@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 24, 25, 32, 33, 64])
def test_the_same_bits_as_with_barriers(ctx, M, H, F, V):
    if M > _capi.lib().ttb_chain_rows(H, F):
        pytest.skip("more rows than the chain takes")
    heads, w, head = H // 64, weights_of(M, H, F, 1), half(V, H, seed=9, scale=0.05)
    for keys in (_capi.CHAIN_KEYS_ROWS, _capi.CHAIN_KEYS_CACHE, _capi.CHAIN_KEYS_MEMORY):
        flow = Flow(2 * (M + 8) * (9 * H + F) * 2 + 8192)
        x = half(M, H, seed=3)
        ops, last = stack(x, heads, F, w, flow, keys)
        hidden, logits = torch.zeros(M, H, device=DEV).half(), torch.zeros(M, V, device=DEV).half()
        ops.append(("linear", dict(A=last, W=head, out=logits, M=M, N=V, K=H, lda=H, ldo=V, eps=1e-5, gamma=w[0]["g"], beta=w[0]["g"], normed=hidden)))
        for seed in (3, 4, 3):  # other inputs over the flow of the call before
            x.copy_(half(M, H, seed=seed))
            ctx.chain_forward(ops)
            want = (hidden.clone(), logits.clone(), w[1]["k"].clone(), w[1]["v"].clone())
            hidden.zero_(), logits.zero_()
            ctx.chain_forward_flow(ops, flow.memory)
            torch.cuda.synchronize()
            assert all(torch.equal(a, b) for a, b in zip((hidden, logits, w[1]["k"], w[1]["v"]), want)) and want[0].abs().max() > 0, (keys, seed)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf"), 65504.0])
def test_results_that_are_not_numbers_are_results(ctx, bad):
    """No NaN that a product makes is the word for `not written`: the chain ends, with what the barriers give."""
    M, H, F = 9, 512, 1024
    w, flow = weights_of(M, H, F, 5), Flow(1 << 20)
    x = half(M, H, seed=3)
    x[4, 77] = bad
    ops, last = stack(x, 8, F, w, flow, _capi.CHAIN_KEYS_CACHE)
    out = torch.zeros(M, H, device=DEV).half()
    ops.append(("linear", dict(A=last, gamma=w[0]["g"], beta=w[0]["g"], normed=out, M=M, N=0, K=H, lda=H, eps=1e-5)))
    ctx.chain_forward(ops)
    want = out.clone()
    ctx.chain_forward_flow(ops, flow.memory)
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int16), want.view(torch.int16)) and ctx.device_status() == 0


def test_what_a_flow_has_to_be(ctx):
    M, H = 4, 512
    w, x = half(H, H, seed=1, scale=0.05), half(M, H, seed=2)
    linear = lambda A, out, **more: ("linear", dict(dict(A=A, W=w, out=out, M=M, N=H, K=H, lda=H, ldo=H), **more))
    flow = Flow(1 << 16)
    first, second = flow.next(M, H), flow.next(M, H)
    ctx.chain_forward_flow([linear(x, first), linear(first, second)], flow.memory)
    for ops in ([linear(x, second), linear(second, first)],            # not in order
                [linear(x, first), linear(first, first)],              # written twice
                [linear(x, first.view(-1)[1:]), linear(x, second)],    # half words
                [linear(x, flow.memory[(1 << 16) - 256:])],            # beyond its end
                [("attention", dict(q=x, out=first, rows=M, heads=2, length=3, ldq=H, ldo=H, k=second, v=second, keys=_capi.CHAIN_KEYS_MEMORY, scale=1.0))]):
        with pytest.raises(_capi.TTBError):
            ctx.chain_forward_flow(ops, flow.memory)
    torch.cuda.synchronize()
    assert ctx.device_status() == 0


def test_a_result_that_nobody_writes_is_waited_for_and_reported(ctx):
    """The wait ends by itself after a second or so, the status word says so, and the next call is in order again."""
    M, H = 2, 512
    w, x, flow = half(H, H, seed=1, scale=0.05), half(M, H, seed=2), Flow(1 << 16)
    never, out = flow.next(M, H), flow.next(M, H)
    op = dict(W=w, out=out, M=M, N=H, K=H, lda=H, ldo=H)
    ctx.chain_forward_flow([("linear", dict(op, A=never))], flow.memory)
    torch.cuda.synchronize()
    assert ctx.device_status() == DEVICE_WAIT and ctx.device_status() == 0
    ctx.chain_forward_flow([("linear", dict(op, A=x))], flow.memory)
    torch.cuda.synchronize()
    want = x.double() @ w.double().T
    assert float((out.double() - want).norm() / want.norm()) < 1e-3 and ctx.device_status() == 0
