"""The gated products with their activation in the epilogue, few tokens (weight streamer) and many (persistent tiles): token counts around
the tiles' edges, one round of CTAs and more CTAs than SMs, each activation, with and without biases, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def gated(kind, limit, g, u):
    if kind == "clamped_swish":
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
        return g * torch.sigmoid(1.702 * g) * (u + 1)
    if kind == "gelu_tanh":
        return torch.nn.functional.gelu(g, approximate="tanh") * u
    return torch.nn.functional.silu(g) * u


@pytest.mark.parametrize("kind,biased", [("silu", False), ("silu", True), ("gelu_tanh", False), ("clamped_swish", True)])
@pytest.mark.parametrize("F,K", [(72, 136), (10040, 72)])
@pytest.mark.parametrize("T,tiles", [(9, False), (16, False), (17, False), (33, False), (64, False), (65, False), (130, False), (130, True), (300, True)])
def test_gated_products(T, tiles, F, K, kind, biased):
    from imparo_b200.kernels import ops
    gen = torch.Generator().manual_seed(T + F)
    x = torch.randn(T, K, generator=gen).to(torch.bfloat16)
    w = (torch.randn(2 * F, K, generator=gen) * K ** -0.5).to(torch.bfloat16)
    bias = torch.randn(2 * F, generator=gen) if biased else None
    out = torch.full((T + 1, F), 7.0, dtype=torch.bfloat16, device=DEV)
    product = ops.gemm_prefill if tiles else ops.gemm_tc
    product(x.to(DEV), w.to(DEV), out[:T], ops.EPI_SWIGLU, None, act=kind, limit=3.0, bias=None if bias is None else bias.to(DEV))
    assert bool((out[T] == 7.0).all())                       # nothing beyond the tokens
    xd, wd = x.double().to(DEV), w.double().to(DEV)
    z, size = xd @ wd.T, xd.abs() @ wd.abs().T
    if biased:
        z, size = z + bias.double().to(DEV), size + bias.double().abs().to(DEV)
    g, u = z[:, :F], z[:, F:]
    want = gated(kind, 3.0, g, u)
    # a sum is off by at most seventeen cuts at 2^-24 of its terms (a matrix instruction's); an activation's slope is at most 1.2, its
    # value at most its argument's; the exponential and the division of the fast kind: 2^-19 of the factor; then bfloat16, 2^-8
    d = 17 * 2 ** -24 * size
    slope = 1.2 * d[:, :F] * (u.abs() + 1) + g.abs() * d[:, F:]
    tol = slope + (2 ** -19 + 2 ** -8) * want.abs() + 2 ** -18 * g.abs() * (u.abs() + 1) * 2 ** -2
    assert bool(((out[:T].double() - want).abs() <= tol).all())
