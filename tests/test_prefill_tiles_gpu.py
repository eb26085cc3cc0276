"""The persistent prompt product's three tiles (csrc/kernels/gemm_prefill.cu): shapes whose rounds choose each of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# (tokens, features, K): tiles of 128 x 256; 256 x 192; 256 x 256.  Tokens one short of a half, one more, second halves of one row, none
SHAPES = [(256, 1000, 200), (1300, 8192, 256), (512, 6912, 1536), (385, 6912, 1536), (257, 6912, 264), (700, 4608, 1024), (641, 4608, 1024),
          (512, 8192, 2048), (300, 8192, 2048), (384, 8192, 520)]


@pytest.mark.parametrize("T,F,K", SHAPES)
def test_gated_products(T, F, K):
    from imparo_b200.kernels import ops as o
    g = torch.Generator(device=DEV).manual_seed(T + F + K)
    x = torch.randn(T, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(2 * F, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    out = torch.full((T, F), float("nan"), dtype=torch.bfloat16, device=DEV)
    st = o.new_status(DEV)
    o.gemm_prefill(x, w, out, o.EPI_SWIGLU, st)
    o.read_status(st)
    gu = x.float() @ w.float().T
    gate, up = gu[:, :F], gu[:, F:]
    want = gate * torch.sigmoid(gate) * up
    # rounded to bfloat16 (half a unit, 2^-8 of itself at most), 32-bit sums of K products and the fast exponential before that
    assert bool(((out.float() - want).abs() <= 2 ** -8 * want.abs() + 1e-4).all())


@pytest.mark.parametrize("T,N,K", [(512, 13824, 1536), (257, 13824, 72), (300, 16384, 512), (129, 520, 64)])
@pytest.mark.parametrize("epilogue", ["store", "float32", "add"])
def test_plain_products(T, N, K, epilogue):
    from imparo_b200.kernels import ops as o
    g = torch.Generator(device=DEV).manual_seed(T + N + K)
    x = torch.randn(T, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    base = torch.randn(T, N, generator=g, device=DEV)
    out = base.clone() if epilogue == "add" else torch.full((T, N), float("nan"), device=DEV, dtype=torch.bfloat16 if epilogue == "store" else torch.float32)
    st = o.new_status(DEV)
    o.gemm_prefill(x, w, out, {"store": o.EPI_STORE_BF16, "float32": o.EPI_STORE_F32, "add": o.EPI_ADD_F32}[epilogue], st)
    o.read_status(st)
    want = (x.double() @ w.double().T + (base.double() if epilogue == "add" else 0.0)).float()
    assert bool(((out.float() - want).abs() <= (2 ** -8 if epilogue == "store" else 0) * want.abs() + 2e-5).all())
