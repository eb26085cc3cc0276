"""The product of at most eight rows (csrc/kernels/gemm_rows.cu) with its norm, gate, add and convolution, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from imparo_b200.kernels import ops as o
    return o


def case(T, N, K, seed, std=None):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g) * K ** -0.5).to(torch.bfloat16)
    return x, w, g


def close(got, want, magnitude, bf16):
    """A 32-bit sum whose terms' magnitudes add up to `magnitude`, in blocks of a few dozen and of eight: 2^-22 of that is four
    roundings of the whole.  A bfloat16 result (8 significant bits) is rounded by half a unit in its last place, at most 2^-8 of
    itself."""
    assert bool(((got.double().cpu() - want).abs() <= 2 ** -22 * magnitude + (2 ** -8 if bf16 else 0) * want.abs()).all())


# rows of W per SM: none or one, part of a tile, one tile, several pairs, the most there is room for; K: one block of 64, part of a
# stage of 512, a stage and part of a second, a stretch of 2,048, part of a second one
@pytest.mark.parametrize("N", [1, 72, 148, 1024, 1200, 2048, 6144, 148 * 128])
@pytest.mark.parametrize("K", [64, 448, 576, 2048, 2304, 8192])
def test_product(N, K):
    o = ops()
    for T in (1, 5, 8):
        x, w, g = case(T, N, K, N * 7 + K + T)
        want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
        xd, wd = x.to(DEV), w.to(DEV)
        assert o._rows_take(xd, wd)
        for dtype in (torch.float32, torch.bfloat16):
            out = torch.full((T, N), float("nan"), dtype=dtype, device=DEV)
            o._gemm_rows(xd, wd, out, o.ROWS_F32 if dtype == torch.float32 else o.ROWS_BF16)
            close(out, want, size, dtype == torch.bfloat16)
        base = torch.randn(T, N, generator=g)
        out = base.to(DEV)
        o._gemm_rows(xd, wd, out, o.ROWS_ADD)
        close(out, want + base.double(), size + base.double().abs(), False)


def test_most_rows_of_w():
    o = ops()
    x, w, _ = case(4, 148 * 128 + 1, 64, 3)
    assert not o._rows_take(x.to(DEV), w.to(DEV))            # 129 rows on one SM: the other product's
    assert not o._rows_take(torch.zeros(4, 72, dtype=torch.bfloat16, device=DEV), torch.zeros(64, 72, dtype=torch.bfloat16, device=DEV))
    assert not o._rows_take(torch.zeros(9, 64, dtype=torch.bfloat16, device=DEV), torch.zeros(64, 64, dtype=torch.bfloat16, device=DEV))


def normed(x, nw, eps):
    """The RMS norm of 32-bit rows in bfloat16, and how far an entry may be off.  The kernel's 32-bit value is within 2^-18 of the exact
    one (a lane's sum of up to 64 squares, half of whose error the root leaves, and four more roundings: under 40 times 2^-24), so an
    entry is the rounding of the exact value unless a boundary lies that near; then it may be the neighbour."""
    h = x.double() / torch.sqrt(x.double().pow(2).mean(1, keepdim=True) + eps) * nw.double()
    low, high = ((h * (1 + s * 2 ** -18)).to(torch.bfloat16).double() for s in (-1, 1))
    return h.to(torch.bfloat16).double(), (high - low).abs()


def product_of_normed(h, off, w):
    """The product and the bound of its error: at most seventeen cuts at 2^-24 of the terms' magnitudes (a matrix instruction's, and the
    warps' sums), and the entries of h that may be the neighbour."""
    wa = w.double().abs()
    return h @ w.double().T, 17 * 2 ** -24 * (h.abs() @ wa.T) + off @ wa.T


def waiting_norm(o, x, nw, eps=1e-5):
    T, K = x.shape
    h = torch.full((T, K), float("nan"), dtype=torch.bfloat16, device=DEV)
    o.rmsnorm(x.to(DEV), nw.to(DEV), eps, h, may_wait=True)
    assert h.data_ptr() in o._S.waiting_norms and bool(h.isnan().all())
    return h


@pytest.mark.parametrize("F,K", [(1, 64), (9, 832), (4608, 1024), (8192, 2048), (148 * 64, 128)])
@pytest.mark.parametrize("act,bias", [("silu", False), ("clamped_swish", True)])
def test_gated_of_a_waiting_norm(F, K, act, bias):
    o = ops()
    for T in (1, 3, min(8, o.FEW_ROWS_STREAM // K)):
        _, w, g = case(T, 2 * F, K, F + K + T)
        x, nw = torch.randn(T, K, generator=g) * 3, 1 + 0.1 * torch.randn(K, generator=g)
        b = torch.randn(2 * F, generator=g) if bias else None
        xd, nd, wd = x.to(DEV), nw.to(DEV), w.to(DEV)
        h2 = torch.full((T, K), float("nan"), dtype=torch.bfloat16, device=DEV)
        o.rmsnorm(xd, nd, 1e-5, h2)
        h = waiting_norm(o, x, nw)
        out = torch.full((T, F), float("nan"), dtype=torch.bfloat16, device=DEV)
        o.linear_gated(h, wd, out, act, limit=7.0, bias=b.to(DEV) if bias else None)
        z, d = product_of_normed(*normed(x, nw, 1e-5), w)
        if bias:
            z = z + b.double()
            d = d + 2 ** -24 * z.abs()
        gate, up, dg, du = z[:, :F], z[:, F:], d[:, :F], d[:, F:]
        if act == "silu":
            want = gate * torch.sigmoid(gate) * up
        else:
            gate, up = gate.clamp(max=7.0), up.clamp(-7.0, 7.0)
            want = gate * torch.sigmoid(1.702 * gate) * (up + 1.0)
        # an activation's slope is at most 1.2 and its value at most its argument's; the fast exponential and division: 2^-18; bfloat16: 2^-8
        tol = 1.2 * dg * (up.abs() + 1 + du) + gate.abs() * du + 2 ** -18 * gate.abs() * (up.abs() + 1) + (2 ** -8 + 2 ** -18) * want.abs()
        assert bool(((out.double().cpu() - want).abs() <= tol).all())
        o.make_waiting(h)
        assert torch.equal(h, h2)                                # the norm itself, when somebody else reads it


@pytest.mark.parametrize("N,K", [(1, 64), (72, 832), (1536, 1024), (3072, 2048), (6144, 1024)])
def test_plain_products_of_a_waiting_norm(N, K):
    """linear into both types, and the one-part product that linear_unfolded leaves to its reader."""
    o = ops()
    for T in (1, 4, min(8, o.FEW_ROWS_STREAM // K)):
        _, w, g = case(T, N, K, N + K + T)
        x, nw = torch.randn(T, K, generator=g) * 3, 1 + 0.1 * torch.randn(K, generator=g)
        want, d = product_of_normed(*normed(x, nw, 1e-5), w)
        wd, h = w.to(DEV), waiting_norm(o, x, nw)

        def near(got, half):
            assert bool(((got.double().cpu() - want).abs() <= d + (2 ** -8 * (want.abs() + d) if half else 0)).all())
        for dtype in (torch.float32, torch.bfloat16):
            out = torch.full((T, N), float("nan"), dtype=dtype, device=DEV)
            o.linear(h, wd, out)
            near(out, dtype == torch.bfloat16)
            out = torch.full((T, N), float("nan"), dtype=dtype, device=DEV)
            made = o.linear_unfolded(h, wd, out)
            assert isinstance(made, o.PartialProduct) and made.splits == 1 and made.shape == (T, N) and bool(out.isnan().all())
            near(made.parts[:T * N].view(T, N), False)
            whole = made.parts[:T * N].view(T, N).to(dtype)
            assert made.tensor() is out and torch.equal(out, whole)
        assert h.data_ptr() in o._S.waiting_norms and bool(h.isnan().all())
        o.forget_waiting(h)


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("F,K,bias", [(5, 64, True), (148, 2048, False), (1024, 1024, False), (1540, 576, True), (4096, 256, False)])
def test_convolution_of_one_token_rows(taps, F, K, bias):
    """The fused kernel and the two kernels apart: same rows to within the roundings of the product, same states."""
    o = ops()
    for T in (1, 6, 8):
        x, w, g = case(T, 3 * F, K, F + K + taps + T)
        tw, b = torch.randn(F, taps, generator=g).to(DEV), torch.randn(F, generator=g).to(DEV) if bias else None
        state = torch.randn(T + 2, taps - 1, F, generator=g).to(DEV)
        iot = torch.arange(T, dtype=torch.int32, device=DEV)
        slots = torch.tensor([(3 * i + 1) % (T + 2) if (T + 2) % 3 else i for i in range(T)], dtype=torch.int32, device=DEV)
        start = torch.arange(T + 1, dtype=torch.int32, device=DEV)
        st = o.new_status(DEV)
        s1, s2 = state.clone(), state.clone()
        y1, y2 = (torch.full((T, F), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2))
        xd, wd = x.to(DEV), w.to(DEV)
        assert o.linear_conv_rows(xd, wd, tw, b, s1, iot, slots, y1, taps, st)
        bcx = (xd.double() @ wd.double().T).to(torch.float32).to(torch.bfloat16)
        o.gated_conv(bcx, tw, b, s2, start, iot, slots, y2, taps, st)
        o.read_status(st)
        # an entry of the product that falls to the other side of a rounding moves a value of b x by 2^-8 of itself
        assert (y1.float() - y2.float()).abs().max() <= 2 ** -6 * y2.float().abs().max()
        assert (s1 - s2).abs().max() <= 2 ** -7 * s2.abs().max()
        assert torch.equal(s1[:, :-1], s2[:, :-1])               # what is only moved on
        untouched = [i for i in range(T + 2) if i not in slots.tolist()]
        assert torch.equal(s1[untouched], state[untouched])


def test_convolution_reports_a_state_slot_out_of_range():
    o = ops()
    x, w, g = case(2, 3 * 64, 64, 1)
    state = torch.randn(2, 2, 64, generator=g).to(DEV)
    before, st = state.clone(), o.new_status(DEV)
    y = torch.zeros(2, 64, dtype=torch.bfloat16, device=DEV)
    assert o.linear_conv_rows(x.to(DEV), w.to(DEV), torch.ones(64, 3, device=DEV), None, state,
                              torch.arange(2, dtype=torch.int32, device=DEV), torch.tensor([2, 0], dtype=torch.int32, device=DEV), y, 3, st)
    with pytest.raises(o.KernelError, match="state slot"):
        o.read_status(st)
    assert torch.equal(state[1], before[1])
