"""The small kernels of a decode step at the edges of their forms: routed experts of few rows (one round of stretches and several, a
round that is partly empty, experts nobody names, a shared expert), the combine of an attention's key chunks (a warp's form up to 32
chunks and the block's beyond), products per head and the choice of experts, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from imparo_b200.kernels import ops as o
    return o


CUTS = 17 * 2 ** -24


def near(got, want, magnitude):
    """Sums in 32 bits of terms whose magnitudes add up to `magnitude`.  A matrix instruction cuts its sixteen products and the sum so
    far at 2^-24 of the largest of them (it does not round): seventeen such cuts, and the largest may be all of the magnitude where
    the terms are few (40)."""
    assert bool(((got.double().cpu() - want).abs() <= CUTS * magnitude).all())


@pytest.mark.parametrize("rows", [1, 8, 9, 17])
@pytest.mark.parametrize("width,ff,s_ff", [(1024, 1536, 0), (1024, 1536, 200), (1288, 1032, 1544), (3080, 72, 40), (24, 2056, 0)])
def test_routed_experts(rows, width, ff, s_ff):
    g = torch.Generator().manual_seed(rows + ff)
    E, top = 12, 2
    h = torch.randn(rows, width, generator=g).to(torch.bfloat16)
    up = (torch.randn(E, ff, width, generator=g) * width ** -0.5).to(torch.bfloat16)
    down = (torch.randn(E, width, ff, generator=g) * ff ** -0.5).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(E - 3, generator=g)[:top] for _ in range(rows)]).int()       # three experts are never named
    wts = torch.rand(rows, top, generator=g)
    mid = torch.empty(rows * top, ff, dtype=torch.bfloat16, device=DEV)
    out = torch.full((rows, width), float("nan"), device=DEV)
    shared = None
    if s_ff:
        su = (torch.randn(s_ff, width, generator=g) * width ** -0.5).to(torch.bfloat16)
        sd = (torch.randn(width, s_ff, generator=g) * s_ff ** -0.5).to(torch.bfloat16)
        s_mid, y = torch.empty(rows, s_ff, dtype=torch.bfloat16, device=DEV), torch.full((rows, width), float("nan"), device=DEV)
        shared = (su.to(DEV), sd.to(DEV), s_mid, y)
    ops().moe_experts(h.to(DEV), up.to(DEV), down.to(DEV), ids.to(DEV), wts.to(DEV), top, False, mid, out, act="plain:relu2", shared=shared)

    def check_mid(got, x, w):
        """relu(z)^2 rounded to bfloat16 (2^-8 of itself); z off by d (as in near) moves it by (2 z + d) d,
        and the square is one more 32-bit rounding."""
        z = x.double() @ w.double().T
        d = CUTS * (x.double().abs() @ w.double().abs().T)
        want = z.clamp_min(0) ** 2
        assert bool(((got.double().cpu() - want).abs() <= 2 ** -8 * want + 1.01 * (2 * z.abs() + d) * d + 2 ** -23 * want + 1e-38).all())

    for r in range(rows):
        for k in range(top):
            check_mid(mid[r * top + k], h[r:r + 1], up[ids[r, k]])
    m = mid.double().cpu().view(rows, top, ff)
    want, size = torch.zeros(rows, width, dtype=torch.float64), torch.zeros(rows, width, dtype=torch.float64)
    for r in range(rows):
        for k in range(top):
            w = down[ids[r, k]].double()
            want[r] += wts[r, k].double() * (w @ m[r, k])
            size[r] += wts[r, k].double() * (w.abs() @ m[r, k].abs())
    near(out, want, size)
    if s_ff:
        check_mid(s_mid, h, su)
        s = s_mid.double().cpu()
        near(y, s @ sd.double().T, s.abs() @ sd.double().abs().T)


@pytest.mark.parametrize("rows,top", [(4, 8), (17, 2), (16, 8), (32, 8)])
@pytest.mark.parametrize("width,ff", [(1024, 1536), (264, 72)])
def test_layers_in_a_row_share_the_choices_buffer(rows, top, width, ff):
    """Every layer's choice goes into the same buffer and the down launch reads it before its wait (32 pairs and more): a chain of
    layers without anything between gives bit for bit what each layer gives alone, from a buffer of its own."""
    o = ops()
    g = torch.Generator().manual_seed(rows * top + ff)
    E, layers = 40, 6
    h = torch.randn(rows, width, generator=g).to(torch.bfloat16).to(DEV)
    up = (torch.randn(E, ff, width, generator=g) * width ** -0.5).to(torch.bfloat16).to(DEV)
    down = (torch.randn(E, width, ff, generator=g) * ff ** -0.5).to(torch.bfloat16).to(DEV)
    logits = torch.randn(layers, rows, E, generator=g).to(DEV)
    mid = torch.empty(rows * top, ff, dtype=torch.bfloat16, device=DEV)
    pair_out = torch.empty(rows * top, width, device=DEV)
    ids, wts = torch.empty(rows, top, dtype=torch.int32, device=DEV), torch.empty(rows, top, device=DEV)

    def layer(i, ids, wts, out):
        o.moe_pick(logits[i], E, 1, top, ids, wts, renormalise=True)
        o.moe_experts(h, up, down, ids, wts, top, False, mid, out, act="plain:relu2", pair_out=pair_out)

    want = torch.full((layers, rows, width), float("nan"), device=DEV)
    for i in range(layers):
        layer(i, torch.empty_like(ids), torch.empty_like(wts), want[i])
        torch.cuda.synchronize()
    for _ in range(3):
        got = torch.full_like(want, float("nan"))
        torch.cuda.synchronize()
        for i in range(layers):
            layer(i, ids, wts, got[i])
        assert torch.equal(got, want)


@pytest.mark.parametrize("sink", [False, True])
@pytest.mark.parametrize("hd", [32, 96, 128, 200])
@pytest.mark.parametrize("splits", [1, 8, 16, 17, 32, 33])
def test_combine(splits, hd, sink):
    g = torch.Generator().manual_seed(splits * hd)
    rows = 6
    acc = torch.randn(rows, splits, hd, generator=g)
    ml = torch.stack([torch.randn(rows, splits, generator=g) * 3, torch.rand(rows, splits, generator=g) + 0.5], dim=-1)
    empty = torch.rand(rows, splits, generator=g) < 0.3
    empty[0] = True                                          # a row without any key
    if splits > 1:
        empty[1, :] = True
        empty[1, splits - 1] = False                         # one whose keys are all in the last chunk
    ml[empty] = torch.tensor([float("-inf"), 0.0])
    acc[empty] = float("nan")                                # what an empty chunk leaves counts for nothing
    out = torch.empty(rows, hd, device=DEV)
    ops().attention_split_combine(acc.to(DEV), ml.contiguous().to(DEV), out, rows, hd, splits, sink=sink)
    m, l = ml[..., 0].double(), ml[..., 1].double()
    top = m.amax(1, keepdim=True)
    if sink:
        top = top.clamp_min(0.0)
    f = torch.where(empty, torch.zeros_like(m), torch.exp(m - top))
    total = (f * l).sum(1, keepdim=True) + (torch.exp(-top) if sink else 0.0)
    a = torch.nan_to_num(acc.double(), nan=0.0)
    dead = (total == 0) | total.isnan()
    want = torch.where(dead, torch.zeros_like(total), (f[..., None] * a).sum(1) / total)
    size = torch.where(dead, torch.zeros_like(total), (f[..., None] * a.abs()).sum(1) / total)
    # expf's own error is two units (2^-22); numerator and denominator have it, and up to 33 terms' roundings each (2^-24)
    assert bool(((out.double().cpu() - want).abs() <= (2 * 2 ** -22 + 2 * 34 * 2 ** -24) * size).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("gate", [None, "each", "head"])
@pytest.mark.parametrize("rows,n_in,n_out", [(1, 1, 3), (8, 96, 64), (9, 128, 5), (3, 130, 64), (17, 300, 6)])
def test_heads(rows, n_in, n_out, gate, dtype):
    g = torch.Generator().manual_seed(n_in)
    heads = 3
    x, w = torch.randn(rows, heads * n_in, generator=g).to(dtype), (torch.randn(heads, n_out, n_in, generator=g) * n_in ** -0.5).to(dtype)
    z = None if gate is None else torch.randn(rows, heads * (n_out if gate == "each" else 1), generator=g)
    out = torch.empty(rows, heads * n_out, dtype=dtype, device=DEV)
    ops().heads_linear(x.to(DEV), w.to(DEV), out, None if z is None else z.to(DEV))
    xd, wd = x.double().view(rows, heads, n_in), w.double()
    want, size = torch.einsum("rhi,hoi->rho", xd, wd), torch.einsum("rhi,hoi->rho", xd.abs(), wd.abs())
    if gate is not None:
        s = torch.sigmoid(z.double()).view(rows, heads, -1)
        want, size = want * s, size * s
    # the sum as above; the sigmoid: expf, an add, a divide and the product, eight units together; bfloat16: half a unit
    tol = (2 ** -22 + 8 * 2 ** -24) * size + (2 ** -8 if dtype == torch.bfloat16 else 0) * want.abs()
    assert bool(((out.double().cpu().view_as(want) - want).abs() <= tol).all())


@pytest.mark.parametrize("experts,parts,correct", [(16, 3, True), (16, 1, False), (80, 3, True), (40, 2, False)])
def test_choice(experts, parts, correct):
    """The pieces of a logit, corrections within and beyond the first 32 experts, weights renormalised and scaled."""
    g = torch.Generator().manual_seed(experts)
    rows, top = 11, 4
    pieces = torch.randn(rows, parts, experts, generator=g) * 0.7
    corr = torch.randn(experts, generator=g) if correct else None
    ids, wts = torch.empty(rows, top, dtype=torch.int32, device=DEV), torch.empty(rows, top, device=DEV)
    ops().moe_pick(pieces.reshape(rows, -1).contiguous().to(DEV), experts, parts, top, ids, wts, renormalise=True, weight_scale=2.5,
                   correction=None if corr is None else corr.to(DEV))
    z = pieces[:, 0].clone()
    for p in range(1, parts):
        z = z + pieces[:, p]                                 # in 32 bits, in order
    score = torch.sigmoid(z.double())
    by = score + corr.double() if correct else z.double()
    best = by.topk(top, dim=1)
    assert float((by.sort(dim=1, descending=True).values[:, :top + 1].diff(dim=1).abs()).min()) > 1e-6      # (no tie to be decided by a rounding)
    assert torch.equal(ids.cpu().long(), best.indices)
    w = score.gather(1, best.indices)
    want = w / w.sum(1, keepdim=True) * 2.5
    # a sigmoid is off by four units (2^-24 each), a weight is two of them (its own and the sum's) and four operations
    assert bool(((wts.double().cpu() - want).abs() <= 16 * 2 ** -24 * want).all())
