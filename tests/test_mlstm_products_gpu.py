"""The matrix memory's chunks as products (csrc/kernels/mlstm_chunk.cu) against the row walk and the recurrence in 64 bits."""
import numpy as np
import pytest

from tests import zepesun_cases as C

pytestmark = pytest.mark.gpu


def run(rows, lens, H, D, V, b_i, b_f, cap, chunk, state=None):
    import torch
    from imparo_b200.kernels import ops
    f32 = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float32, device="cuda")
    i32 = lambda a: torch.as_tensor(a, dtype=torch.int32, device="cuda")
    vb, R, T, qk, vv = ops.mlstm_value_blocks(V), len(lens), len(rows), H * D, H * V
    if state is None:
        state = [torch.zeros(s, device="cuda") for s in ((R + 1, H, D, V), (R + 1, H, vb, D), (R + 1, H, vb))]
    S, n, m = (t.clone() for t in state)
    out = torch.full((T, vv), float("nan"), device="cuda")
    scratch, status = None, ops.new_status("cuda")
    if chunk:
        most = T // chunk + R
        scratch = tuple(torch.full((most * H * k,), float("nan"), device="cuda") for k in (D * V, vb * D, vb * 3))
    x = f32(rows)
    assert ops.mlstm_products_take(x, D, V)
    ops.mlstm_scan(x, 0, qk, 2 * qk, 2 * qk + 2 * vv, 2 * qk + 2 * vv + H, f32(b_i), f32(b_f), cap, D ** -0.5, S, n, m,
                   i32(np.concatenate([[0], np.cumsum(lens)])), i32(list(range(R, 0, -1))), R, out, H, D, V, status, chunk=chunk, scratch=scratch)
    ops.read_status(status)
    return out.cpu().double().numpy(), [t.cpu().double().numpy() for t in (S, n, m)]


# chunks of one row, one short of 64, 64 and one more; key sizes of part of a tile, one tile, part of a second, two; value blocks alike
@pytest.mark.parametrize("H,D,V", [(2, 4, 4), (2, 60, 68), (2, 64, 128), (2, 68, 64), (2, 128, 132), (4, 32, 64)])
def test_products_are_as_exact_as_the_row_walk(H, D, V):
    rng = np.random.default_rng(D + V)
    lens = [1, 63, 64, 65, 200]
    rows, b_i, b_f = C.memory_inputs(rng, sum(lens), H, D, V)
    rows = rows.astype(np.float32).astype(np.float64)
    b_i, b_f = b_i.astype(np.float32).astype(np.float64), b_f.astype(np.float32).astype(np.float64)
    got, gs = run(rows, lens, H, D, V, b_i, b_f, 10.0, 64)
    walk, ws = run(rows, lens, H, D, V, b_i, b_f, 10.0, 0)
    at, errors, states_off = 0, {"products": [], "walk": []}, {"products": 0.0, "walk": 0.0}
    for r, n in enumerate(lens):
        want, states = C.memory_plain(rows[at:at + n], b_i, b_f, H, D, V, 10.0)
        want = want.reshape(n * H, V)
        for name, o, s in (("products", got, gs), ("walk", walk, ws)):
            off = np.linalg.norm(o[at:at + n].reshape(n * H, V) - want, axis=1) / np.linalg.norm(want, axis=1)
            errors[name] += off.tolist()
            for t, w in zip(s, states):
                mine = t[len(lens) - r]
                if mine.ndim > w.ndim:                            # a copy per block of value columns
                    mine, w = mine, np.repeat(np.expand_dims(w, 1), mine.shape[1], 1)
                states_off[name] = max(states_off[name], np.linalg.norm(mine - w) / np.linalg.norm(w))
        at += n
    # both are 32-bit sums of the same terms, grouped differently.  (A row whose n . q nearly cancels is off by more in either way, so
    # rows are compared by their median; the states have no such quotient.)
    assert np.median(errors["products"]) <= max(1.2 * np.median(errors["walk"]), 6e-8), {k: np.median(v) for k, v in errors.items()}
    assert max(errors["products"]) <= 8 * max(errors["walk"])
    assert states_off["products"] <= 1.2 * states_off["walk"], states_off


@pytest.mark.parametrize("bad", [0, 70, 127])
@pytest.mark.parametrize("column", ["k", "v", "i"])
def test_a_row_that_is_not_finite_reaches_no_earlier_row(bad, column):
    H, D, V = 2, 64, 64
    rng = np.random.default_rng(bad)
    rows, b_i, b_f = C.memory_inputs(rng, 150, H, D, V)
    good, _ = run(rows, [150], H, D, V, b_i, b_f, 10.0, 64)
    rows[bad, {"k": H * D, "v": 2 * H * D, "i": 2 * H * (D + V)}[column]] = np.nan
    got, _ = run(rows, [150], H, D, V, b_i, b_f, 10.0, 64)
    assert np.array_equal(got[:bad], good[:bad]) and np.isnan(got[bad]).any()
