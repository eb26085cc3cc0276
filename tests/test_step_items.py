"""A step's items on the host (no GPU): tokens and wanted places as arrays, their checks, and the rules that choose a kernel from a
step's shape."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from imparo_b200.engine import Engine, StepItem
from imparo_b200.engine import engine as engine_module
from imparo_b200.engine.step import int_array


def test_whole_numbers_as_an_array():
    for values in ([5, 0, 7], (5, 0, 7), range(3), np.arange(3), np.arange(3, dtype=np.int8), np.arange(3, dtype=np.uint32), [np.int64(4), True],
                   [torch.tensor(3)]):
        got = int_array(values)
        assert got.dtype == np.int64 and got.tolist() == [int(v) for v in values]
    exact = np.arange(4)
    assert int_array(exact) is exact
    for values in ({1, 2}, [0.5, 1], [2 ** 70], np.array([0.5]), np.array([[1, 2]]), torch.arange(3), {1: 2}, [], "12"):
        assert int_array(values) is None


def _checked(items):
    return Engine._checked(SimpleNamespace(vocab_size=100, ctx=64, cache=SimpleNamespace(has=lambda r: r == 7, cached=lambda r: 50)), items)


@pytest.mark.parametrize("n", [3, 20])
def test_tokens_out_of_the_vocabulary_are_refused(n):
    good = list(range(n))
    for make in (list, tuple, np.array, lambda t: np.array(t, dtype=np.int16), torch.tensor):
        (item,) = _checked([StepItem(1, make(good), (0,))])
        assert [int(t) for t in item.tokens] == good and item.want == (0,) and item.request == 1
        for wrong in (100, -1):
            with pytest.raises(ValueError, match="request 1: token id out of range"):
                _checked([StepItem(1, make(good[:-1] + [wrong]))])
    for wrong in (2 ** 70, -2 ** 70, -0.5, 100.0):
        with pytest.raises(ValueError, match="token id out of range"):
            _checked([StepItem(1, good[:-1] + [wrong])])
    if n > 14:
        with pytest.raises(ValueError, match="exceed the context length"):
            _checked([StepItem(7, good)])


def test_arrays_are_not_walked_entry_by_entry(monkeypatch):
    def walked(values):
        raise AssertionError("walked in Python")
    for name in ("min", "max"):
        monkeypatch.setattr(engine_module, name, walked, raising=False)
    for dtype in (np.int64, np.int32):
        tokens = np.arange(60, dtype=dtype)
        assert np.array_equal(_checked([StepItem(1, tokens)])[0].tokens, tokens)


# both sides of the line where they were measured: portions of one or several requests after thousands of positions, or from position 0
@pytest.mark.parametrize("nh,nkv,hd,rows,requests,from_start,tiles", [
    (16, 8, 64, 8, 1, False, False), (16, 8, 64, 64, 1, False, False), (16, 8, 64, 256, 1, False, True), (32, 8, 64, 64, 1, False, False),
    (32, 8, 64, 256, 1, False, True), (8, 2, 128, 256, 1, False, False), (8, 2, 128, 512, 1, False, True), (4, 4, 64, 256, 1, False, False),
    (4, 4, 64, 512, 1, False, True), (16, 8, 64, 256, 32, False, False), (32, 8, 64, 256, 32, False, False), (16, 8, 64, 400, 4, False, True),
    (16, 8, 64, 80, 16, False, False), (32, 4, 64, 64, 1, False, True), (48, 8, 64, 64, 1, False, True), (16, 2, 64, 16, 1, False, False),
    (16, 8, 16, 256, 1, False, False), (16, 8, 16, 1000, 1, False, True), (16, 8, 32, 128, 1, False, False), (16, 8, 48, 256, 1, False, True),
    (16, 8, 64, 16, 1, True, False), (16, 8, 64, 128, 1, True, True), (32, 8, 64, 64, 1, True, True), (16, 8, 64, 1000, 3, True, True),
    (8, 2, 128, 64, 1, True, False), (4, 4, 64, 64, 1, True, False), (18, 2, 64, 8, 1, False, True)])
def test_where_32_bit_portions_go_to_the_tiles(nh, nkv, hd, rows, requests, from_start, tiles):
    from imparo_b200.kernels import ops
    assert ops.attention_f32_tiles_pay(rows, requests, nh, nkv, hd, from_start) is tiles


@pytest.mark.parametrize("heads,vdim,state,rows,products", [
    (64, 32, 16, 511, True), (64, 32, 16, 1999, False), (64, 32, 128, 256, True), (64, 32, 128, 511, False), (64, 16, 16, 256, False),
    (64, 16, 16, 100, True), (32, 16, 64, 511, True), (32, 16, 128, 1999, False), (64, 36, 16, 1999, True), (64, 64, 128, 1999, True),
    (8, 8, 8, 1999, True)])
def test_where_state_space_chunks_run_as_products(heads, vdim, state, rows, products):
    from imparo_b200.kernels import ops
    assert ops.mamba2_products_pay(heads, vdim, state, rows // 64 + 1) is products


# walk / chunks in us where both were measured: the portions' lengths, whose longest the rule sees rounded up to a power of two
@pytest.mark.parametrize("heads,dim,vdim,portions,chunks", [
    (8, 64, 128, [256], False), (8, 64, 128, [257], False), (8, 64, 128, [512], True), (8, 64, 128, [8] * 31 + [300], False),
    (8, 64, 128, [16] * 8 + [300], True), (8, 64, 128, [64] * 8 + [512], True), (64, 64, 64, [400], False), (64, 64, 64, [512], True),
    (64, 64, 64, [257] * 4, False), (128, 64, 64, [512], False), (128, 32, 32, [1000, 1000], False), (32, 64, 128, [100] * 10 + [600], True),
    (16, 128, 128, [257], True), (16, 128, 128, [16] * 8 + [300], False), (16, 128, 128, [64] * 8 + [512], True), (32, 128, 128, [512], True),
    (32, 128, 128, [8] * 31 + [300], False), (2, 64, 64, [16] * 16 + [400], True), (32, 16, 16, [300], True), (4, 128, 256, [2048], True)])
def test_where_the_delta_rule_runs_in_chunks(heads, dim, vdim, portions, chunks):
    from imparo_b200.parts.delta_rule import GatedDeltaRule
    part = GatedDeltaRule({"hidden": 64, "heads": heads, "kv_heads": heads, "dim": dim, "vdim": vdim, "conv": 4, "decay_rank": 8, "gate_rank": 8,
                           "eps": 1e-6}, "L.", None)
    assert part._in_chunks(1 << (max(portions) - 1).bit_length(), sum(portions), len(portions)) is chunks
