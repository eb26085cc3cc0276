"""The scratch for cut 32-bit operands on the host (no GPU): its size follows the products a model makes, and an engine does without it
where there is no room."""
import pytest
import torch

from imparo_b200.config.engine import EngineConfig
from imparo_b200.config.registry import load_config
from imparo_b200.kernels import lib, ops
from imparo_b200.parts.base import Runtime, Workspace
from imparo_b200.parts.model import Model


def bytes_for(M, N, K):
    return 6 * ((K + 7) // 8 * 8) * (M + N) if K % 4 == 0 else 0


@pytest.fixture
def state(monkeypatch):
    entries = type("Entries", (), {"imparo_sgemm_cut_bytes": staticmethod(bytes_for)})()
    monkeypatch.setattr(lib, "kernels", lambda: entries)
    previous = ops.use_state(ops.LaunchState())
    yield ops._S
    ops.use_state(previous)


def lfm2(width, heads, ff, vocab):
    return {"architectures": ["Lfm2ForCausalLM"], "model_type": "lfm2", "vocab_size": vocab, "hidden_size": width, "num_hidden_layers": 2,
            "layer_types": ["conv", "full_attention"], "num_attention_heads": heads, "num_key_value_heads": 8, "block_ff_dim": ff,
            "block_auto_adjust_ff_dim": False, "conv_L_cache": 3, "conv_bias": False, "rope_theta": 1000000.0, "norm_eps": 1e-5,
            "tie_embedding": True, "max_position_embeddings": 4096}


def bound(config):
    """The model with its tensors bound, without memory behind them."""
    arch, cfg = load_config(config)
    device = torch.device("meta")
    rt = Runtime(precision="float32", device=device, workspace=Workspace(device))
    model = Model(arch.model_spec(cfg), rt)
    model.bind({w.name: torch.empty(w.shapes[0], dtype=torch.float32, device=device) for w in model.weight_specs()})
    return model


@pytest.mark.parametrize("width,heads,ff", [(1024, 16, 4608), (1536, 24, 6912), (2048, 32, 8192)])
def test_the_scratch_is_as_large_as_the_layers_products_need(state, width, heads, ff):
    """2,048-token steps of the three preset sizes with a vocabulary of 65,536: the products of the layers as their parts stacked them
    (gate and up together), and a head that only ever sees the wanted rows."""
    tokens, wanted = 2056, 10
    model = bound(lfm2(width, heads, ff, 65536))
    matrices = model.product_matrices(wanted)
    qkv = (heads + 2 * 8) * 64
    assert (width, 3) in matrices                               # (the convolution's taps: rows of no 16-byte groups, never cut)
    assert set(matrices) - {(width, 3)} == {(3 * width, width), (width, width), (qkv, width), (2 * ff, width), (width, ff), (65536, width, wanted)}
    ops.prepare_cut("cpu", tokens, matrices)
    assert state.planes[0].numel() == 6 * max(width * (tokens + 2 * ff), ff * (tokens + width))     # gate and up, or down


def test_products_that_are_never_cut_take_no_room(state):
    ops.prepare_cut("cpu", 64, [(1024, 4608)])                  # fewer rows than cutting starts with
    assert not state.planes
    ops.prepare_cut("cpu", 2048, [(1024, 4608, 10), (1 << 20, 4096)])       # too few of the head's rows; more than there may be
    assert not state.planes
    assert ops._cut_pays(130, 1024, 4608)
    ops.prepare_cut("cpu", 130, [(1024, 4608)])
    assert state.planes[0].numel() == bytes_for(130, 1024, 4608)


def test_a_device_without_room_is_no_failure(state, monkeypatch):
    def full(*args, **kwargs):
        raise torch.OutOfMemoryError("no room")
    monkeypatch.setattr(torch, "empty", full)
    ops.prepare_cut("cpu", 2048, [(9216, 1024)])
    assert not state.planes and state.generation == 0


def test_the_switch_leaves_the_scratch_out(state):
    state.switches = EngineConfig.resolve(flags={"cut_f32": False}, env={}).switches
    ops.prepare_cut("cpu", 2048, [(9216, 1024)])
    assert not state.planes
