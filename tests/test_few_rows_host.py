"""The rules around products of few rows on the host (no GPU; the launches are left out): what a step of more rows asks, which norms
may be left to the products that read them, and what becomes of such a norm."""
import pytest
import torch

from imparo_b200.kernels import lib, ops


@pytest.fixture
def launches(monkeypatch):
    """The launchers on CPU tensors: entry points are noted by name and do nothing (a plan cuts K in two)."""
    noted = []

    class Entries:
        def __getattr__(self, name):
            def entry(*args):
                if name == "imparo_gemm_tc_plan":
                    T, N, _, _, nt, splits, floats, counters = args
                    nt._obj.value, splits._obj.value, floats._obj.value, counters._obj.value = 16, 2, 2 * T * N, 128
                    return 0
                if name == "imparo_gemm_rows_takes":
                    return 1
                noted.append(name[len("imparo_"):])
                return 0
            return entry

    entries = Entries()
    monkeypatch.setattr(lib, "kernels", lambda: entries)
    monkeypatch.setattr(ops, "_cuda", lambda *tensors: None)
    monkeypatch.setattr(ops, "_need", lambda cond, text: None)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "_sm_count", {0: 148})
    monkeypatch.setattr(ops, "_tc_plans", {})
    monkeypatch.setattr(ops, "_rows_plans", {})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    state = ops.LaunchState()
    previous = ops.use_state(state)
    yield noted
    ops.use_state(previous)


def _sizes(T, K=256, F=128):
    half = dict(dtype=torch.bfloat16)
    return {"x": torch.zeros(T, K), "norm": torch.ones(K), "h": torch.zeros(T, K, **half), "w": torch.zeros(2 * F, K, **half),
            "product": torch.zeros(T, 2 * F, **half), "gated": torch.zeros(T, F, **half)}


class _Asked(dict):
    def _ask(self, *args):
        raise AssertionError("a step of more rows asks for norms that wait")
    __contains__ = get = pop = _ask


@pytest.mark.parametrize("T", [9, 64, 131])
def test_more_rows_ask_nothing_of_the_rule_for_few(launches, monkeypatch, T):
    """Their launches are issued from Python whenever a step is not replayed, and each question costs host time."""
    monkeypatch.setattr(ops._S, "waiting_norms", _Asked())
    monkeypatch.setattr(ops, "_few_rows", lambda *args: pytest.fail("asked"))
    t = _sizes(T)
    ops.rmsnorm(t["x"], t["norm"], 1e-5, t["h"], may_wait=True)
    ops.linear_swiglu(t["h"], t["w"], t["gated"], tmp=t["product"])
    ops.linear_gated(t["h"], t["w"], t["gated"], "gelu_tanh", tmp=t["product"])
    ops.linear_unfolded(t["h"], t["w"], t["product"])
    monkeypatch.setattr(torch.Tensor, "is_cuda", True)
    ops.linear(t["h"], t["w"], t["product"])
    ops.forget_waiting(t["h"])
    assert launches[0] == "rmsnorm" and len(launches) >= 5


# ---- which norms may wait ------------------------------------------------------------------------------------------------------

def _block(norm_cls, mixer_cls):
    from imparo_b200.parts.base import Runtime, Workspace, register_part
    from imparo_b200.parts.block import PreNormResidualBlock
    from imparo_b200.parts.spec import LayerSpec, PartSpec
    register_part("norm", "few_rows_test", norm_cls, replace=True)
    register_part("mixer", "few_rows_test", mixer_cls, replace=True)
    cpu = torch.device("cpu")
    rt = Runtime(precision="bfloat16", device=cpu, workspace=Workspace(cpu))
    norm = PartSpec("few_rows_test", {"width": 64, "eps": 1e-5, "name": "n"})
    layer = LayerSpec(prefix="", mixer=PartSpec("few_rows_test", {}), mixer_norm=norm, feed_forward=None, feed_forward_norm=None)
    return PreNormResidualBlock({"layer": layer}, "", rt)


def _noting_parts():
    from imparo_b200.parts.base import Part
    noted = []

    class DocumentedNorm(Part):
        def forward(self, x32, rows=None, n_rows=None, tag="normed"):
            noted.append("documented")
            return x32.to(torch.bfloat16)

    class WaitingNorm(Part):
        def forward(self, x32, rows=None, n_rows=None, tag="normed", may_wait=False):
            noted.append(may_wait)
            return x32.to(torch.bfloat16)

    class Reader(Part):
        input_by_products = True

        def forward(self, x, batch, caches, residual):
            noted.append(tuple(x.shape))

    return noted, DocumentedNorm, WaitingNorm, Reader


def test_a_norm_with_the_documented_signature_runs(launches):
    noted, documented, waiting, reader = _noting_parts()
    x = torch.zeros(3, 64)
    _block(documented, reader).forward(x, None, ())
    assert noted == ["documented", (3, 64)]
    noted.clear()
    _block(waiting, reader).forward(x, None, ())
    assert noted == [True, (3, 64)]


def test_a_subclass_does_not_inherit_how_its_input_is_read(launches):
    noted, _, waiting, reader = _noting_parts()

    class ReadsItself(reader):
        def forward(self, x, batch, caches, residual):
            residual += x.float()

    class ReadsInAHelper(reader):
        pass

    class SaysSo(reader):
        input_by_products = True

    x = torch.zeros(3, 64)
    for cls, waits in ((ReadsItself, False), (ReadsInAHelper, False), (SaysSo, True), (reader, True)):
        noted.clear()
        block = _block(waiting, cls)
        block.forward(x, None, ())
        assert noted[0] is waits, cls
    from imparo_b200.parts.attention import AttentionMixer
    from imparo_b200.parts.base import reads_by_products
    from imparo_b200.parts.feedforward import SwiGLU
    from imparo_b200.parts.shortconv import ShortConvMixer
    for cls in (AttentionMixer, SwiGLU, ShortConvMixer):
        part = cls.__new__(cls)
        assert reads_by_products(part)
        part.forward = lambda *args: None
        assert not reads_by_products(part)


# ---- what becomes of a norm that waits -------------------------------------------------------------------------------------------

@pytest.mark.parametrize("product", ["linear", "linear_unfolded", "linear_swiglu", "linear_gated"])
def test_a_matrix_off_its_alignment_gets_the_norm_made(launches, monkeypatch, product):
    """A matrix that no own product takes goes to the library's, as for any other input; the norm is made first."""
    monkeypatch.setattr(torch.Tensor, "is_cuda", True)
    monkeypatch.setattr(ops, "_gemm_ws", {0: None})

    def need(cond, text):
        if not cond:
            raise ops.KernelError(text)
    monkeypatch.setattr(ops, "_need", need)
    t = _sizes(4)
    w = torch.zeros(t["w"].numel() + 4, dtype=torch.bfloat16)[4:].view(t["w"].shape)      # 8 bytes off
    assert w.data_ptr() % 16 == 8
    ops.rmsnorm(t["x"], t["norm"], 1e-5, t["h"], may_wait=True)
    assert launches == [] and t["h"].data_ptr() in ops._S.waiting_norms
    if product in ("linear", "linear_unfolded"):
        out = getattr(ops, product)(t["h"], w, t["product"])
        assert out is None or out is t["product"]
        tail = []
    elif product == "linear_swiglu":
        ops.linear_swiglu(t["h"], w, t["gated"], tmp=t["product"])
        tail = ["swiglu_act"]
    else:
        ops.linear_gated(t["h"], w, t["gated"], "gelu_tanh", tmp=t["product"])
        tail = ["gated_act"]
    assert launches == ["rmsnorm", "gemm_bf16_nt"] + tail and not ops._S.waiting_norms


@pytest.mark.parametrize("start", ["embed_gather", "embed_copies"])
def test_a_stream_that_starts_voids_what_a_step_left(launches, start):
    """A step that raised may leave a norm waiting; the next step's choice of kernels follows nothing of it, however the stream starts."""
    t = _sizes(4)
    ops.rmsnorm(t["x"], t["norm"], 1e-5, t["h"], may_wait=True)
    assert ops._S.waiting_norms and ops._S.rows_width == 256
    ids, table, status = torch.zeros(4, dtype=torch.int32), torch.zeros(9, 256, dtype=torch.bfloat16), torch.zeros(4, dtype=torch.int32)
    getattr(ops, start)(table, ids, t["x"], status)
    assert not ops._S.waiting_norms and ops._S.rows_width == 0


def test_another_norm_of_the_same_buffer_takes_the_place_of_one_that_waits(launches):
    t = _sizes(4)
    for again in (lambda: ops.group_rmsnorm(t["x"], t["norm"], 1e-5, 4, t["h"]),
                  lambda: ops.streams_norm(t["x"], 1, None, t["norm"], 1e-5, t["h"]),
                  lambda: ops.rmsnorm(t["x"], t["norm"], 1e-5, t["h"])):
        ops.rmsnorm(t["x"], t["norm"], 1e-5, t["h"], may_wait=True)
        launches.clear()
        again()
        assert not ops._S.waiting_norms
        ops.linear_swiglu(t["h"], t["w"], t["gated"])
        assert launches[1:] == ["gemm_rows"] and len(launches) == 2


def test_a_model_whose_embedding_is_its_own_starts_clean(launches):
    """An embedding that does not go through the launchers leaves the state to Model.forward."""
    from imparo_b200.parts.model import Model
    t = _sizes(4)
    ops.rmsnorm(t["x"], t["norm"], 1e-5, t["h"], may_wait=True)
    seen = []

    class Embedding:
        def forward(self, batch):
            seen.append((dict(ops._S.waiting_norms), ops._S.rows_width))
            return t["x"]
    model = Model.__new__(Model)
    model.embedding, model.schedule, model.rt = Embedding(), [], type("Rt", (), {"probe": None, "probe_now": False})()
    model.forward(None, None)
    assert seen == [({}, 0)]
