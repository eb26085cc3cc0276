"""32-bit products whose operands are cut beforehand: the bits of the product that cuts them itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def both(x, w, base=None):
    from imparo_b200.kernels import lib, ops as o
    M, K = x.shape
    N = w.shape[0]
    outs = []
    st = o.new_status(DEV)
    for cut in (False, True):
        out = torch.full((M, N), 3.0, device=DEV) if base is None else base.clone()
        args = (x.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, x.stride(0), N, int(base is not None))
        stream = torch.cuda.current_stream().cuda_stream
        if cut:
            n = lib.kernels().imparo_sgemm_cut_bytes(M, N, K)
            assert n > 0
            scratch = torch.full((n + 64,), 255, dtype=torch.uint8, device=DEV)              # (every 16 bits a NaN)
            assert lib.kernels().imparo_sgemm_cut(*args, scratch.data_ptr(), st.data_ptr(), stream) == 0
            assert bool((scratch[n:] == 255).all())
        else:
            assert lib.kernels().imparo_sgemm_nt(*args, st.data_ptr(), stream) == 0
        outs.append(out)
    o.read_status(st)
    return outs


def same(a, b):
    return torch.equal(a.view(torch.int32), b.view(torch.int32))


# tiles of 128 rows and 64 or 128 columns and their edges; K: less than a stretch of 64, no multiple of 8, several stretches
@pytest.mark.parametrize("M", [1, 65, 129, 1000])
@pytest.mark.parametrize("N,K", [(1, 4), (63, 60), (130, 68), (1024, 516), (1300, 1024)])
def test_the_same_bits(M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    x, w = torch.randn(M, K + 8, generator=g).to(DEV)[:, 4:4 + K], torch.randn(N, K, generator=g).to(DEV)
    a, b = both(x, w)
    assert same(a, b)
    want = x.double() @ w.double().T
    assert (b.double() - want).norm() <= 1e-6 * want.norm()
    a, b = both(x, w, base=torch.randn(M, N, generator=g).to(DEV))
    assert same(a, b)


def test_operands_at_the_ends_of_the_range():
    g = torch.Generator().manual_seed(5)
    x, w = torch.randn(300, 256, generator=g).to(DEV), torch.randn(200, 256, generator=g).to(DEV)
    x[3] *= 2.0 ** -130
    x[5, 7], x[6, 9], x[299, 0] = float("inf"), float("nan"), 3.4e38
    w[11] *= 2.0 ** -125
    w[0, 3], w[199, 255] = float("-inf"), 3.4e38
    a, b = both(x, w)
    assert same(a.nan_to_num(7.0), b.nan_to_num(7.0)) and torch.equal(a.isnan(), b.isnan())


def test_the_rule_and_the_room(monkeypatch):
    """Where the scratch is too small, or is not there, the product cuts its operands itself; what both launch gives the same bits."""
    from imparo_b200.kernels import ops as o
    assert o._cut_pays(1000, 9216, 1024) and o._cut_pays(65, 1024, 4608)
    assert not o._cut_pays(64, 1024, 4608) and not o._cut_pays(65, 9216, 1024) and not o._cut_pays(257, 16384, 2048)
    state = o.LaunchState()
    old = o.use_state(state)
    try:
        x, w = torch.randn(500, 512, device=DEV), torch.randn(640, 512, device=DEV)
        outs = [torch.empty(500, 640, device=DEV) for _ in range(3)]
        assert o._cut_scratch(x, w) is None
        o.linear(x, w, outs[0])
        o.prepare_cut(DEV, 499, [(640, 512)])
        assert o._cut_scratch(x, w) is None
        o.linear(x, w, outs[1])
        o.prepare_cut(DEV, 500, [(640, 512), (1 << 20, 4096)])
        assert o._cut_scratch(x, w) is not None
        o.linear(x, w, outs[2])
        assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    finally:
        o.use_state(old)


def test_a_model_with_cut_operands_and_without():
    """The engine's switch: a 32-bit prompt and a mixed step give the same bits either way, through other launches."""
    from imparo_b200.engine import Engine, StepItem
    from imparo_b200.kernels import ops as o
    cfg = {"architectures": ["Lfm2ForCausalLM"], "vocab_size": 512, "hidden_size": 512, "num_hidden_layers": 2,
           "layer_types": ["conv", "full_attention"], "num_attention_heads": 8, "num_key_value_heads": 4, "block_ff_dim": 2048,
           "block_auto_adjust_ff_dim": False, "conv_L_cache": 3, "conv_bias": False, "rope_theta": 1000000.0, "norm_eps": 1e-5,
           "tie_embedding": True, "max_position_embeddings": 2048}
    tokens = torch.arange(700).remainder(509).tolist()
    outs, launched = [], []
    for on in (True, False):
        eng = Engine(config=cfg, seed=3, dtype="float32", ctx=1024, parallel=3, page_size=16, max_step_tokens=1024, switches={"cut_f32": on})
        assert bool(eng.rt.launch_state.planes) == on
        before = o.COUNTS["own"]
        eng.add_request(1)
        eng.add_request(2)
        rows = [eng.step([StepItem(1, tokens[:600], list(range(600)))]),
                eng.step([StepItem(1, tokens[600:601], [0]), StepItem(2, tokens[:300], [0, 299])])]
        eng.check_device_status()
        outs.append(torch.cat(rows).cpu())
        launched.append(o.COUNTS["own"] - before)
        del eng
    assert same(*outs) and launched[0] > launched[1]
