"""Who lets the kernel behind a small-batch projection in before its sums: passes that know that nothing of another stream runs beside it, never the plain
entry points, which the Python schedules call (the ladder's two streams among them)."""
import pytest
import torch

import migosun_util as mu
import patevik_util as pu


class _Recorder:
    def __init__(self, lib):
        self.lib, self.calls = lib, []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append(name)
            return 0
        return call


PLAIN = ["lri_linear", "lri_linear_f32", "lri_gateup_glu"]


def test_only_who_asks(monkeypatch):
    from gpt_fast import _C
    from gpt_fast.ops import CudaOps, OneSmOps
    monkeypatch.setattr(_C, "require_cuda", lambda *t: None)
    monkeypatch.setattr(_C, "stream_handle", lambda: 0)
    x, w, y = torch.zeros(16, 16), torch.zeros(32, 16), torch.zeros(16, 32)
    for ops in (CudaOps, OneSmOps):
        for kw, names in (({}, PLAIN), (dict(early=True), [n + "_early" for n in PLAIN])):
            lib = _Recorder(_C.lib)
            with monkeypatch.context() as m:
                m.setattr(_C, "lib", lib)
                ops.linear(x, w, y, 16, **kw)
                ops.linear_f32(x, w, y, 16, **kw)
                ops.gateup_glu(x, w, y, 16, (1.0, 1.0, 1.0), **kw)
            assert lib.calls == names


def test_plain_calls_of_the_two_stream_schedule(monkeypatch):
    """The ladder's Python form on two streams, as it runs with several ranks."""
    import gpt_fast
    from gpt_fast import _C, gpt_ladder_TP
    monkeypatch.setitem(gpt_ladder_TP.transformer_configs, "early-start", dict(block_size=64, vocab_size=64, n_layer=2, n_head=4, n_local_heads=4, dim=64,
                                                                             intermediate_size=96))
    model = gpt_fast.GPTLadder.from_name("early-start").to(torch.bfloat16).eval()
    model.setup_caches(max_batch_size=16, max_seq_length=8)
    engine, lib = model._engine, _Recorder(_C.lib)

    class Event:
        def record(self, *a):
            pass
    import contextlib
    engine.overlap_sublayers, engine._events, engine._splits = True, [Event()] * 8, 1
    engine.side_stream = type("", (), {"wait_event": lambda self, e: None})()
    engine.normed_m = engine.normed
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: engine.side_stream)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(_C, "require_cuda", lambda *t: None)
    monkeypatch.setattr(_C, "stream_handle", lambda: 0)
    monkeypatch.setattr(_C, "lib", lib)
    engine._run_ladder(16, 16, 1, torch.zeros(1, dtype=torch.int32))
    assert lib.calls.count("lri_linear") == 4 and not [n for n in lib.calls if n.endswith("_early")]


@pytest.mark.parametrize("util,eagerly", [(mu, True), (pu, False)])
def test_which_layer_engines_ask(util, eagerly):
    from gpt_fast.ops import CudaOps
    case = next(iter(util.CONFIGS.values()))
    engine = util.build(case[0] if util is mu else case, util.weights(case), torch.bfloat16, "cpu", 1, 16)._engine
    assert engine._nothing_beside() is eagerly

    class Own(CudaOps):
        pass
    engine.ops = Own
    assert not engine._nothing_beside()


@pytest.mark.gpu
@pytest.mark.parametrize("util,eagerly", [(mu, {"early": True}), (pu, {})])
def test_experts_ask_in_captures_alone(util, eagerly):
    case = next(iter(util.CONFIGS.values()))
    model = util.build(case[0] if util is mu else case, util.weights(case), torch.bfloat16, "cuda", 16, 16)
    tok, pos = torch.zeros(16, 1, dtype=torch.int32, device="cuda"), torch.tensor([0], dtype=torch.int32, device="cuda")
    with torch.no_grad():
        eager = model(tok, pos)
        assert model._engine.alone == eagerly
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            logits = model(tok, pos)
        assert model._engine.alone == {"early": True}
        graph.replay()
        assert torch.equal(eager, logits)
        model(tok, pos)
        assert model._engine.alone == eagerly


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [9, 16, 17, 33, 64])
def test_same_bits(dtype, rows):
    """Chains of projections, each on its own or with the next let in early."""
    from gpt_fast import _C
    from gpt_fast.ops import CudaOps as ops
    g = torch.Generator(device="cuda").manual_seed(rows)

    def randn(*shape, scale=1.0):
        return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)
    d, ff = 520, 1000
    x0, w1, w2, w3 = randn(rows, d), randn(2 * ff, d, scale=d ** -0.5), randn(d, ff, scale=ff ** -0.5), randn(d, d, scale=d ** -0.5)
    ws = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")
    results = []
    for early in (False, True):
        x, h, y, f = x0.clone(), randn(rows, ff), torch.zeros_like(x0), torch.zeros(rows, d, device="cuda")
        for _ in range(20):
            ops.gateup_glu(x, w1, h, rows, (1.7, 7.0, 1.0), workspace=ws[: 16 << 20], early=early)
            ops.linear(h, w2, y, rows, addend=x, workspace=ws[16 << 20: 32 << 20], early=early)
            ops.linear_f32(y, w3, f, rows, workspace=ws[32 << 20:], early=early)
            ops.linear(y, w3, x, rows, workspace=ws[:16 << 20], early=early)
        results.append((x, f))
    for a, b in zip(*results):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b)
    assert _C.lib.lri_gemm_status() == 0
