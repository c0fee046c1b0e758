"""How many token rows a decode step may have on two streams: the kernel on pairs of SMs, which takes projections of more than 128 rows, never runs
beside another stream's tensor-memory kernel."""
import contextlib

import pytest
import torch

SHAPE = dict(block_size=64, vocab_size=64, n_layer=2, n_head=4, n_local_heads=4, dim=1024, intermediate_size=96)


@contextlib.contextmanager
def _option(name, value):
    from gpt_fast import _C
    before = _C.option(name)
    _C.check(_C.lib.lri_set_option(name.encode(), value))
    try:
        yield
    finally:
        _C.check(_C.lib.lri_set_option(name.encode(), before))


def _engine(family, monkeypatch, batch, dim=1024):
    import gpt_fast
    from gpt_fast import gpt_ladder_TP, gpt_parallel_TP
    mod, cls = {"ladder": (gpt_ladder_TP, gpt_fast.GPTLadder), "parallel": (gpt_parallel_TP, gpt_fast.GPTParallel)}[family]
    monkeypatch.setitem(mod.transformer_configs, "two-streams-rows", dict(SHAPE, dim=dim))
    model = cls.from_name("two-streams-rows").to(torch.bfloat16).eval()
    model.setup_caches(max_batch_size=batch, max_seq_length=8)
    engine = model._engine
    engine.overlap_sublayers, engine.sms = True, 148
    return engine


@pytest.mark.parametrize("capturing", [False, True])
@pytest.mark.parametrize("family", ["ladder", "parallel"])
def test_rows_of_native_passes(family, capturing, monkeypatch):
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing)
    engine = _engine(family, monkeypatch, 130)
    assert [b for b in (64, 65, 128, 129, 130) if engine._two_streams(b)] == [64, 65, 128]
    engine.d = 512
    assert [b for b in (8, 9, 128, 129, 130) if engine._many_of_a_small_ladder(b)] == ([9, 128] if family == "ladder" else [])


def test_rows_of_the_python_schedule(monkeypatch):
    engine = _engine("ladder", monkeypatch, 130)
    ran = []
    monkeypatch.setattr(engine, "_run_ladder_two_streams", lambda rows, *a: ran.append(rows))
    monkeypatch.setattr(engine, "_norm", lambda *a, **k: None)
    monkeypatch.setattr(engine, "_attention", lambda *a, **k: None)
    monkeypatch.setattr(engine, "_mlp", lambda *a, **k: None)
    monkeypatch.setattr(engine, "_issue", lambda *a: None)
    for b in (1, 64, 65, 128, 129, 130):
        engine._run_ladder(b, b, 1, torch.zeros(1, dtype=torch.int32))
    assert ran == [1, 64, 65, 128]
    ran.clear()
    with _option("gemm_pair", 128):
        for b in (64, 65, 128):
            engine._run_ladder(b, b, 1, torch.zeros(1, dtype=torch.int32))
    assert ran == [64]


def test_two_streams_need_a_second_one():
    """Without one the kernels would go to the legacy stream, which no capture allows."""
    import ctypes
    from gpt_fast import _C
    some = (ctypes.c_void_p * 8)()
    for given in ({}, dict(events=ctypes.cast(some, ctypes.c_void_p)), dict(side=ctypes.addressof(some))):
        p = _C.LlamaPass(schedule=_C.PARALLEL_TWO_STREAMS, layers=ctypes.addressof(some), **given)
        assert _C.lib.lri_llama_run(ctypes.byref(p)) == -1 and b"second stream" in _C.lib.lri_last_error()


@pytest.mark.parametrize("family,few", [("ladder", list(range(1, 9))), ("parallel", list(range(1, 65)))])
def test_small_models_called_eagerly(family, few, monkeypatch):
    """One stream where the host is the limit: few sequences of a ladder model, any of parallel blocks; captured steps take two."""
    engine = _engine(family, monkeypatch, 64, dim=512)
    capturing = False
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing)
    assert [b for b in range(1, 65) if not (engine._two_streams(b) or engine._many_of_a_small_ladder(b))] == few
    capturing = True
    engine.hd = 64
    assert all(engine._two_streams(b) for b in range(1, 65))


@pytest.mark.parametrize("kv_heads,one", [(8, [1, 17, 18, 19, 20, 21, 22, 23]), (4, [1])])
def test_one_head_an_sm(kv_heads, one, monkeypatch):
    """Parallel blocks with about one 128-wide (sequence, head) pair an SM stay on one stream, but not where query heads share keys."""
    monkeypatch.setitem(SHAPE, "n_head", 8)
    monkeypatch.setitem(SHAPE, "n_local_heads", kv_heads)
    engine = _engine("parallel", monkeypatch, 64)
    assert engine.hd == 128
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    assert [b for b in range(1, 65) if not engine._two_streams(b)] == one
