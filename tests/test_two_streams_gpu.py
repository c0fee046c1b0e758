"""Decode passes whose layers run on two streams: captured steps (two streams, half of the ring in the small-batch projections) against eager ones of the same
small model (one stream, whole ring), bit for bit, many replays behind one another; and the rule that chooses."""
import pytest
import torch

from test_llama_pass_gpu import _model, _only

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch", [1, 2, 5, 8, 9, 16, 17, 33, 64])
@pytest.mark.parametrize("family", ["ladder", "parallel"])
@pytest.mark.parametrize("sizes", [{}, dict(dim=960, n_head=15, n_local_heads=5, intermediate_size=2056)], ids=["256", "960"])
def test_captured_steps_on_two_streams(family, batch, dtype, sizes):
    model = _model(family, dtype, batch, **sizes)
    engine = model._engine
    _only(engine, True)
    tok = torch.randint(0, 512, (batch, 1), generator=torch.Generator().manual_seed(1)).to(torch.int32).cuda()
    pos = torch.tensor([0], dtype=torch.int32, device="cuda")
    assert engine.overlap_sublayers and not engine._two_streams(batch)
    with torch.no_grad():
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            model(tok, pos)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            assert engine._two_streams(batch)
            logits = model(tok, pos)
        for p in (1, 2, 40, 150):
            pos.fill_(p)
            for _ in range(5):
                graph.replay()
            captured = logits.clone()
            assert torch.isfinite(captured.float()).all() and torch.equal(captured, model(tok, pos))
    torch.cuda.synchronize()
    from gpt_fast import _C
    assert _C.lib.lri_gemm_status() == 0


def test_choice_of_streams():
    """Wide models take two streams eagerly too; parallel blocks not where attention has about one 128-wide pair an SM."""
    engine = _model("parallel", torch.bfloat16, 2, dim=2048, n_head=16, n_local_heads=16, intermediate_size=512)._engine
    engine.sms = 148
    assert [b for b in range(1, 65) if not engine._two_streams(b)] == [1, 9, 10, 11]
    engine.hd = 64
    assert [b for b in range(1, 65) if not engine._two_streams(b)] == [1]
    engine = _model("ladder", torch.bfloat16, 2, dim=2048, n_head=16, n_local_heads=16, intermediate_size=512)._engine
    assert all(engine._two_streams(b) for b in range(1, 65))
    assert not _model("dense", torch.bfloat16, 2)._engine._two_streams(1)


@pytest.mark.parametrize("family", ["ladder", "parallel"])
def test_more_rows_run_on_one_stream(family):
    """Whoever asks for two streams with more rows than they are made for gets one: no event is recorded, and the results are those of one stream."""
    results = []
    for asked in (False, True):
        model = _model(family, torch.bfloat16, 129)
        engine = model._engine
        _only(engine, True)
        engine._two_streams = lambda B: asked
        engine._events = [type("", (), {"cuda_event": None})()] * 8
        tok = torch.arange(129, dtype=torch.int32, device="cuda").view(129, 1)
        with torch.no_grad():
            results.append(model(tok, torch.tensor([0], dtype=torch.int32, device="cuda")))
    assert torch.isfinite(results[0].float()).all() and torch.equal(*results)


def test_parallel_passes_of_one_stream_read_no_events(monkeypatch):
    """LRI_PARALLEL with events and without a second stream: one stream, as before there was a schedule of two."""
    from gpt_fast.ops import CudaOps
    run, null = CudaOps.run_layers, [type("", (), {"cuda_event": None})()] * 8
    tok, pos = torch.arange(9, dtype=torch.int32, device="cuda").view(9, 1), torch.tensor([0], dtype=torch.int32, device="cuda")
    results = []
    for events in (None, null):
        model = _model("parallel", torch.bfloat16, 9)
        _only(model._engine, True)

        def given(schedule, layers, above, _, main, side, *rest, **kw):
            assert side is None
            return run(schedule, layers, above, events, main, None, *rest, **kw)
        monkeypatch.setattr(CudaOps, "run_layers", staticmethod(given))
        with torch.no_grad():
            results.append(model(tok, pos))
    assert torch.isfinite(results[0].float()).all() and torch.equal(*results)


@pytest.mark.parametrize("family,batches", [("ladder", [2, 3, 4, 5, 8, 20]), ("parallel", [2, 8, 9, 20, 33, 40, 49])])
def test_large_projections_beside_each_other(family, batches):
    """Projections of 15 M weights and more take the small-batch kernel from two rows on, so that its rings of every length run beside another stream's:
    eager and captured steps on two streams against one, bit for bit."""
    from gpt_fast import _C
    for batch in batches:
        model = _model(family, torch.bfloat16, batch, n_layer=2, dim=2048, n_head=16, n_local_heads=8, intermediate_size=8192)
        engine = model._engine
        _only(engine, True)
        tok = torch.randint(0, 512, (batch, 1), generator=torch.Generator().manual_seed(1)).to(torch.int32).cuda()
        pos = torch.tensor([0], dtype=torch.int32, device="cuda")

        def step(overlap):
            engine.overlap_sublayers = overlap
            assert engine._two_streams(batch) is overlap
            return model(tok, pos)
        with torch.no_grad():
            for p in range(3):  # (each writes the row that the next ones read)
                pos.fill_(p)
                got, want = step(True), step(False)
                assert torch.isfinite(got.float()).all() and torch.equal(got, want)
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                logits = step(True)
            torch.cuda.current_stream().wait_stream(side)
            for p in (3, 50):
                pos.fill_(p)
                for _ in range(5):
                    graph.replay()
                captured = logits.clone()
                assert torch.equal(captured, step(False))
        torch.cuda.synchronize()
        assert _C.lib.lri_gemm_status() == 0
        del model, graph
