"""The output projection of few sequences: on the streaming kernel whatever its size, whole and in the slices of the greedy and sampled
heads."""
import types

import pytest
import torch

ROWS = [1, 2, 5, 8, 9, 16]


def _recorded(monkeypatch, dim=32, vocab=64):
    """An engine whose trunk does nothing and whose projections are written down."""
    from gpt_fast.engine import Engine
    calls = []

    class Ops:
        @staticmethod
        def linear(x, w, out, rows, addend=None, workspace=None):
            calls.append((rows, workspace))
            out.view(-1)[: rows * w.shape[0]] = torch.arange(rows * w.shape[0]).to(out.dtype) % 7

    cfg = types.SimpleNamespace(dim=dim, vocab_size=vocab)
    model = types.SimpleNamespace(config=cfg, output=types.SimpleNamespace(weight=torch.zeros(vocab, dim)))
    engine = Engine(model, "dense", ops=Ops, comm=types.SimpleNamespace(world=1, rank=0))
    engine.d, engine.dtype, engine.max_batch, engine.fused_head = dim, torch.float32, 16, False
    engine.resid = engine.normed = torch.zeros(64, dim)
    engine.ws_head = torch.zeros(8, dtype=torch.uint8)
    engine.vocab_lo, engine.vocab_hi = 0, vocab
    engine.head_logits, engine.head_best = torch.zeros(16 * vocab), torch.zeros(1, 16, 2)
    monkeypatch.setattr(engine, "_trunk", lambda idx, pos: (idx.shape[0], idx.shape[1], idx.numel()))
    return engine, calls


@pytest.mark.parametrize("stream_rows", [4, 8])
@pytest.mark.parametrize("rows", ROWS)
def test_which_calls_get_a_workspace(rows, stream_rows, monkeypatch):
    from gpt_fast import _C
    engine, calls = _recorded(monkeypatch)
    _C.check(_C.lib.lri_set_option(b"stream_rows", stream_rows))
    try:
        one = torch.zeros(rows, 1, dtype=torch.int32)
        engine.forward(one, None)
        engine.forward_last(torch.zeros(rows, 3, dtype=torch.int32), None)
        engine.forward_greedy(one, None)
        engine.forward_sample(one, None)
    finally:
        _C.check(_C.lib.lri_set_option(b"stream_rows", 8))
    assert len(calls) == 4
    for n, workspace in calls:
        assert n == rows and (workspace is None if rows <= stream_rows else workspace is engine.ws_head)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_large_vocabulary(dtype):
    """32000 rows of 4096, which as a layer's projection would take the stream-K kernel: logits as the streaming kernel gives them, slices
    and arg-max up to one rounding."""
    import gpt_fast
    from gpt_fast import gpt_dense_TP
    from gpt_fast.ops import CudaOps as ops
    gpt_dense_TP.transformer_configs["large-head"] = dict(block_size=64, vocab_size=32000, n_layer=1, n_head=32, n_local_heads=8, dim=4096,
                                                          intermediate_size=512)
    with torch.device("meta"):
        model = gpt_fast.GPTDense.from_name("large-head")
    model = model.to(dtype=dtype).to_empty(device="cuda").eval()
    g = torch.Generator(device="cuda").manual_seed(11)
    with torch.no_grad():
        for name, p in model.named_parameters():
            p.normal_(1.0 if "norm" in name else 0.0, 0.1 if "norm" in name else p.shape[-1] ** -0.5, generator=g)
    with torch.device("cuda"):
        model.setup_caches(max_batch_size=9, max_seq_length=32)
    w, engine = model.output.weight, model._engine
    ulp = 2.0 ** (-7 if dtype == torch.bfloat16 else -10)
    for rows in (2, 5, 8, 9):
        tok = torch.randint(0, 32000, (rows, 1), dtype=torch.int32, device="cuda", generator=g)
        pos = torch.tensor([3], dtype=torch.int32, device="cuda")
        with torch.no_grad(), torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            logits = model(tok, pos)
            torch.cuda.synchronize()
        last = max((e for e in prof.events() if "lri::" in e.name), key=lambda e: e.time_range.start)
        assert ("streamk" in last.name) == (rows > 8), last.name
        want = engine.normed[:rows].double() @ w.double().T
        assert ((logits[:, 0].double() - want).abs() <= ulp * want.abs() + 1e-4).all()
        if rows <= 8:
            for lo, hi in ((0, 32000), (0, 16000), (16000, 32000), (28000, 32000)):
                part = torch.empty(rows, hi - lo, dtype=dtype, device="cuda")
                ops.linear(engine.normed, w[lo:hi], part, rows)
                if hi - lo == 32000:
                    assert torch.equal(part, logits[:, 0])
                assert ((part.double() - logits[:, 0, lo:hi].double()).abs() <= ulp * want[:, lo:hi].abs() + 1e-4).all()
        with torch.no_grad():
            got = model.decode_greedy(tok, pos)
        best = want.amax(-1)
        assert (want.gather(1, got.long())[:, 0] >= best - 2 * ulp * best.abs()).all()
    torch.cuda.synchronize()
