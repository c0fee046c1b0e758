"""The layers of a pass launched by one native call against the same schedule launched call by call: bit for bit, for every schedule, decode
and prompt, and errors of the entry points below reach the caller."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPE = dict(block_size=256, vocab_size=512, n_layer=3, n_head=4, n_local_heads=2, dim=256, intermediate_size=512, rope_base=500000)


def _model(family, dtype, batch, overlap=True, **extra):
    import gpt_fast
    from gpt_fast import gpt_dense_TP, gpt_desync_TP, gpt_ladder_TP, gpt_parallel_TP
    mod, cls = {"dense": (gpt_dense_TP, gpt_fast.GPTDense), "ladder": (gpt_ladder_TP, gpt_fast.GPTLadder),
                "parallel": (gpt_parallel_TP, gpt_fast.GPTParallel), "desync": (gpt_desync_TP, gpt_fast.GPTDesync)}[family]
    mod.transformer_configs["native-pass"] = dict(SHAPE, **extra)
    with torch.device("meta"):
        model = cls.from_name("native-pass")
    model = model.to(dtype=dtype).to_empty(device="cuda").eval()
    g = torch.Generator(device="cuda").manual_seed(5)
    with torch.no_grad():
        for name, p in model.named_parameters():
            p.normal_(1.0 if "norm" in name else 0.0, 0.1, generator=g)
    with torch.device("cuda"):
        model.setup_caches(max_batch_size=batch, max_seq_length=200)
    if family == "ladder":
        model._engine.overlap_sublayers = overlap
    return model


def _only(engine, native):
    """Passes of this engine run in the native call alone, or never there."""
    if not native:
        engine._run_native = lambda *a: False
        return

    def refuse(*a):
        raise AssertionError("the Python schedule ran")
    engine._run_dense = engine._run_ladder = engine._run_parallel = engine._run_desync = refuse


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch", [1, 3, 20])
@pytest.mark.parametrize("family,extra", [("dense", {}), ("ladder", {}), ("ladder", {"overlap": False}), ("parallel", {}), ("desync", {}),
                                          ("desync", {"reduce_pattern": [{"attention": i % 2 == 0, "mlp": i == 1} for i in range(3)]})])
def test_native_pass_equals_calls(dtype, batch, family, extra):
    results = []
    for native in (True, False):
        model = _model(family, dtype, batch, **extra)
        _only(model._engine, native)
        ids = torch.randint(0, SHAPE["vocab_size"], (batch, 70), generator=torch.Generator().manual_seed(1)).cuda()
        out = []
        with torch.no_grad():
            out.append(model(ids, torch.arange(70, device="cuda")))
            for i in range(3):
                out.append(model(ids[:, i:i + 1].to(torch.int32), torch.tensor([70 + i], dtype=torch.int32, device="cuda")))
        results.append(out)
    for a, b in zip(*results):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b)


def test_weights_are_read_for_every_pass_and_errors_arrive():
    model = _model("dense", torch.bfloat16, 1)
    _only(model._engine, True)
    tok, pos = torch.tensor([[3]], dtype=torch.int32, device="cuda"), torch.tensor([0], dtype=torch.int32, device="cuda")
    with torch.no_grad():
        first = model(tok, pos)
        ff = model.layers[1].feed_forward
        ff.w2.weight = torch.nn.Parameter(ff.w2.weight * 2)
        assert not torch.equal(first, model(tok, pos))
        ff.w2.weight = torch.nn.Parameter(torch.empty(ff.w2.weight.numel() + 4, dtype=torch.bfloat16, device="cuda")[4:].view_as(ff.w2.weight))
        with pytest.raises(RuntimeError, match="aligned"):
            model(tok, pos)
        ff.w2.weight = torch.nn.Parameter(ff.w2.weight.detach().cpu())
        with pytest.raises(RuntimeError, match="CUDA"):
            model(tok, pos)
    torch.cuda.synchronize()


def test_layers_of_unequal_sizes_run_as_before():
    """A narrower feed-forward in one layer and a shorter cache in another: read at their own sizes."""
    results = []
    for native in (True, False):
        model = _model("dense", torch.bfloat16, 2)
        engine = model._engine
        if not native:
            engine._run_native = lambda *a: False
        ff, cache = model.layers[1].feed_forward, model.layers[2].attention.kv_cache
        up, gate = ff.w1.weight.detach().chunk(2)
        ff.w1.weight = torch.nn.Parameter(torch.cat([up[:384], gate[:384]]))
        ff.w2.weight = torch.nn.Parameter(ff.w2.weight.detach()[:, :384].contiguous())
        cache.k_cache, cache.v_cache = cache.k_cache[:, :, :96].contiguous(), cache.v_cache[:, :, :96].contiguous()
        ids = torch.randint(0, SHAPE["vocab_size"], (2, 80), generator=torch.Generator().manual_seed(2)).cuda()
        out = []
        with torch.no_grad():
            out.append(model(ids, torch.arange(80, device="cuda")))
            for i in range(3):
                out.append(model(ids[:, i:i + 1].to(torch.int32), torch.tensor([80 + i], dtype=torch.int32, device="cuda")))
        results.append(out)
    torch.cuda.synchronize()
    for a, b in zip(*results):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b)
