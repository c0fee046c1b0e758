"""Which passes the native call takes: only those whose layers have the sizes that it is given once for all."""
import pytest
import torch
import torch.nn.utils.parametrize

SHAPE = dict(block_size=64, vocab_size=64, n_layer=3, n_head=4, n_local_heads=2, dim=64, intermediate_size=96)


class Called(Exception):
    pass


def _model(family, monkeypatch):
    import gpt_fast
    from gpt_fast import gpt_dense_TP, gpt_desync_TP, gpt_ladder_TP, gpt_parallel_TP
    mod, cls = {"dense": (gpt_dense_TP, gpt_fast.GPTDense), "ladder": (gpt_ladder_TP, gpt_fast.GPTLadder),
                "parallel": (gpt_parallel_TP, gpt_fast.GPTParallel), "desync": (gpt_desync_TP, gpt_fast.GPTDesync)}[family]
    monkeypatch.setitem(mod.transformer_configs, "native-pass-sizes", dict(SHAPE))
    model = cls.from_name("native-pass-sizes").to(torch.bfloat16).eval()
    model.setup_caches(max_batch_size=2, max_seq_length=32)
    return model


def _narrow(layer, family, w1, w2):
    if family == "parallel":
        layer.attention.wqkv1.weight = torch.nn.Parameter(layer.attention.wqkv1.weight[: layer.attention.wqkv1.weight.shape[0] - w1])
        layer.attention.w2.weight = torch.nn.Parameter(layer.attention.w2.weight[:, : 96 - w2].contiguous())
    else:
        layer.feed_forward.w1.weight = torch.nn.Parameter(layer.feed_forward.w1.weight[: 192 - w1].contiguous())
        layer.feed_forward.w2.weight = torch.nn.Parameter(layer.feed_forward.w2.weight[:, : 96 - w2].contiguous())


def _shorter_cache(layer, family):
    cache = layer.attention.kv_cache
    cache.k_cache, cache.v_cache = cache.k_cache[:, :, :24].contiguous(), cache.v_cache[:, :, :24].contiguous()


def _other(name):
    def change(layer, family):
        owner = getattr(layer.attention, "wqkv1" if family == "parallel" and name == "wqkv" else name)
        owner.weight = torch.nn.Parameter(owner.weight[:, : owner.weight.shape[1] - 8].contiguous())
    return change


def _computed(layer, family):
    """A weight that is no plain parameter."""
    torch.nn.utils.parametrize.register_parametrization(layer.attention.wo, "weight", torch.nn.Identity())


CHANGES = {"computed weight": _computed, "narrower feed-forward": lambda la, f: _narrow(la, f, 16, 8), "w1 alone": lambda la, f: _narrow(la, f, 16, 0),
           "w2 alone": lambda la, f: _narrow(la, f, 0, 8), "cache": _shorter_cache, "wo": _other("wo"), "wqkv": _other("wqkv")}


@pytest.mark.parametrize("family", ["dense", "ladder", "parallel", "desync"])
@pytest.mark.parametrize("change", [None] + list(CHANGES))
@pytest.mark.parametrize("at", [0, 2])
def test_layers_of_other_sizes_stay_in_python(family, change, at, monkeypatch):
    model = _model(family, monkeypatch)
    engine = model._engine
    engine._splits = 1
    if change:
        CHANGES[change](model.layers[at], family)

    def called(*args, **kwargs):
        raise Called

    monkeypatch.setattr(torch.cuda, "current_stream", called)  # the next thing that it needs, a GPU's
    pos = torch.zeros(1, dtype=torch.int32)
    if change:
        assert engine._run_native(1, 1, pos) is False
    else:
        with pytest.raises(Called):
            engine._run_native(1, 1, pos)


@pytest.mark.parametrize("family", ["dense", "ladder"])
def test_another_number_of_layers_stays_in_python(family, monkeypatch):
    model = _model(family, monkeypatch)
    engine = model._engine
    engine._splits = 1
    for n in (2, 0):
        model.layers = model.layers[:n]
        assert engine._run_native(1, 1, torch.zeros(1, dtype=torch.int32)) is False


def test_ops_of_the_callers_own_are_called(monkeypatch):
    """An ops object derived from the package's own may replace any of its calls: it is not passed by."""
    from gpt_fast.ops import CudaOps

    class Own(CudaOps):
        pass

    engine = _model("dense", monkeypatch)._engine
    engine._splits, engine.ops = 1, Own
    assert engine._run_native(1, 1, torch.zeros(1, dtype=torch.int32)) is False


def test_the_pass_has_the_size_that_callers_know():
    """It has no field for its size: one more member would be read behind the struct of whoever was compiled without it."""
    import ctypes
    from gpt_fast import _C
    ints, wide, pointers, sizes = 12 + 1, 2, 2 + 3 + 8 + 5 + 3, 5
    assert ctypes.sizeof(_C.LlamaPass) == 4 * ints + 4 + 8 * (wide + pointers + sizes)
    assert _C.LlamaPass._fields_[-1][0] == "events"


def test_a_desync_pass_on_one_gpu_asks_no_layer_what_it_reduces(monkeypatch):
    """Its sums are the same whichever layers do; the walk over the layers bounds a small model's step."""
    model = _model("desync", monkeypatch)
    engine = model._engine
    engine._splits = 1
    for layer in model.layers:
        del layer.do_attention_all_reduce, layer.do_mlp_all_reduce

    def called(*args, **kwargs):
        raise Called

    monkeypatch.setattr(torch.cuda, "current_stream", called)
    with pytest.raises(Called):
        engine._run_native(1, 1, torch.zeros(1, dtype=torch.int32))
