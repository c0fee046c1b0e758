"""Decode steps of one sequence whose projections take the norm in front of them: the bits of the schedules that launch the norms, at one and several
chunks of a row, ragged ones, and the widest that are taken; wider models and captured steps keep their kernels."""
import pytest
import torch

from test_llama_pass_gpu import _model, _only

pytestmark = pytest.mark.gpu


def _steps(family, extra, dtype, native):
    from gpt_fast import _C
    model = _model(family, dtype, 1, **extra)
    _only(model._engine, native)
    out, launches = [], []
    with torch.no_grad():
        ids = torch.randint(0, 512, (1, 40), generator=torch.Generator().manual_seed(1)).cuda()
        model(ids, torch.arange(40, device="cuda"))
        for i in range(4):
            before = _C.lib.lri_launch_count()
            out.append(model(ids[:, i:i + 1].to(torch.int32), torch.tensor([40 + i], dtype=torch.int32, device="cuda")))
            launches.append(_C.lib.lri_launch_count() - before)
    kept = [c for layer in model.layers for c in (layer.attention.kv_cache.k_cache, layer.attention.kv_cache.v_cache)]
    del model
    return out + kept, launches


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("family,overlap", [("dense", True), ("ladder", True), ("ladder", False), ("parallel", True), ("desync", True)])
@pytest.mark.parametrize("dim,heads,inter", [(64, 1, 128), (128, 1, 136), (256, 4, 256), (512, 8, 264), (576, 9, 136), (768, 12, 256), (1024, 16, 512),
                                             (1024, 8, 264), (1088, 17, 128)])
def test_bits_of_separate_norms(family, overlap, dim, heads, inter, dtype):
    if family == "desync":
        pattern = dict(reduce_pattern=[{"attention": i % 2 == 0, "mlp": i == 1} for i in range(3)])
    else:
        pattern = {}
    extra = dict(dim=dim, n_head=heads, n_local_heads=heads, intermediate_size=inter, overlap=overlap, **pattern)
    (got, few), (want, many) = (_steps(family, extra, dtype, native) for native in (True, False))
    for a, b in zip(got, want):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b)
    # embedding, five launches a layer, final norm and head
    separate = 3 + (6 if family == "parallel" else 7) * 3
    assert few == [3 + 5 * 3 if dim <= 1024 else separate] * 4 and many[0] >= separate


def test_captured_and_eager_steps_are_the_same():
    model = _model("ladder", torch.bfloat16, 1, dim=768, n_head=12, n_local_heads=12, intermediate_size=512)
    tok, pos = torch.tensor([[3]], dtype=torch.int32, device="cuda"), torch.tensor([0], dtype=torch.int32, device="cuda")
    with torch.no_grad():
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            model(tok, pos)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            logits = model(tok, pos)
        for p in range(1, 120, 17):
            tok.fill_(p)
            pos.fill_(p)
            graph.replay()
            captured = logits.clone()
            assert torch.equal(captured, model(tok, pos))
