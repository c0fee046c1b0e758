"""Prompt passes of designs with side-by-side mixers, whose attention runs on a second stream: no projection of theirs takes the kernel on
pairs of SMs, and passes that follow one another without a wait finish with the first one's results."""
import pytest
import torch

import migosun_util as mu
import patevik_util as pu


class _Recorder:
    def __init__(self, lib):
        self.lib, self.dtypes = lib, {}

    def __getattr__(self, name):
        if name not in ("lri_linear", "lri_linear_f32", "lri_gateup_glu"):
            return getattr(self.lib, name)
        return lambda dtype, *args: self.dtypes.setdefault(name, dtype) and 0


def test_projections_ask_for_single_sms(monkeypatch):
    from gpt_fast import _C
    from gpt_fast.ops import CudaOps, OneSmOps
    monkeypatch.setattr(_C, "require_cuda", lambda *t: None)
    monkeypatch.setattr(_C, "stream_handle", lambda: 0)
    x, w, y = torch.zeros(200, 16), torch.zeros(32, 16), torch.zeros(200, 32)
    for ops, flag in ((CudaOps, 0), (OneSmOps, _C.ONE_SM)):
        lib = _Recorder(_C.lib)
        monkeypatch.setattr(_C, "lib", lib)
        ops.linear(x, w, y, 200, workspace=None)
        ops.linear_f32(x, w, y, 200, workspace=None)
        ops.gateup_glu(x, w, y, 200, (1.0, 1.0, 1.0), workspace=None)
        assert lib.dtypes == {k: _C.FP32 | flag for k in ("lri_linear", "lri_linear_f32", "lri_gateup_glu")}
        monkeypatch.setattr(_C, "lib", lib.lib)


def test_the_flag_is_no_type():
    from gpt_fast import _C
    for fn, tail in ((_C.lib.lri_linear, (None, None, None, None, 0, 8, 8, None, 0, None)), (_C.lib.lri_linear_f32, (None, None, None, 0, 8, 8, None, 0, None)),
                     (_C.lib.lri_gateup_glu, (None, None, None, 0, 8, 8, 1.0, 1.0, 1.0, None, 0, None))):
        for dtype in (-1, 3, _C.ONE_SM + 3, 2 * _C.ONE_SM):
            assert fn(dtype, *tail) == -3  # unsupported type
        assert fn(_C.ONE_SM, *tail) == -1  # a known type: the NULL pointers are what is refused


def test_which_designs_stay_on_single_sms():
    from gpt_fast.ops import CudaOps, OneSmOps
    case = mu.CONFIGS["tiles"]
    model = mu.build(case[0], mu.weights(case), torch.bfloat16, "cpu", 1, 16)
    assert model._engine.ops is OneSmOps
    case = next(iter(pu.CONFIGS.values()))
    model = pu.build(case, pu.weights(case), torch.bfloat16, "cpu", 1, 16)
    assert model._engine.ops is CudaOps


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,tokens", [(2, 1500), (3, 333)])
def test_passes_behind_one_another(dtype, batch, tokens):
    from gpt_fast import _C
    case = mu.config(1024, 640, 3, [(mu.side_by_side((16, 4, 64, 64, 4096, 32, 1e4, 0.2), (8, 8, 64, 64, 4, (16, 64))), mu.dense(2048)),
                                    (mu.side_by_side((16, 4, 64, 64, 256, 64, 1e4, 0.2), (8, 4, 64, 64, 4, (64, 16))), mu.dense(2048))])
    model = mu.build(case[0], mu.weights(case, 3), dtype, "cuda", batch, tokens)
    ids = torch.stack([mu.tokens(case[0], tokens, i) for i in range(batch)]).cuda()
    pos = torch.arange(tokens, device="cuda")
    with torch.no_grad(), torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        first = model(ids, pos)
        torch.cuda.synchronize()
    names = [e.key for e in prof.key_averages()]
    assert any("window_attention_tc" in n for n in names) and any("gemm_tcgen05" in n for n in names)
    assert not any("gemm_pair" in n for n in names)
    with torch.no_grad():
        for _ in range(40):
            last = model(ids, pos)
    torch.cuda.synchronize()
    _C.check(_C.lib.lri_gemm_status())
    assert torch.isfinite(first.float()).all() and torch.equal(first, last)
