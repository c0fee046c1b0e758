"""Matrix-state recurrences in segments that run side by side, against the recurrence token by token in 64 bits: every number of segments, segments of
one stage and ragged last ones, from zero and from a state, and calls whose workspace is too small for them."""
import pytest
import torch

from oracle import migosun_oracle as mo
from test_migosun_gpu import _Delta, _randn, _rel

pytestmark = pytest.mark.gpu
# Everything is fp32: the bound of the one-segment form's own tests
BOUND = 3e-6


@pytest.fixture
def segments(monkeypatch):
    from gpt_fast import _C
    from gpt_fast.ops import CudaOps
    scan = CudaOps.state_scan
    ws = torch.full((64 << 20,), 255, dtype=torch.uint8, device="cuda")  # (NaN where nothing was written)
    state = {"bytes": ws.numel()}
    monkeypatch.setattr(CudaOps, "state_scan", staticmethod(lambda *a: scan(*a, workspace=ws[: state["bytes"]])))

    def choose(n, nbytes=ws.numel()):
        state["bytes"] = nbytes
        _C.check(_C.lib.lri_set_option(b"scan_segments", n))
    yield choose
    _C.check(_C.lib.lri_set_option(b"scan_segments", 0))
    assert _C.lib.lri_gemm_status() == 0


SIZES = [(1, 33, 2, 1, 12, 20), (2, 60, 4, 2, 64, 64), (1, 130, 2, 2, 128, 96), (1, 270, 3, 3, 48, 128), (1, 75, 1, 1, 100, 36)]


@pytest.mark.parametrize("n", [1, 2, 3, 7, 16])
@pytest.mark.parametrize("size", SIZES, ids=str)
def test_delta_rule(segments, size, n):
    B, S = size[:2]
    for bias in (-3.0, 3.0):
        segments(n)
        c = _Delta(torch.float32, *size, 4, 8, 8, bias)
        first = S // 3
        got = torch.cat([c.blocks(0, first), c.blocks(first, S - first)], 1)  # the second call goes on from the first one's state
        for b in range(B):
            out, st, _ = c.oracle(b)
            assert _rel(got[b], out) < BOUND and _rel(c.state[b], st) < BOUND


@pytest.mark.parametrize("n", [1, 2, 3, 7, 16])
@pytest.mark.parametrize("B,S,H,C,E", [(1, 33, 2, 12, 20), (2, 60, 3, 64, 128), (1, 270, 2, 128, 200), (1, 100, 1, 4, 4)])
def test_gated_linear_attention(segments, B, S, H, C, E, n):
    from gpt_fast.ops import CudaOps as ops
    segments(n)
    g = torch.Generator().manual_seed(S)
    ld = H * (2 * C + E)
    ld += -ld % 8
    proj, z, bias, st0 = _randn(g, B * S, ld), _randn(g, B * S, H * C), _randn(g, H * C), _randn(g, B, H, C, E)
    for pos0 in (0, 5):
        nb = B * ops.state_blocks(S)
        blocks = [torch.full((r, w), float("nan"), device="cuda") for r, w in ((4 * nb, H * C), (0, H * C), (4 * nb, H * C), (nb, H * C), (nb, H * 32))]
        state, o = st0.clone().cuda(), torch.full((B * S, H, E), float("nan"), device="cuda")
        x = proj.cuda()
        ops.gla_blocks(x, ld, (0, H * C), z.cuda(), bias.cuda(), 4.0, blocks, B, S, H, C)
        ops.state_scan(blocks, False, x.view(-1)[2 * H * C:], ld, state, torch.arange(pos0, pos0 + S).cuda(), o, B, S)
        p = proj.double().view(B, S, ld)
        for b in range(B):
            q, k, v = p[b, :, :H * C].view(S, H, C) * C ** -0.5, p[b, :, H * C:2 * H * C].view(S, H, C), p[b, :, 2 * H * C:2 * H * C + H * E].view(S, H, E)
            dec = torch.exp(torch.nn.functional.logsigmoid(z.double().view(B, S, H, C)[b] + bias.double().view(H, C)) / 4.0)
            out, st = mo.linear_attention_recurrence(q, k, v, dec, st0[b].double() if pos0 else None)
            assert _rel(o.view(B, S, H, E)[b], out) < BOUND and _rel(state[b], st) < BOUND


def test_chosen_segments_and_small_workspaces(segments):
    """The sizes from which segments are chosen; a workspace that is too small gives the one-segment result."""
    from gpt_fast.ops import CudaOps as ops
    assert ops.state_scan_workspace_bytes(1, 1199, 16, 64, 64, True) == 0 and ops.state_scan_workspace_bytes(1, 447, 16, 64, 128, False) == 0
    need = ops.state_scan_workspace_bytes(1, 1216, 2, 64, 64, True)
    assert need > 0 and ops.state_scan_workspace_bytes(1, 4096, 16, 64, 64, True) >= ops.state_scan_workspace_bytes(1, 1300, 16, 64, 64, True)
    results = []
    for nbytes in (need, need - 4, 0):
        segments(0, nbytes)
        c = _Delta(torch.float32, 1, 1216, 2, 1, 64, 64, 4, 8, 8, -3.0)
        got = c.blocks(0, 1216)
        out, st, _ = c.oracle(0)
        assert _rel(got[0], out) < BOUND and _rel(c.state[0], st) < BOUND
        results.append(got)
    assert torch.equal(results[1], results[2]) and not torch.equal(results[0], results[1])
