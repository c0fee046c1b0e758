"""HGRN2 blocks on 256 threads (heads of up to 64 channels and 64 values): the edges of that shape, every number of segments, and the calls just
outside it, against the recurrence token by token in 64 bits."""
import pytest
import torch

from oracle import patevik_oracle as po

pytestmark = pytest.mark.gpu
EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}  # rounding of the stored results


def _rel(a, b):
    return ((a.double().cpu() - b).norm() / b.norm()).item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,S,H,C,E", [(1, 16, 1, 64, 64), (1, 17, 2, 4, 16), (2, 63, 3, 60, 48), (1, 128, 2, 64, 64), (1, 191, 2, 32, 64), (1, 333, 1, 64, 32),
                                       (1, 447, 2, 64, 64), (1, 528, 2, 64, 64), (3, 600, 16, 64, 64), (1, 300, 2, 68, 64), (1, 300, 2, 64, 80)])
def test_narrow_heads(dtype, B, S, H, C, E):
    from gpt_fast.ops import CudaOps as ops
    g = torch.Generator().manual_seed(S + C)

    def randn(*shape):
        return torch.randn(*shape, generator=g)

    ld = H * (2 * C + E) + 8
    ld += -ld % 8
    proj = randn(B * S, ld)
    q_off, f_off, v_off = 8, 8 + H * C, 8 + 2 * H * C
    fb, norm = randn(H * C).to(dtype), randn(E).to(dtype)
    low = (torch.rand(H * C, generator=g) * 0.98).to(dtype)
    st0 = randn(B, H, C, E)
    x = proj.double()
    q = torch.nn.functional.silu(x[:, q_off:f_off]).view(B, S, H, C)
    f = (low.double() + (1 - low.double()) * torch.sigmoid(x[:, f_off:v_off] + fb.double())).view(B, S, H, C)
    v = x[:, v_off:v_off + H * E].to(dtype).double().view(B, S, H, E)
    for pos0 in (0, 9):
        st, out = st0.clone().cuda(), torch.full((B * S, H * E), float("nan"), dtype=dtype, device="cuda")
        ws = torch.full((ops.hgrn2_workspace_bytes(dtype, B, S, H, C, E),), 255, dtype=torch.uint8, device="cuda")
        ops.hgrn2(proj.cuda(), ld, q_off, f_off, v_off, fb.cuda(), low.cuda(), norm.cuda(), 1e-4, st, torch.arange(pos0, pos0 + S).cuda(), out, B, S, H,
                  C, E, ws)
        for b in range(B):
            want, state = po.hgrn2_recurrence(q[b], f[b], v[b], st0[b].double() if pos0 else None)
            assert _rel(st[b], state) < 5e-6
            assert _rel(out.view(B, S, -1)[b], po.rms_norm(want, norm.double(), 1e-4).reshape(S, H * E)) < EPS[dtype]


# Few heads run on 512 threads; these, more (sequence, head) pairs than SMs or twice the segments that 512 threads would have, on 256: one segment and
# several, whole and ragged blocks, one wave and two.
MANY = [(1, 16, 160, 64, 64), (1, 17, 149, 4, 16), (2, 63, 80, 60, 48), (1, 191, 150, 32, 64), (1, 40, 300, 64, 64), (1, 333, 75, 64, 32), (1, 447, 37, 64, 64),
        (1, 528, 40, 64, 64)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,S,H,C,E", MANY)
def test_many_narrow_heads(dtype, B, S, H, C, E):
    test_narrow_heads(dtype, B, S, H, C, E)
