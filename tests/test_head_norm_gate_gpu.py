"""Norm and gate of a recurrence's results at the edges of the vector form (heads of 4 to 256 values, pitches and first columns in whole vectors) and
just outside it, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = {torch.float32: 1e-6, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}  # rounding of the stored results


@pytest.mark.parametrize("dtype", list(EPS))
@pytest.mark.parametrize("act", ["sigmoid", "silu"])
@pytest.mark.parametrize("rows,H,E,shift", [(1, 1, 4, 0), (7, 3, 64, 0), (5, 2, 68, 8), (33, 16, 128, 4), (2, 5, 252, 8), (3, 1, 256, 0), (3, 1, 260, 0), (9, 2, 66, 0),
                                            (4, 3, 64, 1), (4, 3, 64, 2)])
def test_head_norm_gate(dtype, act, rows, H, E, shift):
    from gpt_fast.ops import CudaOps as ops
    g = torch.Generator(device="cuda").manual_seed(rows + E)
    o, w = torch.randn(rows, H, E, device="cuda", generator=g), torch.randn(E, device="cuda", generator=g).to(dtype)
    ld, out_ld = H * E + 12, H * E + 8
    gate = torch.randn(rows, ld, device="cuda", generator=g)
    out = torch.full((rows * out_ld + shift,), float("nan"), dtype=dtype, device="cuda")
    ops.head_norm_gate(o, w, 1e-4, gate.view(-1)[shift // 4 * 4:], ld, act, 0.7, out[shift:], out_ld, rows, H)
    cols = gate.double().view(-1)[shift // 4 * 4:]
    cols = torch.as_strided(cols, (rows, H * E), (ld, 1), cols.storage_offset()).reshape(rows, H, E)
    x = o.double()
    gated = torch.sigmoid(cols) if act == "sigmoid" else torch.nn.functional.silu(cols)
    want = 0.7 * x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-4) * w.double() * gated
    got = torch.as_strided(out, (rows, out_ld), (out_ld, 1), shift) if rows * out_ld + shift <= out.numel() else None
    assert ((got[:, :H * E].double().view(rows, H, E) - want).norm() / want.norm()).item() < EPS[dtype]
    assert torch.isnan(got[:, H * E:].float()).all()
