"""2 to 8 token rows of large projections: on either side of the size from which they take the stream-K kernel, with the workspace it
needs and without, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# the result is rounded once to the storage type; the gate's silu and its product once more
TOL = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def _randn(*shape, dtype):
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    return torch.randn(*shape, device="cuda", generator=g).to(dtype)


def _rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("dtype", list(TOL))
@pytest.mark.parametrize("rows", [1, 2, 7, 8])
@pytest.mark.parametrize("n,k", [(3838, 4096), (3840, 4096), (3842, 4104), (3850, 4088), (1922, 8200)])
@pytest.mark.parametrize("with_workspace", [False, True])
def test_plain_and_fp32(dtype, rows, n, k, with_workspace):
    from gpt_fast.ops import CudaOps as ops
    x, w, add = _randn(rows, k, dtype=dtype), _randn(n, k, dtype=dtype), _randn(rows, n, dtype=dtype)
    want = x.double() @ w.double().T
    ws = torch.empty(max(ops.linear_workspace_bytes(64, n), ops.linear_f32_workspace_bytes(64, n)), dtype=torch.uint8, device="cuda") if with_workspace else None
    y, yf = torch.empty(rows, n, dtype=dtype, device="cuda"), torch.empty(rows, n, device="cuda")
    ops.linear(x, w, y, rows, workspace=ws)
    assert _rel(y, want) < TOL[dtype]
    ops.linear(x, w, y, rows, addend=add, workspace=ws)
    assert _rel(y, want + add.double()) < 2 * TOL[dtype]
    ops.linear_f32(x, w, yf, rows, workspace=ws)
    assert _rel(yf, want) < 1e-5


@pytest.mark.parametrize("dtype", list(TOL))
@pytest.mark.parametrize("rows", [1, 2, 7, 8])
@pytest.mark.parametrize("n,k", [(1918, 4096), (1920, 4096), (3840, 2048), (3842, 2056), (7000, 1128)])
@pytest.mark.parametrize("with_workspace", [False, True])
def test_gated(dtype, rows, n, k, with_workspace):
    from gpt_fast import _C
    from gpt_fast.ops import CudaOps as ops
    x, w = _randn(rows, k, dtype=dtype), (_randn(2 * n, k, dtype=dtype) * k ** -0.5).to(dtype)
    u, g = (x.double() @ w.double().T).chunk(2, dim=-1)
    ws = torch.empty(_C.lib.lri_gateup_workspace_bytes(64, n), dtype=torch.uint8, device="cuda") if with_workspace else None
    h = torch.empty(rows, n, dtype=dtype, device="cuda")
    ops.gateup_swiglu(x, w, h, rows, ws)
    assert _rel(h, torch.nn.functional.silu(g) * u) < 3 * TOL[dtype]
    ops.gateup_glu(x, w, h, rows, (1.702, 7.0, 1.0), workspace=ws)
    g = g.clamp(max=7.0)
    assert _rel(h, g * torch.sigmoid(1.702 * g) * (u.clamp(-7, 7) + 1)) < 3 * TOL[dtype]


@pytest.mark.parametrize("dtype", list(TOL))
@pytest.mark.parametrize("B,pos", [(2, 0), (8, 37), (16, 62), (40, 63)])
@pytest.mark.parametrize("k", [4096, 4088])
def test_qkv(dtype, B, pos, k):
    """Rotation and cache rows behind stream-K products (4096: from 2 rows on) and streaming ones, at the cache's first and last position."""
    from gpt_fast.ops import CudaOps as ops
    nh, nkv, hd, smax = 32, 8, 128, 64
    x, w = _randn(B, k, dtype=dtype), (_randn((nh + 2 * nkv) * hd, k, dtype=dtype) * k ** -0.5).to(dtype)
    ang = torch.outer(torch.arange(smax, device="cuda").double(), 1e4 ** (-torch.arange(0, hd, 2, device="cuda").double() / hd))
    table = torch.stack([ang.cos(), ang.sin()], dim=-1).to(dtype).contiguous()
    q, kc, vc = (torch.zeros(*s, dtype=dtype, device="cuda") for s in ((B, nh, hd), (B, nkv, smax, hd), (B, nkv, smax, hd)))
    ws = torch.empty(ops.qkv_workspace_bytes(64, nh, nkv, hd), dtype=torch.uint8, device="cuda")
    ops.qkv_rope_kvcache(x, w, table, False, torch.tensor([pos], device="cuda"), q, kc, vc, B, 1, nh, nkv, hd, ws)
    y = (x.double() @ w.double().T).view(B, nh + 2 * nkv, hd)
    c, s = table[pos].double().unbind(-1)
    a, b = y[..., 0::2], y[..., 1::2]
    turned = torch.stack([a * c - b * s, b * c + a * s], dim=-1).flatten(-2)
    # rounded after the product and after the rotation
    assert _rel(q, turned[:, :nh]) < 2 * TOL[dtype] and _rel(kc[:, :, pos], turned[:, nh:nh + nkv]) < 2 * TOL[dtype]
    assert _rel(vc[:, :, pos], y[:, nh + nkv:]) < TOL[dtype]
    others = [p for p in range(smax) if p != pos]
    assert not kc[:, :, others].any() and not vc[:, :, others].any()
