"""The prefill GEMM on pairs of SMs: every tile width and epilogue against plain fp32 matrix products, at sizes around the edges of
its 256-row tiles, and the widths that it chooses on the host."""
import ctypes
import math

import pytest
import torch

from oracle import ladder_oracle as lo

DTYPES = [torch.bfloat16, torch.float16]
ROUNDING = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def _lib():
    from gpt_fast import _C
    return _C


@pytest.fixture
def width():
    C = _lib()
    yield lambda bn: C.check(C.lib.lri_set_option(b"gemm_pair", bn))
    C.check(C.lib.lri_set_option(b"gemm_pair", 1))


def _close(got, ref, dtype, sums):
    """One rounding of the result, and fp32 sums of `sums` products in another order (each at most half an fp32 ulp of the largest
    partial sum, which random signs keep within a few times the row's scale)."""
    _lib().check(_lib().lib.lri_gemm_status())
    got, ref = got.float().cpu(), ref.float()
    bound = ref.abs() * ROUNDING[dtype] + 4 * math.sqrt(sums) * 2.0 ** -23 * ref.abs().mean() + 1e-6
    assert torch.isfinite(got).all() and ((got - ref).abs() <= bound).all(), ((got - ref).abs() / bound).max()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("bn", [64, 160, 224, 256])
@pytest.mark.parametrize("m,n,k", [(129, 8, 8), (255, 264, 72), (256, 256, 64), (257, 520, 1000), (700, 1288, 136), (1030, 24, 520)])
def test_plain_and_fp32(width, dtype, bn, m, n, k):
    from gpt_fast.ops import CudaOps as ops
    width(bn)
    g = torch.Generator().manual_seed(m + n + k)
    x, w = torch.randn(m, k, generator=g).to(dtype), (torch.randn(n, k, generator=g) / math.sqrt(k)).to(dtype)
    ref = x.float() @ w.float().T
    y = torch.full((m, n), float("nan"), dtype=dtype, device="cuda")
    ops.linear(x.cuda(), w.cuda(), y, m)
    _close(y, ref, dtype, k)
    f = torch.full((m, n), float("nan"), device="cuda")
    ops.linear_f32(x.cuda(), w.cuda(), f, m)
    torch.cuda.synchronize()
    assert (f.cpu() - ref).norm() <= 1e-6 * math.sqrt(k) * ref.norm()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("bn", [64, 96, 192, 256])
@pytest.mark.parametrize("m,inter,k", [(130, 8, 16), (256, 128, 64), (300, 200, 264), (513, 1000, 136)])
def test_gated_units(width, dtype, bn, m, inter, k):
    from gpt_fast.ops import CudaOps as ops
    g = torch.Generator().manual_seed(m + inter + k)
    x, w = torch.randn(m, k, generator=g).to(dtype), (torch.randn(2 * inter, k, generator=g) * 2 / math.sqrt(k)).to(dtype)
    ug = x.float() @ w.float().T
    width(bn)
    h = torch.full((m, inter), float("nan"), dtype=dtype, device="cuda")
    ops.gateup_swiglu(x.cuda(), w.cuda(), h, m, None)
    ref = lo.swiglu(ug.to(dtype)).float()
    torch.cuda.synchronize()
    _lib().check(_lib().lib.lri_gemm_status())
    # up, gate, silu(gate) and the result are rounded, so sums in another order may flip each by an ulp (twice ROUNDING): an ulp of
    # the gate moves silu, whose slope is at most 1.1, by 2.2 ROUNDING |gate|, the three others move the result by 2 ROUNDING each
    bound = ROUNDING[dtype] * (6 * ref.abs() + 2.2 * (ug[:, inter:] * ug[:, :inter]).abs()) + 1e-5
    assert ((h.float().cpu() - ref).abs() <= bound).all()
    glu = (1.702, 1.2, 1.0)
    ops.gateup_glu(x.cuda(), w.cuda(), h, m, glu)
    gate, up = ug[:, inter:].clamp(max=glu[1]), ug[:, :inter].clamp(-glu[1], glu[1])
    ref = gate * torch.sigmoid(glu[0] * gate) * (up + glu[2])
    bound = ref.abs() * ROUNDING[dtype] + 1e-5 * math.sqrt(k)
    torch.cuda.synchronize()
    _lib().check(_lib().lib.lri_gemm_status())
    assert ((h.float().cpu() - ref).abs() <= bound).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("bn", [64, 160, 256])
@pytest.mark.parametrize("B,S,nh,nkv,hd,first", [(1, 129, 4, 2, 32, 0), (2, 150, 6, 2, 64, 7), (3, 171, 2, 1, 128, 40)])
def test_query_key_value(width, dtype, bn, B, S, nh, nkv, hd, first):
    """The fused epilogue against the single-CTA kernel's: the same sums, rotated and scattered."""
    from gpt_fast.ops import CudaOps as ops
    k, smax = 264, first + S + 8
    g = torch.Generator().manual_seed(S + hd)
    x, w = torch.randn(B * S, k, generator=g).to(dtype).cuda(), (torch.randn((nh + 2 * nkv) * hd, k, generator=g) / math.sqrt(k)).to(dtype).cuda()
    table = torch.randn(smax, hd // 2, 2, generator=g).to(dtype).cuda()
    pos = torch.arange(first, first + S).cuda()
    got = []
    for v in (0, bn):
        width(v)
        q = torch.zeros(B * S, nh * hd, dtype=dtype, device="cuda")
        kc, vc = torch.zeros(B, nkv, smax, hd, dtype=dtype, device="cuda"), torch.zeros(B, nkv, smax, hd, dtype=dtype, device="cuda")
        ops.qkv_rope_kvcache(x, w, table, False, pos, q, kc, vc, B, S, nh, nkv, hd, None)
        torch.cuda.synchronize()
        _lib().check(_lib().lib.lri_gemm_status())
        got.append((q, kc, vc))
    for a, b in zip(*got):
        assert (a.float() - b.float()).norm() <= ROUNDING[dtype] * a.float().norm() and torch.equal(a == 0, b == 0)


def test_option_values():
    C = _lib()
    v = ctypes.c_int(-1)
    for bad in (-1, 2, 63, 100, 257):
        assert C.lib.lri_set_option(b"gemm_pair", bad) == -1
    C.check(C.lib.lri_get_option(b"gemm_pair", ctypes.byref(v)))
    assert v.value == 1


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,flag,pairs", [(128, 4096, 1024, False, False), (129, 4096, 1024, False, True), (129, 4096, 1024, True, False),
                                              (300, 1024, 128, False, False), (300, 1024, 136, False, True), (2048, 4096, 504, False, False),
                                              (2048, 4096, 512, False, True)])
def test_which_products_take_pairs(m, n, k, flag, pairs):
    """By rows, depth and width, and by what the caller says; either kernel gives the same products."""
    from gpt_fast.ops import CudaOps as ops
    g = torch.Generator(device="cuda").manual_seed(m + k)
    x, w = (torch.randn(r, k, generator=g, device="cuda").bfloat16() for r in (m, n))
    y, f, h = torch.empty(m, n, dtype=torch.bfloat16, device="cuda"), torch.empty(m, n, device="cuda"), torch.empty(m, n // 2, dtype=torch.bfloat16, device="cuda")
    flags = _lib().ONE_SM if flag else 0
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        ops.linear(x, w, y, m, flags=flags)
        ops.linear_f32(x, w, f, m, flags=flags)
        ops.gateup_glu(x, w, h, m, (1.702, 1.2, 1.0), flags=flags)
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if "gemm" in e.name and e.device_type == torch.autograd.DeviceType.CUDA]
    assert len(names) == 3 and all(("gemm_pair" in name) == pairs for name in names), names
    _close(y, (x.double() @ w.double().T).float().cpu(), torch.bfloat16, k)
    assert torch.equal(f.bfloat16(), y)
