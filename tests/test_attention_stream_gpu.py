"""Decode attention as one stream of cache rows (attention_stream.cu): runs that end inside a pair, at its end and behind several
pairs, lengths around its units of 32 positions and around the shortest pair that is cut, groups of 1 to 16 query heads, cache
rows past the position that hold NaN, and the masked form, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _force_stream():
    from gpt_fast import _C
    _C.check(_C.lib.lri_set_option(b"attn_mma", 1))
    yield
    _C.check(_C.lib.lri_set_option(b"attn_mma", -1))
    _C.check(_C.lib.lri_gemm_status())


def _case(dtype, B, nh, nkv, dim, vdim, smax, pos, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + pos)

    def randn(*shape):
        return torch.randn(*shape, device="cuda", generator=g).to(dtype)

    q, kc, vc = randn(B, nh, dim), randn(B, nkv, smax, dim), randn(B, nkv, smax, vdim)
    kc[:, :, pos + 1:] = float("nan")
    vc[:, :, pos + 1:] = float("nan")
    return q, kc, vc, torch.tensor([pos], dtype=torch.int32, device="cuda")


def _want(q, kc, vc, lo, pos, scale, sink=None):
    B, nh, dim = q.shape
    nkv = kc.shape[1]
    k, v = (t[:, :, lo:pos + 1].double().repeat_interleave(nh // nkv, dim=1) for t in (kc, vc))
    s = torch.einsum("bhd,bhjd->bhj", q.double(), k) * scale
    if sink is not None:
        s = torch.cat([s, sink.double()[None, :, None].expand(B, nh, 1)], dim=-1)
    w = torch.softmax(s, dim=-1)[..., : k.shape[2]]
    return torch.einsum("bhj,bhjd->bhd", w, v)


# probabilities and the result are rounded once to the storage type: at most two half units in the last place of the result's scale
TOL = {torch.bfloat16: 2 * 2 ** -8, torch.float16: 2 * 2 ** -11}


@pytest.mark.parametrize("dtype", list(TOL))
@pytest.mark.parametrize("B,nh,nkv,hd", [(1, 1, 1, 128), (3, 32, 2, 128), (5, 20, 4, 64), (20, 32, 8, 64), (13, 24, 24, 128), (41, 24, 8, 64),
                                             (6, 16, 4, 64), (38, 12, 12, 64)])
@pytest.mark.parametrize("pos", [0, 31, 32, 479, 480, 481, 527, 995, 1022])
def test_stream(dtype, B, nh, nkv, hd, pos):
    from gpt_fast.ops import CudaOps as ops, decode_splits
    smax = 1023
    q, kc, vc, ipos = _case(dtype, B, nh, nkv, hd, hd, smax, pos)
    want = _want(q, kc, vc, 0, pos, hd ** -0.5)
    for slots in (decode_splits(B, nh, nkv, smax, hd), 4):
        scratch = torch.zeros(ops.attn_decode_scratch_bytes(B, nh, nkv, hd, slots), dtype=torch.uint8, device="cuda")
        for _ in range(2):  # the counters are left at zero
            out = torch.full((B, nh, hd), float("nan"), dtype=dtype, device="cuda")
            ops.attention(q, kc, vc, ipos, out, B, 1, nh, nkv, hd, scratch, 1 if slots == 1 else 2)
            assert ((out.double() - want).norm() / want.norm()).item() < TOL[dtype]


@pytest.mark.parametrize("dtype", list(TOL))
@pytest.mark.parametrize("B,nh,nkv,dim,vdim,window,chunk", [(2, 4, 1, 128, 128, 0, 0), (16, 32, 8, 128, 128, 0, 256), (3, 6, 2, 96, 40, 100, 0),
                                                            (20, 16, 16, 64, 64, 33, 0), (2, 16, 1, 40, 128, 70, 64)])
@pytest.mark.parametrize("pos", [0, 31, 32, 63, 64, 255, 256, 699])
def test_stream_masked(dtype, B, nh, nkv, dim, vdim, window, chunk, pos):
    from gpt_fast.ops import CudaOps as ops
    q, kc, vc, ipos = _case(dtype, B, nh, nkv, dim, vdim, 700, pos)
    lo = max(0, pos - window + 1 if window else 0, pos // chunk * chunk if chunk else 0)
    kc[:, :, :lo] = float("nan")
    vc[:, :, :lo] = float("nan")
    for sink in (None, torch.linspace(-2, 3, nh, device="cuda").to(dtype)):
        want = 1.5 * _want(q, kc, vc, lo, pos, dim ** -0.5, sink)
        out = torch.full((B, nh * vdim + 8), float("nan"), dtype=dtype, device="cuda")
        ops.grouped_attention(q, kc, vc, sink, out, nh * vdim + 8, 1.5, ipos, window, chunk, dim ** -0.5, B, 1, nh)
        got = out[:, : nh * vdim].view(B, nh, vdim)
        # probabilities keep 16 bits and more here: the result is rounded once
        assert ((got.double() - want).norm() / want.norm()).item() < TOL[dtype] / 2
        assert out[:, nh * vdim:].isnan().all()


@pytest.mark.parametrize("dtype", list(TOL))
@pytest.mark.parametrize("B,nh,nkv,hd,pos", [(1, 32, 8, 128, 1022), (2, 32, 8, 128, 1022), (15, 32, 8, 128, 700), (5, 20, 4, 64, 527), (31, 24, 4, 64, 995)])
def test_probabilities_keep_more_than_the_storage_type(dtype, B, nh, nkv, hd, pos):
    """Below 128 pairs of a sequence and a KV head, in whichever kernel, rounding the result is all the error there is: a sequence loses no
    bits when others join it.  Probabilities rounded to the storage type would add an error of the same size (1.2 to 1.4 times in all); as two
    numbers of it they add 2^-8 of that (bf16), and the fp32 sums less than 1 % (fp16)."""
    from gpt_fast import _C
    from gpt_fast.ops import CudaOps as ops, decode_splits
    _C.check(_C.lib.lri_set_option(b"attn_mma", -1))
    q, kc, vc, ipos = _case(dtype, B, nh, nkv, hd, hd, 1023, pos)
    want = _want(q, kc, vc, 0, pos, hd ** -0.5)
    splits = decode_splits(B, nh, nkv, 1023, hd)
    scratch = torch.zeros(ops.attn_decode_scratch_bytes(B, nh, nkv, hd, splits), dtype=torch.uint8, device="cuda")
    out = torch.full((B, nh, hd), float("nan"), dtype=dtype, device="cuda")
    ops.attention(q, kc, vc, ipos, out, B, 1, nh, nkv, hd, scratch, splits)
    rounding = (want.to(dtype).double() - want).norm()
    assert ((out.double() - want).norm() / rounding).item() < 1.02
