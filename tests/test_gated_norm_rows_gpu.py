"""Gated residual and norm at the edges of its forms (a row an SM, widths of one and more vectors a thread, slots summed in any number) against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}  # rounding of the stored norm; the residual is fp32


@pytest.mark.parametrize("dtype", list(EPS))
@pytest.mark.parametrize("dim", [8, 2048, 2056])
@pytest.mark.parametrize("more", [None, 0, 1])  # one row, a row an SM, one row more than that
@pytest.mark.parametrize("n_slots", [1, 2, 5])
def test_gated_norm_add(dtype, dim, more, n_slots):
    from gpt_fast.ops import CudaOps as ops
    rows = 1 if more is None else torch.cuda.get_device_properties(0).multi_processor_count + more
    g = torch.Generator(device="cuda").manual_seed(dim + rows)

    def randn(*shape, to=torch.float32):
        return torch.randn(*shape, device="cuda", generator=g).to(to)
    y_rows = n_slots * rows + 3
    y, resid, gate = randn(y_rows, dim, to=dtype), randn(rows, dim), randn(rows, dim + 4)
    bias, post, nxt = (randn(dim, to=dtype) for _ in range(3))
    slots = torch.randint(0, y_rows, (rows, n_slots), generator=g, device="cuda").int()
    got, normed = resid.clone(), torch.full((rows, dim), float("nan"), dtype=dtype, device="cuda")
    ops.gated_norm_add(got, y, gate, dim + 4, bias, post, 1e-3, nxt, normed, rows, n_slots, slots, y_rows)

    def norm(x, w):
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-3) * w.double()

    def far(x, want):
        return ((x.double() - want).norm() / want.norm()).item()
    gated = y.double()[slots.long()].sum(1) * torch.sigmoid(gate[:, :dim].double() + bias.double())
    want = resid.double() + norm(gated, post)
    assert far(got, want) < 2e-6
    assert far(normed, norm(want, nxt)) < EPS[dtype]


@pytest.mark.parametrize("dtype", list(EPS))
@pytest.mark.parametrize("dim,n_slots", [(d, n) for d in (4096, 4104, 8192) for n in (1, 2, 3, 5)] + [(d, 3) for d in (8, 2048, 2056)])
@pytest.mark.parametrize("more", [None, 0, 1])
def test_gated_norm_add_wide_and_three_results(dtype, dim, more, n_slots):
    test_gated_norm_add(dtype, dim, more, n_slots)
