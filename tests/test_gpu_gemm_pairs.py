"""The two-CTA GEMM where its 256-row pairs, 256-column tiles and 4096-row groups do not
come out even.  Needs a B200."""

import pytest
import torch

from h3_optimizations_b200 import workloads
from oracle import h3_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(native_lib):
    from h3_optimizations_b200 import ops as module

    return module


# one row; a second CTA with no row at all, with one row, with all but one; a second row group of one row
@pytest.mark.parametrize("rows", [1, 128, 129, 255, 257, 4097])
def test_integer_gemm_is_exact_at_the_edges_of_a_pair(ops, rows):
    heads, hidden = 1, 256                                             # 384 columns: a half-filled column tile
    x, w, w_scale = workloads.projection_inputs(rows, hidden=hidden, heads=heads, seed=rows)
    x_i8, x_scale = oracle.convrot_quantize_rows(x)
    ref = oracle.qkv_project_int8(x_i8, x_scale, w, w_scale)
    staging = torch.full((3 * heads, rows + 8, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    ops.qkv_gemm_chunk(x_i8.cuda(), x_scale.cuda(), w.cuda(), w_scale.cuda(), staging, status=status)
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    got = staging[:, :rows].permute(1, 0, 2).reshape(rows, 3 * heads * 128).cpu()
    assert torch.equal(got.view(torch.int16), ref.view(torch.int16))
    assert bool(torch.isnan(staging[:, rows:].float()).all()), "rows past the last stay untouched"


@pytest.mark.parametrize("rows,n_out", [(1, 8), (129, 136), (257, 264), (4225, 520)])
def test_dense_gemm_stores_only_its_rows_and_columns(ops, rows, n_out):
    gen = torch.Generator().manual_seed(rows)
    k = 256
    a = torch.randint(-8, 9, (rows, k), generator=gen).to(torch.int8)
    b = torch.randint(-8, 9, (n_out, k), generator=gen).to(torch.int8)
    wide = torch.full((rows + 1, n_out + 8), float("nan"), dtype=torch.bfloat16, device="cuda")
    scales = torch.rand((n_out + 1,), generator=gen).cuda()
    # column vectors that are not 16-byte aligned take scalar loads
    ops.dense_gemm(a.cuda(), b.cuda(), col_scale=scales[1:], out=wide[:rows, :n_out])
    want = ((a.double() @ b.double().T).float() * scales[1:].cpu()).to(torch.bfloat16)  # exact sums, one product
    assert torch.equal(wide[:rows, :n_out].cpu(), want)
    assert bool(torch.isnan(wide[rows:].float()).all()) and bool(torch.isnan(wide[:, n_out:].float()).all())


def test_gelu_keeps_its_relative_accuracy_for_negative_values(ops):
    x = torch.cat([torch.linspace(-12, 12, 4801), torch.tensor([0.0, -0.0, 1e-30, -1e-30, 60.0, -60.0, 3e38, -3e38])])
    x = x.to(torch.bfloat16)
    a = torch.zeros((x.numel(), 64), dtype=torch.bfloat16)
    a[:, 0] = x
    b = torch.zeros((8, 64), dtype=torch.bfloat16)
    b[:, 0] = 1.0
    got = ops.dense_gemm(a.cuda(), b.cuda(), activation="gelu_tanh")[:, 0].cpu().double()
    v = x.double()
    u = 0.7978845608028654 * (v + 0.044715 * v * v * v)
    want = v / (1.0 + torch.exp(-2.0 * u))
    # half a bf16 ulp (8 significant bits: up to 2^-8 of a value), plus the fp32 error of the exponent 2u: 2^-23 of it; a reciprocal below
    # 2^-126 is flushed to zero, times |x| of about 10 where that happens
    bound = want.abs() * (2.0 ** -8 * 1.01 + 2.0 * u.abs().clamp(max=90) * 2.0 ** -23) + 16 * 2.0 ** -126
    assert bool(((got - want).abs() <= bound).all())
