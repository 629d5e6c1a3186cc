"""The dense GEMM with column tiles of every width that its rule takes, 256 down to 64, at ragged ends of rows and columns.
Needs a B200."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# (rows, columns) and the width that 74 pairs of SMs get; the last tile of columns is a partial one each time
@pytest.mark.parametrize("rows,n_out", [(1, 8), (130, 264), (600, 2056), (1000, 2056), (2305, 1000), (1000, 3080), (2305, 3080), (1000, 4104)],
                         ids=["64 of 8", "64", "96", "128", "160", "192", "224", "256"])
@pytest.mark.parametrize("gelu", [False, True])
def test_every_width_gives_the_exact_sums(native_lib, rows, n_out, gelu):
    from h3_optimizations_b200 import ops

    gen = torch.Generator().manual_seed(rows + n_out)
    k = 256
    a = torch.randint(-8, 9, (rows, k), generator=gen).to(torch.int8)
    b = torch.randint(-8, 9, (n_out, k), generator=gen).to(torch.int8)
    scale = (torch.rand((n_out,), generator=gen) * 0.01).cuda()
    wide = torch.full((rows + 1, n_out + 8), float("nan"), dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    ops.dense_gemm(a.cuda(), b.cuda(), col_scale=scale, activation="gelu_tanh" if gelu else "none", out=wide[:rows, :n_out], status=status)
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    value = (a.double() @ b.double().T).float() * scale.cpu()  # exact sums, one product
    got = wide[:rows, :n_out].cpu()
    if gelu:
        v = value.double()
        u = 0.7978845608028654 * (v + 0.044715 * v * v * v)
        want = v / (1.0 + torch.exp(-2.0 * u))
        # half a bf16 ulp, and the fp32 error of the exponent
        assert bool(((got.double() - want).abs() <= want.abs() * (2.0 ** -8 * 1.01 + 2.0 * u.abs() * 2.0 ** -23) + 1e-30).all())
    else:
        assert torch.equal(got, value.to(torch.bfloat16))
    assert bool(torch.isnan(wide[rows:].float()).all()) and bool(torch.isnan(wide[:, n_out:].float()).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float8_e4m3fn], ids=["bf16", "fp16", "e4m3"])
@pytest.mark.parametrize("rows,n_out", [(130, 264), (600, 2056), (1000, 3080)], ids=["64", "96", "192"])
def test_narrow_tiles_of_the_other_types(native_lib, rows, n_out, dtype):
    from h3_optimizations_b200 import ops

    gen = torch.Generator().manual_seed(rows)
    a = torch.randint(-4, 5, (rows, 256), generator=gen).to(dtype)  # every product and sum is exact in fp32
    b = torch.randint(-4, 5, (n_out, 256), generator=gen).to(dtype)
    got = ops.dense_gemm(a.cuda(), b.cuda()).cpu()
    assert torch.equal(got, (a.double() @ b.double().T).to(torch.bfloat16))
