"""The dense GEMM with column tiles of every width that its rule takes, 256 down to 64, at ragged ends of rows and columns.
Needs a B200."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _takes(native_lib, rows, n_out, k_bytes, width):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert native_lib.h3s_dense_gemm_columns(rows, n_out, k_bytes, sms) == width


# (rows, columns) and the width that 74 pairs of SMs get; the last tile of columns is a partial one each time
WIDTHS = [(1, 8, 64), (130, 264, 64), (600, 2056, 96), (1000, 2056, 128), (2305, 1000, 160), (1000, 3080, 192), (2305, 3080, 224), (1000, 4104, 256)]


@pytest.mark.parametrize("rows,n_out,width", WIDTHS, ids=["64 of 8", "64", "96", "128", "160", "192", "224", "256"])
@pytest.mark.parametrize("gelu", [False, True])
def test_every_width_gives_the_exact_sums(native_lib, rows, n_out, width, gelu):
    from h3_optimizations_b200 import ops

    gen = torch.Generator().manual_seed(rows + n_out)
    k = 256
    _takes(native_lib, rows, n_out, k, width)
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
@pytest.mark.parametrize("rows,n_out,width", [(130, 264, 64), (600, 2056, 96), (1000, 3080, 192)], ids=["64", "96", "192"])
def test_narrow_tiles_of_the_other_types(native_lib, rows, n_out, width, dtype):
    from h3_optimizations_b200 import ops

    _takes(native_lib, rows, n_out, 256 * dtype.itemsize, width)
    gen = torch.Generator().manual_seed(rows)
    a = torch.randint(-4, 5, (rows, 256), generator=gen).to(dtype)  # every product and sum is exact in fp32
    b = torch.randint(-4, 5, (n_out, 256), generator=gen).to(dtype)
    got = ops.dense_gemm(a.cuda(), b.cuda()).cpu()
    assert torch.equal(got, (a.double() @ b.double().T).to(torch.bfloat16))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float8_e4m3fn], ids=["bf16", "e4m3"])
@pytest.mark.parametrize("rows,n_out,width", [(130, 264, 64), (600, 2056, 96), (2305, 1000, 160), (2305, 3080, 224)], ids=["64", "96", "160", "224"])
@pytest.mark.parametrize("gelu", [False, True])
@pytest.mark.parametrize("aligned", [True, False])
def test_scaled_floating_point_rows_of_narrow_tiles(native_lib, rows, n_out, width, dtype, gelu, aligned):
    """Column scale, bias and GELU behind floating-point products: packed where scale and bias are 16-byte aligned, else one by one."""
    from h3_optimizations_b200 import ops

    _takes(native_lib, rows, n_out, 256 * dtype.itemsize, width)
    gen = torch.Generator().manual_seed(rows)
    a = torch.randint(-4, 5, (rows, 256), generator=gen).to(dtype)  # every product and sum is exact in fp32
    b = torch.randint(-4, 5, (n_out, 256), generator=gen).to(dtype)
    shift = 0 if aligned else 1
    scale, bias = ((torch.rand((n_out + 1,), generator=gen) * top - low).cuda()[shift:][:n_out] for top, low in ((0.02, 0.0), (2.0, 1.0)))
    row_scale = (torch.rand((rows,), generator=gen) + 0.5).cuda()
    got = ops.dense_gemm(a.cuda(), b.cuda(), row_scale=row_scale, col_scale=scale, bias=bias, activation="gelu_tanh" if gelu else "none").cpu().double()
    product = (a.double() @ b.double().T) * row_scale.cpu().double()[:, None] * scale.cpu().double()[None, :]
    want = product + bias.cpu().double()[None, :]
    # fp32 roundings: two of the product, one of the sum
    error = 2.0 ** -24 * (2.0 * product.abs() + want.abs())
    relative = 2.0 ** -8 * 1.01  # half a bf16 ulp
    if gelu:
        u = 0.7978845608028654 * (want + 0.044715 * want ** 3)
        want = want / (1.0 + torch.exp(-2.0 * u))
        error *= 1.13                                  # the largest slope of GELU
        relative = relative + 2.0 * u.abs() * 2.0 ** -23  # the fp32 error of the exponent
    assert bool(((got - want).abs() <= want.abs() * relative + error + 1e-30).all())
