"""Row kernels at the edges of their widths, and batches written in place.  Needs a B200.

The row kernels are exact restatements of torch expressions, so codes and scales are compared
bit for bit."""

import pytest
import torch

from h3_optimizations_b200 import workloads
from oracle import h3_oracle as oracle

pytestmark = pytest.mark.gpu


# each register width of the warp kernel, one vector less and more, and the first width of the CTA kernel
@pytest.mark.parametrize("channels", [8, 1016, 1024, 1032, 2048, 2056, 3072, 3080, 4096, 4104])
@pytest.mark.parametrize("rows", [1, 7])
def test_row_codes(native_lib, rows, channels):
    from h3_optimizations_b200 import ops

    gen = torch.Generator().manual_seed(channels + rows)
    wide = torch.randn((rows, channels + 8), generator=gen).to(torch.bfloat16)
    wide[0, :channels] = 0.0 if rows > 1 else wide[0, :channels]                  # a zero row takes the smallest scale
    codes, scale = ops.quant_rows_fp8(wide.cuda()[:, :channels])                  # strided rows
    x = wide[:, :channels].float()
    want = (x.abs().amax(dim=1) / 448.0).clamp_min(1.0e-20)
    assert torch.equal(scale.cpu(), want)
    assert torch.equal(codes.cpu().view(torch.uint8), (x / want[:, None]).to(torch.float8_e4m3fn).view(torch.uint8))


# one to 32 groups of 256 channels; 3 columns of a warp's lanes unevenly filled
@pytest.mark.parametrize("hidden", [256, 768, 1280, 8192])
@pytest.mark.parametrize("rows", [1, 6])
def test_rotated_codes(native_lib, rows, hidden):
    from h3_optimizations_b200 import ops

    gen = torch.Generator().manual_seed(hidden + rows)
    x = torch.randn((rows, hidden), generator=gen).to(torch.bfloat16)
    codes, scale = ops.convrot_quant_rows(x.cuda())
    want_codes, want_scale = oracle.convrot_quantize_rows(x)
    assert torch.equal(scale.cpu(), want_scale) and torch.equal(codes.cpu(), want_codes)


# wide rows, on both sides of the lines between one and four to a block
@pytest.mark.parametrize("rows,hidden", [(296, 8192), (297, 8192), (592, 8192), (593, 8192), (299, 3328), (2368, 3328), (2369, 3328)])
def test_rotated_codes_of_wide_rows(native_lib, rows, hidden):
    from h3_optimizations_b200 import ops

    gen = torch.Generator().manual_seed(hidden + rows)
    x = torch.randn((rows, hidden), generator=gen).to(torch.bfloat16)
    codes, scale = ops.convrot_quant_rows(x.cuda())
    want_codes, want_scale = oracle.convrot_quantize_rows(x)
    assert torch.equal(scale.cpu(), want_scale) and torch.equal(codes.cpu(), want_codes)


@pytest.mark.parametrize("batch", [1, 2, 3])
def test_a_batch_equals_its_elements(native_lib, batch):
    from h3_optimizations_b200 import B200SparseBackend, HybridSparseConfig, runtime_options

    spec = workloads.small_spec("batch", 2, 100, 900)
    q, k, v = (torch.cat([workloads.gaussian_qkv(spec, seed=s)[i] for s in range(batch)]).cuda() for i in range(3))
    backend = B200SparseBackend(HybridSparseConfig(video_budget=0.3))
    options = runtime_options(spec.layout())
    out = backend.forward(q, k, v, layer_index=0, transformer_options=options)
    assert out.shape == q.shape and out.dtype == q.dtype
    assert batch == 1 or out.is_contiguous()
    for b in range(batch):
        one = backend.forward(q[b:b + 1], k[b:b + 1], v[b:b + 1], layer_index=0, transformer_options=options)
        # the K mean's FP64 sum is gathered with atomics, in any order: its rounding is the same but for ties
        assert (out[b:b + 1].float() - one.float()).abs().max() <= 2.0 ** -8 * one.float().abs().max()


@pytest.mark.parametrize("hidden", [512, 3328])
def test_rotated_codes_of_unusual_rows(native_lib, hidden):
    """A NaN counts as nothing and takes code 0, as whatever an infinite scale divides; scales down to the smallest."""
    from h3_optimizations_b200 import ops

    gen = torch.Generator().manual_seed(hidden)
    x = torch.randn((8, hidden), generator=gen).to(torch.bfloat16)
    x[0], x[1], x[2] = 0.0, x[1] * 2.0 ** -120, x[2] * 2.0 ** 120
    x[3] = 0.0
    x[3, 7] = 2.0 ** -133  # a scale below the smallest normal number
    without = x.clone()
    x[4, 5], without[4, :256] = float("nan"), 0.0
    x[5, 300] = float("inf")
    x[6, 3], x[6, 4] = float("inf"), float("nan")
    codes, scale = (t.cpu() for t in ops.convrot_quant_rows(x.cuda()))
    want_codes, want_scale = oracle.convrot_quantize_rows(without)
    rows = [0, 1, 2, 3, 4, 7]
    assert torch.equal(scale[rows], want_scale[rows]) and torch.equal(codes[rows], want_codes[rows])
    assert scale[5] == float("inf") and not codes[5].any()
    # the group of row 6 has nothing but NaN; the others are quantised by their own largest magnitude
    other = x[6:7].clone()
    other[0, :256] = 0.0
    want_codes, want_scale = oracle.convrot_quantize_rows(other)
    assert torch.equal(codes[6:7], want_codes) and torch.equal(scale[6:7], want_scale)
