"""Tile means and column sums of the carrier epilogue, value for value.  Needs a B200.

The partial sums of eight rows are FP32, their totals as good as in 64 bits: finite wherever the
partial sums are, and without a bit lost where the partial sums are exact.  One weight column per channel and one
scale per row make every projected value w[channel] * scale[row], exact in bf16."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _project(native_lib, weight, row_scale, summary_dtype, smooth_k):
    from h3_optimizations_b200 import ops

    rows = row_scale.numel()
    x = torch.zeros((rows, 128), dtype=torch.int8)
    x[:, 0] = 1
    w = torch.zeros((384, 128), dtype=torch.int8)
    w[:, 0] = weight
    empty = lambda *shape, dtype: torch.empty(shape, dtype=dtype, device="cuda")
    blocks = lambda tile: -(-rows // tile)
    out = {"q_int8": empty(1, 1, rows, 128, dtype=torch.int8), "q_scale": empty(1, 1, blocks(128), dtype=torch.float32),
           "q_summary": empty(1, 1, blocks(128), 128, dtype=summary_dtype), "k_summary": empty(1, 1, blocks(64), 128, dtype=summary_dtype),
           "v_stage": empty(1, 1, rows, 128, dtype=torch.bfloat16), "stats": ops.column_stats_scratch(1, "cuda")}
    if smooth_k:
        out["k_stage"] = empty(1, 1, rows, 128, dtype=torch.bfloat16)
    else:
        out.update(k_int8=empty(1, 1, rows, 128, dtype=torch.int8), k_scale=empty(1, 1, blocks(64), dtype=torch.float32))
    ops.qkv_gemm_chunk_carriers(x.cuda(), row_scale.cuda(), w.cuda(), torch.ones(384).cuda(), heads=1, row_start=0, **out)
    return {name: t.cpu() for name, t in out.items()}


def _totals(weight, exponent, tile):
    """Exact in 64 bits: the sum of a tile's scales first, then the weight."""
    return torch.stack([(2.0 ** e.double()).sum() * weight.double() for e in exponent.split(tile)])


@pytest.mark.parametrize("summary_dtype", [torch.float64, torch.float32, torch.bfloat16])
@pytest.mark.parametrize("smooth_k", [True, False])
def test_totals_beyond_the_range_of_a_float(native_lib, summary_dtype, smooth_k):
    """Values of 2^124: eight of them are a finite float, sixteen are not.  Whole tiles and a ragged one."""
    gen = torch.Generator().manual_seed(1)
    weight = (torch.randint(0, 2, (384,), generator=gen) * 2 - 1).to(torch.int8)
    got = _project(native_lib, weight, torch.full((200,), 2.0 ** 124), summary_dtype, smooth_k)
    want = weight.double() * 2.0 ** 124
    assert torch.equal(got["q_summary"][0, 0].double(), want[:128].expand(2, 128))
    assert torch.equal(got["k_summary"][0, 0].double(), want[128:256].expand(4, 128))
    if smooth_k:
        assert torch.equal(got["stats"].view(torch.float64)[:128], want[128:256] * 200)


@pytest.mark.parametrize("smooth_k", [True, False])
def test_totals_of_exact_partial_sums_are_exact(native_lib, smooth_k):
    """Four sizes of rows, 2^24 down to 2^-19: a total has up to 53 bits.  Rows that are added up in FP32 have one size."""
    gen = torch.Generator().manual_seed(2)
    weight = (torch.randint(-64, 64, (384,), generator=gen) * 2 + 1).to(torch.int8)
    exponent = torch.tensor([24.0, 2.0, -12.0, -19.0]).repeat_interleave(2).repeat(24)      # of row r: by (r % 8) // 2
    got = _project(native_lib, weight, 2.0 ** exponent, torch.float64, smooth_k)
    assert torch.equal(got["q_summary"][0, 0], _totals(weight[:128], exponent, 128) / torch.tensor([[128.0], [64.0]]))
    assert torch.equal(got["k_summary"][0, 0], _totals(weight[128:256], exponent, 64) / 64)
    if smooth_k:
        assert torch.equal(got["stats"].view(torch.float64)[:128], _totals(weight[128:256], exponent, 192)[0])


def test_means_in_fp32_are_the_nearest(native_lib):
    """The same rows: the exact total, rounded once."""
    gen = torch.Generator().manual_seed(3)
    weight = (torch.randint(-64, 64, (384,), generator=gen) * 2 + 1).to(torch.int8)
    for exponents in ([24.0, 2.0, -12.0, -19.0], [0.0, -16.0, -16.0, -41.0], [0.0, -17.0, -25.0, -40.0]):
        exponent = torch.tensor(exponents).repeat_interleave(2).repeat(24)
        got = _project(native_lib, weight, 2.0 ** exponent, torch.float32, False)
        assert torch.equal(got["q_summary"][0, 0], (_totals(weight[:128], exponent, 128) / torch.tensor([[128.0], [64.0]])).float())
        assert torch.equal(got["k_summary"][0, 0], (_totals(weight[128:256], exponent, 64) / 64).float())
