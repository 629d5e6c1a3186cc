"""The carrier epilogue in all forms of its rotation table and tile means.  Needs a B200.

Tables in bf16 and FP32; packed with rows on 32 and on 16 bytes, and in a layout that is read element by
element; tile means of every type; K smoothed and not.  Codes and scales are the oracle's bit for bit.  A tile mean comes
from FP32 sums of eight values and an exact total, rounded to its type."""

from types import SimpleNamespace

import pytest
import torch

from h3_optimizations_b200 import workloads
from oracle import h3_oracle as oracle

pytestmark = pytest.mark.gpu

SEQUENCE, HIDDEN, HEADS = 700, 512, 2  # five whole tiles and 60 rows


def _table(dtype, form):
    rope = oracle.make_rope(SEQUENCE).to(dtype)
    if form == "sectors":
        return rope, rope.cuda()
    if form == "chunks":  # rows begin 16 bytes off a sector
        ahead = 16 // rope.element_size()
        rows = torch.zeros((SEQUENCE, 192 + 2 * ahead), dtype=dtype, device="cuda")
        view = rows[:, ahead:ahead + 192].unflatten(1, (48, 2, 2))[None, :, None]
        view.copy_(rope)
        assert view.data_ptr() % 32 == 16 and view.stride(1) * view.element_size() % 32 == 0
        return rope, view
    rows = torch.zeros((SEQUENCE, 2, 48, 2), dtype=dtype, device="cuda")  # "strided": another order of the axes
    view = rows.permute(0, 2, 1, 3)[None, :, None]
    view.copy_(rope)
    return rope, view


def _project(rope, view, smooth_k, summary_dtype):
    from h3_optimizations_b200 import ChunkedSparseQKVProjector

    x, w, w_scale = workloads.projection_inputs(SEQUENCE, hidden=HIDDEN, heads=HEADS, seed=21)
    gen = torch.Generator().manual_seed(4)
    norm = lambda: SimpleNamespace(weight=(torch.rand(128, generator=gen) + 0.5).to(torch.bfloat16).cuda(), eps=1e-6)
    module = SimpleNamespace(heads=HEADS, head_dim=128, qkv_weight_int8=w.cuda(), qkv_weight_scale=w_scale.cuda(), q_norm=norm(), k_norm=norm())
    got = ChunkedSparseQKVProjector(chunk_rows=256, smooth_k=smooth_k, summary_dtype=summary_dtype).project(
        module, x.cuda(), view, layer_index=0, transformer_options={})
    x_i8, x_scale = oracle.convrot_quantize_rows(x)
    y = oracle.rms_norm_rope_split_half(oracle.qkv_project_int8(x_i8, x_scale, w, w_scale), HEADS, module.q_norm.weight.cpu(),
                                        module.k_norm.weight.cpu(), 1e-6, rope)
    return got, oracle.split_heads_hnd(y, HEADS)


def _check(got, qkv, smooth_k, summary_dtype):
    from h3_optimizations_b200 import ops

    q, k, v = qkv
    mean = ops.column_stats(k.cuda().contiguous(), None)[0].cpu() if smooth_k else None
    for name, codes, scale, want in (("q", got.q_int8, got.q_scale, oracle.quantize_blocks(q, 128)),
                                     ("k", got.k_int8, got.k_scale, oracle.quantize_blocks(k, 64, mean=mean))):
        assert torch.equal(codes.cpu(), want[0]) and torch.equal(scale.cpu(), want[1]), name
    carrier, v_scale = oracle.v_fp8_carrier(v)
    assert torch.equal(got.v_scale.cpu(), v_scale)
    assert torch.equal(got.v_carrier.cpu().view(torch.uint8), carrier.view(torch.uint8))
    unit = {torch.float64: 2.0 ** -52, torch.float32: 2.0 ** -24, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[summary_dtype]
    for summary, values, block in ((got.q_summary, q, 128), (got.k_summary, k, 64)):
        assert summary.dtype == summary_dtype
        exact, size = (oracle.mean_pool(t.double(), block) for t in (values, values.abs()))
        # seven FP32 roundings of partial sums, each at most half a unit of the sum of magnitudes, and the type's own
        bound = 7 * 2.0 ** -24 * size + 2 * unit * exact.abs() + 1e-7
        assert bool(((summary.cpu().double() - exact).abs() <= bound).all())


@pytest.mark.parametrize("form", ["sectors", "chunks", "strided"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("smooth_k", [True, False])
def test_every_form_of_the_table(native_lib, dtype, form, smooth_k):
    got, qkv = _project(*_table(dtype, form), smooth_k, torch.float32)
    _check(got, qkv, smooth_k, torch.float32)


@pytest.mark.parametrize("summary_dtype", [torch.float64, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("smooth_k", [True, False])
def test_every_type_of_tile_means(native_lib, summary_dtype, smooth_k):
    got, qkv = _project(*_table(torch.bfloat16, "sectors"), smooth_k, summary_dtype)
    _check(got, qkv, smooth_k, summary_dtype)
