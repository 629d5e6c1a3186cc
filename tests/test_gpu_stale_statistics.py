"""Carriers are made with the statistics of their own call, although each kernel starts while the one before it ends and the allocator
hands out the same memory call after call.  Needs a B200.

Inputs of very different size take turns, so that a scale or mean of the call before shows in every code."""

import pytest
import torch

from h3_optimizations_b200 import workloads

pytestmark = pytest.mark.gpu


def _divide(x, by):
    return x / torch.full_like(x, by)  # by a number torch multiplies with the reciprocal


def _v_carrier(v):
    """Codes (an E4M3 zero as 0) and scales of V (1, H, S, 128) by plain torch."""
    scale = _divide(v.float().abs().amax(dim=2), 448.0).clamp_min(1.0e-20)
    codes = (v.float() / scale[:, :, None]).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).view(torch.uint8)
    return torch.where(codes == 0x80, 0, codes).transpose(-1, -2), scale


def _k_carrier(k, smooth_k):
    """Codes and scales of K's blocks of 64 rows; the sequence a multiple of 64."""
    x = k.float()
    if smooth_k:
        x = x - k.double().mean(dim=2, keepdim=True).to(torch.float32).to(k.dtype).float()
    blocks = x.view(1, x.shape[1], -1, 64, 128)
    scale = _divide(blocks.abs().amax(dim=(-2, -1)), 127.0) + 1e-7
    q = blocks / scale[..., None, None]
    return (q + torch.where(q >= 0, 0.5, -0.5)).to(torch.int8).view_as(x), scale


def _same(sparse, k, v, smooth_k):
    codes, scale = _v_carrier(v)
    got = sparse.v_carrier.view(torch.uint8)[..., :v.shape[2]]
    assert torch.equal(sparse.v_scale, scale) and torch.equal(torch.where(got == 0x80, 0, got), codes)
    codes, scale = _k_carrier(k, smooth_k)
    assert torch.equal(sparse.k_scale, scale) and torch.equal(sparse.k_int8, codes)


@pytest.mark.parametrize("budget", [1.0, 0.3])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("smooth_k", [True, False])
@pytest.mark.parametrize("heads,sequence,rows", [(6, 12544, None), (3, 2304, 0), (3, 2304, None)], ids=["long", "short on two streams", "short"])
def test_layers(native_lib, monkeypatch, heads, sequence, rows, smooth_k, dtype, budget):
    from h3_optimizations_b200 import B200SparseBackend, HybridSparseConfig, backend as module, runtime_options

    if rows is not None:
        monkeypatch.setattr(module, "ONE_STREAM_ROWS", rows)
    spec = workloads.small_spec("stale", heads, 256, sequence - 256)
    backend = B200SparseBackend(HybridSparseConfig(video_budget=budget), smooth_k=smooth_k)
    options = runtime_options(spec.layout(), step_index=5, total_steps=20)
    gen = torch.Generator(device="cuda").manual_seed(heads)
    sets = [[(torch.randn((1, heads, sequence, 128), generator=gen, device="cuda") * size + size * shift).to(dtype) for shift in (0.0, 0.5, -0.2)]
            for size in (1.0, 60.0, 0.01)]
    for turn in range(6):
        q, k, v = sets[turn % 3]
        prepared = backend.prepare(q, k, v, layer_index=0, transformer_options=options)
        backend.execute(prepared)
        _same(prepared.sparse, k, v, smooth_k)


@pytest.mark.parametrize("smooth_k", [True, False])
@pytest.mark.parametrize("heads,sequence", [(8, 12544), (3, 2304)], ids=["long", "short"])
def test_projections(native_lib, heads, sequence, smooth_k):
    from h3_optimizations_b200 import ops
    from h3_optimizations_b200.projector import run_chunked_sparse_qkv

    x, w, w_scale = (t.cuda() for t in workloads.projection_inputs(sequence, hidden=256, heads=heads, seed=3))
    for turn in range(6):
        here = w_scale * (1.0, 60.0, 0.01)[turn % 3]
        got = run_chunked_sparse_qkv(x, w, here, heads=heads, chunk_rows=4096, smooth_k=smooth_k)
        codes, scale = ops.convrot_quant_rows(x)
        torch.cuda.synchronize()
        values = (codes.double() @ w.double().T).float() * (scale[:, None] * here[None, :])  # exact sums, the scales' product first
        _, k, v = values.to(torch.bfloat16).view(sequence, 3, heads, 128).permute(1, 2, 0, 3)[:, None].unbind(0)
        _same(got, k.contiguous(), v.contiguous(), smooth_k)
