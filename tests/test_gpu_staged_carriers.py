"""K and V of a projected layer, on both sides of the line between one launch and several, bit for bit.  Needs a B200."""

import pytest
import torch

from h3_optimizations_b200 import workloads
from oracle import h3_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("smooth_k", [True, False])
@pytest.mark.parametrize("heads,sequence", [(1, 1), (3, 63), (2, 65), (3, 129), (2, 1000), (1, 100_000), (1, 100_001)])
def test_against_the_oracle(native_lib, heads, sequence, smooth_k):
    from h3_optimizations_b200.projector import run_chunked_sparse_qkv

    x, w, w_scale = workloads.projection_inputs(sequence, hidden=256, heads=heads, seed=sequence)
    w_scale[heads * 128 + 3] = w_scale[2 * heads * 128 + 7] = 0.0  # a channel of K and one of V that are zero throughout
    w_scale[heads * 128 + 90] *= 1000.0
    got = run_chunked_sparse_qkv(x.cuda(), w.cuda(), w_scale.cuda(), heads=heads, chunk_rows=512 if sequence < 2000 else 4096, smooth_k=smooth_k)
    x_i8, x_scale = oracle.convrot_quantize_rows(x)
    _, k, v = oracle.split_heads_hnd(oracle.qkv_project_int8(x_i8, x_scale, w, w_scale), heads)
    mean = k.double().mean(dim=2).to(torch.float32).to(torch.bfloat16).float() if smooth_k else None
    codes, scale = oracle.quantize_blocks(k, 64, mean=mean)
    assert torch.equal(got.k_int8.cpu(), codes) and torch.equal(got.k_scale.cpu(), scale)
    carrier, v_scale = oracle.v_fp8_carrier(v)
    half = got._v.half.cpu()
    assert torch.equal(got.v_scale.cpu(), v_scale)
    codes, want = got.v_carrier.cpu().view(torch.uint8), carrier.view(torch.uint8)
    want[want == 0x80] = 0  # -0 of the zero channel is written as 0
    assert torch.equal(torch.where(codes == 0x80, 0, codes), want) and torch.equal(half, got.v_carrier.cpu().to(torch.float16))
