"""RMS norm in the carrier epilogue over the range of its sums of squares.  Needs a B200.

The sum is kept as a pair of floats while every step is exact, else in 64 bits: heads whose
values lie on both sides of both ends of that range, and a head of zeros, have to give the oracle's codes."""

from types import SimpleNamespace

import pytest
import torch

from h3_optimizations_b200 import workloads
from oracle import h3_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("epsilon", [1e-6, 1e-30])
def test_codes_of_heads_of_all_sizes(native_lib, epsilon):
    from h3_optimizations_b200 import ChunkedSparseQKVProjector

    sizes = (1.0, 0.0, 1e-13, 1e-11, 1e16, 1e18, 1e20)  # the last one's sum is infinite
    heads, hidden, rows = len(sizes), 512, 300
    x, w, w_scale = workloads.projection_inputs(rows, hidden=hidden, heads=heads, seed=11)
    w_scale = w_scale * torch.tensor(sizes).repeat_interleave(128).repeat(3)
    gen = torch.Generator().manual_seed(5)
    weight = (torch.rand(128, generator=gen) + 0.5).to(torch.bfloat16)
    norm = SimpleNamespace(weight=weight.cuda(), eps=epsilon)
    module = SimpleNamespace(heads=heads, head_dim=128, qkv_weight_int8=w.cuda(), qkv_weight_scale=w_scale.cuda(),
                             q_norm=norm, k_norm=norm)
    got = ChunkedSparseQKVProjector(smooth_k=False).project(module, x.cuda(), None, layer_index=0, transformer_options={})
    x_i8, x_scale = oracle.convrot_quantize_rows(x)
    y = oracle.rms_norm_rope_split_half(oracle.qkv_project_int8(x_i8, x_scale, w, w_scale), heads, weight, weight, epsilon, None)
    q, k, _ = oracle.split_heads_hnd(y, heads)
    for name, values, block, codes, scale in (("q", q, 128, got.q_int8, got.q_scale), ("k", k, 64, got.k_int8, got.k_scale)):
        want, want_scale = oracle.quantize_blocks(values, block)
        assert torch.equal(scale.cpu().reshape(want_scale.shape), want_scale), name
        assert torch.equal(codes.cpu().reshape(want.shape), want), name
