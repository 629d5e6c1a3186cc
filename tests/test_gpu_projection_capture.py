"""The whole attention block under CUDA graph capture, with and without K smoothing (only the
former uses the second stream).  Needs a B200."""

from types import SimpleNamespace

import pytest
import torch

from h3_optimizations_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("smooth_k", [True, False])
def test_a_captured_block_replays_on_new_inputs(native_lib, smooth_k):
    from h3_optimizations_b200 import B200SparseBackend, ChunkedSparseQKVProjector, HybridSparseConfig, runtime_options
    from h3_optimizations_b200.attention_forward import make_forward

    heads, hidden = 2, 512
    spec = workloads.small_spec("capture", heads, 100, 600)
    x, w, w_scale = workloads.projection_inputs(spec.sequence, hidden=hidden, heads=heads, seed=1)
    other = workloads.projection_inputs(spec.sequence, hidden=hidden, heads=heads, seed=2)[0].cuda()
    out_proj = torch.nn.Linear(heads * 128, hidden, bias=False, device="cuda", dtype=torch.bfloat16)
    module = SimpleNamespace(heads=heads, head_dim=128, out_proj=out_proj, qkv_weight_int8=w.cuda(), qkv_weight_scale=w_scale.cuda())
    forward = make_forward(module, 0, backend=B200SparseBackend(HybridSparseConfig(video_budget=0.4), smooth_k=smooth_k),
                           projector=ChunkedSparseQKVProjector(chunk_rows=256, smooth_k=smooth_k))
    options = runtime_options(spec.layout())
    held = x.cuda()
    with torch.no_grad():
        for _ in range(2):
            forward(held, None, options)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = forward(held, None, options)
        held.copy_(other)
        graph.replay()
        want = forward(other, None, options)
    torch.cuda.synchronize()
    # the K mean's FP64 sum is gathered with atomics, in any order: equal but for a rare rounding
    assert (out.float() - want.float()).abs().max() <= 2.0 ** -7 * want.float().abs().max()
