"""Arguments of the chunked projection that end in an error, or in a default value.  Needs a B200."""

import pytest
import torch

from h3_optimizations_b200 import workloads

pytestmark = pytest.mark.gpu


def test_a_refused_projection_leaves_a_capture_usable(native_lib):
    """The second stream joins only what it was forked from: a call that is refused before the fork must not
    make the captured stream wait for one outside the capture."""
    from h3_optimizations_b200.errors import FusedQKVError
    from h3_optimizations_b200.projector import run_chunked_sparse_qkv

    heads, hidden = 1, 128                                                         # ConvRot works on groups of 256
    x = torch.randn((300, hidden), device="cuda").to(torch.bfloat16)
    w = torch.zeros((3 * heads * 128, hidden), dtype=torch.int8, device="cuda")
    scale = torch.ones(3 * heads * 128, device="cuda")
    with pytest.raises(FusedQKVError, match="multiple of 256"):                    # the first call makes the second stream
        run_chunked_sparse_qkv(x, w, scale, heads=heads)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        with pytest.raises(FusedQKVError, match="multiple of 256"):
            run_chunked_sparse_qkv(x, w, scale, heads=heads)
        doubled = x + x
    x.fill_(3.0)
    graph.replay()
    torch.cuda.synchronize()
    assert bool((doubled == 6.0).all())


def test_summary_type_none_is_the_default_type(native_lib):
    from h3_optimizations_b200.projector import run_chunked_sparse_qkv

    x, w, w_scale = (t.cuda() for t in workloads.projection_inputs(300, hidden=256, heads=1, seed=4))
    default = run_chunked_sparse_qkv(x, w, w_scale, heads=1)
    none = run_chunked_sparse_qkv(x, w, w_scale, heads=1, summary_dtype=None)
    assert none.q_summary.dtype == torch.float32
    assert torch.equal(none.q_summary, default.q_summary) and torch.equal(none.k_summary, default.k_summary)
