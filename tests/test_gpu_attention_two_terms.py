"""The tcgen05 kernel that reads the E4M3 carrier itself.  Needs a B200."""

import pytest
import torch

from h3_optimizations_b200 import workloads
from oracle import h3_oracle as oracle

from .test_gpu_attention import _carriers, _run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(native_lib):
    from h3_optimizations_b200 import ops as module

    return module


def _case(sequence, video_start, heads, budget, seed):
    spec = workloads.small_spec("terms", heads, video_start, sequence - video_start)
    q, k, v = workloads.gaussian_qkv(spec, seed=seed, widen=True)
    geo, _, _, route = oracle.build_route(q, k, sequence, video_start, budget)
    return _carriers(q, k, v), geo, route


def test_the_single_term_may_be_asked_for_by_its_flag(ops):
    carriers, geo, route = _case(640, 128, 2, 0.3, seed=2)
    named = _run(ops, carriers, route, geo, out_dtype=torch.float32, single_term_p=True)
    assert torch.equal(_run(ops, carriers, route, geo, out_dtype=torch.float32, extra_flags=ops.ATTN_P_SINGLE), named)
