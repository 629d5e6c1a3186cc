"""Dense rows whose tile list is cut into parts.  Needs a B200.  Inputs, oracle and bound are
those of test_gpu_attention_tiles; the reference points are integers, so adding up the parts
is exact but for the order of the FP32 sums, for which that bound has room."""

import pytest
import torch

from h3_optimizations_b200 import workloads
from oracle import h3_oracle as oracle

from .test_gpu_attention_tiles import _check

pytestmark = pytest.mark.gpu


def _workspace(heads, sequence, route_len=0, q_start=0, q_stop=0):
    from h3_optimizations_b200 import _native

    return _native.load().h3s_sparse_attn_half_workspace_bytes(heads, sequence, route_len, q_start, q_stop)


# 25 tiles: parts of 13 and 12; a last part of one ragged tile less; more parts
@pytest.mark.parametrize("heads,sequence", [(2, 1537), (1, 64 * 49 + 1), (3, 4000)])
def test_all_rows_dense(native_lib, heads, sequence):
    assert _workspace(heads, sequence) > 0
    spec = workloads.small_spec("split", heads, 0, sequence)
    q, k, v = workloads.gaussian_qkv(spec, seed=sequence, widen=True)
    _check(native_lib, q, k, v, oracle.geometry(sequence, 0), None)


def test_long_rows_beside_routed_ones(native_lib):
    context, sequence = 300, 300 + 3700
    spec = workloads.small_spec("split", 2, context, 3700)
    q, k, v = workloads.gaussian_qkv(spec, seed=9, widen=True)
    geo, _, _, route = oracle.build_route(q, k, sequence, context, 0.1)
    assert _workspace(2, sequence, route.shape[-1], geo.pure_video_q_start, geo.pure_video_q_stop) > 0
    _check(native_lib, q, k, v, geo, route)


@pytest.mark.parametrize("low", [slice(0, 900), slice(900, 1601), slice(0, 64)])
def test_parts_whose_scores_lie_hundreds_of_bits_apart(native_lib, low):
    """One part's sums vanish beside another's, or a part has to come back to tiles that it left out."""
    sequence = 1601
    assert _workspace(2, sequence) > 0
    spec = workloads.small_spec("split", 2, 0, sequence)
    q, k, v = workloads.gaussian_qkv(spec, seed=4, widen=True)
    sign = torch.ones(sequence)
    sign[low] = -1.0
    q, k = q + 3.0, k + 3.0 * sign[:, None]
    _check(native_lib, q, k, v, oracle.geometry(sequence, 0), None)


def test_no_parts_where_the_rows_fill_the_chip(native_lib):
    assert _workspace(24, 33272) == 0 and _workspace(8, 700) == 0
    assert _workspace(24, 33272, 162, 4, 260) == 0 and _workspace(3, 33272, 162, 4, 260) > 0
