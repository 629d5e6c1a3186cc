"""Attention CTAs that go through several items.  Needs a B200.

A CTA takes query tile after query tile; four softmax groups take every fourth KV tile, and
which group begins, which slot and which barrier phase an item begins with depend on the items before it.
So: more items than SMs, lists of all lengths around the numbers of groups, slots and
stages, both output layouts; inputs, oracle and bound are those of test_gpu_attention_tiles."""

import pytest
import torch

from h3_optimizations_b200 import workloads
from oracle import h3_oracle as oracle

from .test_gpu_attention_tiles import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 5, 7, 9, 16, 17])
def test_more_lists_than_processors(native_lib, tiles):
    sequence, heads = 64 * tiles - 7, 640 // (tiles + 1)
    spec = workloads.small_spec("items", heads, 0, sequence)
    q, k, v = workloads.gaussian_qkv(spec, seed=tiles, widen=True)
    _check(native_lib, q, k, v, oracle.geometry(sequence, 0), None)


@pytest.mark.parametrize("keep", [1, 5, 6])
def test_lists_of_two_lengths(native_lib, keep):
    """Dense items, then routed ones of another length; some are walked again."""
    context, sequence, heads = 130, 130 + 1400, 40
    spec = workloads.small_spec("items", heads, context, 1400)
    q, k, v = workloads.gaussian_qkv(spec, seed=keep, widen=True)
    geo, _, _, route = oracle.build_route(q, k, sequence, context, keep / 21)
    sign = -torch.ones(sequence)  # every third head: the first tiles, walked last, about 300 bits above the others
    sign[:128] = 1.0
    q[:, ::3] += 3.0
    k[:, ::3] += 3.0 * sign[:, None]
    _check(native_lib, q, k, v, geo, route)


def test_results_do_not_depend_on_the_items_before(native_lib):
    """The same rows, bit for bit, whatever their place in the launch."""
    from h3_optimizations_b200 import ops

    sequence, heads = 64 * 11 - 3, 200
    spec = workloads.small_spec("items", heads, 0, sequence)
    q, k, v = (t[:, :1].expand(1, heads, sequence, 128).contiguous() for t in workloads.gaussian_qkv(spec, seed=1, widen=True))
    q8, qs = oracle.quantize_blocks(q[:, :1], 128)
    k8, ks = oracle.quantize_blocks(k[:, :1], 64)
    vc, vs = oracle.v_fp8_carrier(v[:, :1])
    args = [t.repeat(1, heads, *[1] * (t.ndim - 2)).contiguous().cuda() for t in (q8, k8, vc, qs, ks, vs)]
    geo = oracle.geometry(sequence, 0)
    out = ops.sparse_attention(*args, None, q_start=geo.pure_video_q_start, q_stop=geo.pure_video_q_stop, out_dtype=torch.float32)
    assert torch.equal(out, out[:, :1].expand_as(out))
