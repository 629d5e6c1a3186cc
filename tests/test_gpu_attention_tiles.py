"""Attention kernel at the edges of its tile loop.  Needs a B200.

Each of four softmax groups takes every fourth KV tile, and three tiles of scores are ahead of them, so lists of
one to six tiles are the interesting lengths, with full and ragged last tiles.  The bound
is elementwise, 2^-8 * sum(p |v|) / sum(p) from the same oracle on |V|: room for probabilities of
eight significant bits, or for FP16's where one key has nearly all the weight and the others lie
close to its smallest value.  test_gpu_attention_precision has the close bound for FP16, and the
tiles that a row leaves out and comes back to."""

import pytest
import torch

from h3_optimizations_b200 import workloads
from oracle import h3_oracle as oracle

pytestmark = pytest.mark.gpu


def _check(native_lib, q, k, v, geo, route):
    from h3_optimizations_b200 import ops

    q8, qs = oracle.quantize_blocks(q, 128)
    k8, ks = oracle.quantize_blocks(k, 64)
    vc, vs = oracle.v_fp8_carrier(v)
    va, _ = oracle.v_fp8_carrier(v.abs())  # |V| has the same scales
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out = ops.sparse_attention(
        *(t.cuda() for t in (q8, k8, vc, qs, ks, vs)), None if route is None else route.cuda().contiguous(),
        q_start=geo.pure_video_q_start, q_stop=geo.pure_video_q_stop, status=status, out_dtype=torch.float32).cpu()
    assert status.tolist() == [0, 0, 0, 0]
    ref = oracle.sparse_attention_int8_fp8(q8, qs, k8, ks, vc, vs, geo, route)
    size = oracle.sparse_attention_int8_fp8(q8, qs, k8, ks, va, vs, geo, route)
    assert bool(((out - ref).abs() <= 2.0 ** -8 * size + 1e-6).all()), float(((out - ref).abs() / size).max())


@pytest.mark.parametrize("sequence", [1, 63, 64, 65, 128, 129, 192, 257, 320, 384, 2112])
def test_dense_lists_of_few_tiles(native_lib, sequence):
    spec = workloads.small_spec("edge", 2, 0, sequence)
    q, k, v = workloads.gaussian_qkv(spec, seed=sequence, widen=True)
    _check(native_lib, q, k, v, oracle.geometry(sequence, 0), None)


@pytest.mark.parametrize("keep", [1, 2, 3])
def test_routed_lists_of_few_tiles(native_lib, keep):
    sequence = 640 + 17
    spec = workloads.small_spec("edge", 1, 0, sequence)
    q, k, v = workloads.gaussian_qkv(spec, seed=keep, widen=True)
    geo, _, _, route = oracle.build_route(q, k, sequence, 0, keep / 11)
    assert route.shape[-1] == keep
    _check(native_lib, q, k, v, geo, route)


@pytest.mark.parametrize("tiles", [2, 3, 5, 8])
def test_scores_that_outgrow_the_first_tile(native_lib, tiles):
    """The first tile scores about -150 bits, the last ones +150."""
    sequence = 64 * tiles - 5
    spec = workloads.small_spec("edge", 2, 0, sequence)
    q, k, v = workloads.gaussian_qkv(spec, seed=tiles, widen=True)
    sign = torch.ones(sequence)
    sign[:64] = -1.0
    q, k = q + 3.0, k + 3.0 * sign[:, None]
    _check(native_lib, q, k, v, oracle.geometry(sequence, 0), None)


def test_many_short_lists_that_are_walked_again(native_lib):
    """The first of the tiles, walked last, is far above the others: three passes over a list of three tiles, one of which
    is noted, in item after item."""
    sequence, heads = 187, 900                                                    # 1800 items on 148 SMs
    spec = workloads.small_spec("edge", heads, 0, sequence)
    q, k, v = workloads.gaussian_qkv(spec, seed=12, widen=True)
    sign = -torch.ones(sequence)
    sign[:64] = 1.0
    q, k = q + 3.0, k + 3.0 * sign[:, None]
    _check(native_lib, q, k, v, oracle.geometry(sequence, 0), None)
