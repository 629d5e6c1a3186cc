"""The attention kernel's own error, and tiles that a row leaves out and comes back to.  Needs a B200.

P is rounded once to FP16: |error| <= 2^-11 * sum(p |v|) / sum(p), elementwise; the same oracle on
|V| gives that sum, and a factor of 2 leaves room for ex2.approx, the exponent's rounding (2^-15 of a
tile at these scales) and the FP32 order of summation.  In the 2-norm the rounding is a quarter of
that again; two E4M3 terms leave 1.2e-3 there, BF16 1.65e-3."""

import pytest
import torch

from h3_optimizations_b200 import workloads
from oracle import h3_oracle as oracle

pytestmark = pytest.mark.gpu


def _compare(q, k, v, geo, route, tiles=None):
    from h3_optimizations_b200 import ops

    sequence = q.shape[2]
    q8, qs = oracle.quantize_blocks(q, 128)
    k8, ks = oracle.quantize_blocks(k, 64)
    vc, vs = oracle.v_fp8_carrier(v)
    va, _ = oracle.v_fp8_carrier(v.abs())  # |V| has the same scales
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out = ops.sparse_attention(
        *(t.cuda() for t in (q8, k8, vc, qs, ks, vs)), None if route is None else route.cuda().contiguous(),
        q_start=geo.pure_video_q_start, q_stop=geo.pure_video_q_stop, status=status, out_dtype=torch.float32).cpu()
    assert status.tolist() == [0, 0, 0, 0]
    ref = oracle.sparse_attention_int8_fp8(q8, qs, k8, ks, vc, vs, geo, route, q_tile_subset=tiles)
    size = oracle.sparse_attention_int8_fp8(q8, qs, k8, ks, va, vs, geo, route, q_tile_subset=tiles)
    if tiles is not None:
        rows = torch.cat([torch.arange(t * 128, min(t * 128 + 128, sequence)) for t in tiles])
        out, ref, size = out[:, :, rows], ref[:, :, rows], size[:, :, rows]
    assert bool(((out - ref).abs() <= 2.0 ** -10 * size + 1e-6).all()), float(((out - ref).abs() / size).max())
    return float((out.double() - ref.double()).norm() / ref.double().norm())


@pytest.mark.parametrize("sequence", [64, 320, 2111, 4000])
def test_dense_error(native_lib, sequence):
    q, k, v = workloads.gaussian_qkv(workloads.small_spec("precision", 2, 0, sequence), seed=sequence, widen=True)
    assert _compare(q, k, v, oracle.geometry(sequence, 0), None) <= 5e-4


def test_routed_error(native_lib):
    q, k, v = workloads.gaussian_qkv(workloads.small_spec("precision", 2, 300, 3700), seed=5, widen=True)
    geo, _, _, route = oracle.build_route(q, k, 4000, 300, 0.2)
    assert _compare(q, k, v, geo, route) <= 5e-4


def _spikes(sequence, heads, tiles, seed):
    """Scores of every third row jump by 33, 98 or 163 bits in some tiles; other rows stay as they are."""
    q, k, v = workloads.gaussian_qkv(workloads.small_spec("spikes", heads, 0, sequence), seed=seed, widen=True)
    q[:, :, ::3] += 2.0
    for i, tile in enumerate(tiles):
        k[:, :, tile * 64:tile * 64 + 64] += (1.0, 3.0, 5.0)[i % 3]
    return q, k, v


# The walk begins with tiles 16 and 17.  One tile; neighbours, so that either group has some; a sum that overflows
# (the third); the ragged last tile; a reference tile; all but the reference tiles
@pytest.mark.parametrize("tiles", [[2], [7], [18, 19], [0, 9, 20], [1, 2, 3, 32], [32], [16, 3], [30, 17, 31],
                                   [t for t in range(33) if t not in (16, 17)]])
def test_tiles_left_out(native_lib, tiles):
    sequence = 64 * 32 + 40
    q, k, v = _spikes(sequence, 8, tiles, seed=len(tiles) + tiles[0])
    _compare(q, k, v, oracle.geometry(sequence, 0), None)


def test_tiles_left_out_of_parts_and_routed_lists(native_lib):
    heads, context, sequence = 2, 300, 4000
    q, k, v = _spikes(sequence, heads, [3, 20, 41, 62], seed=3)
    geo, _, _, route = oracle.build_route(q, k, sequence, context, 0.4)
    _compare(q, k, v, geo, route)


def test_tiles_left_out_of_a_list_longer_than_the_note(native_lib):
    """2188 tiles: a bit of the note stands for two."""
    sequence = 64 * 2187 + 9
    q, k, v = _spikes(sequence, 1, [2, 700, 701, 1500, 2186, 2187], seed=1)
    _compare(q, k, v, oracle.geometry(sequence, 0), None, tiles=[0, 500, 1093])


@pytest.mark.parametrize("scale", [1e2, 1e4, 1e5])
def test_scores_of_a_hundred_to_a_million_bits(native_lib, scale):
    """Finite, and no further off than at ordinary scales: what has the weight there is left out at first and walked
    again with the exponent's offset taken off exactly.  Against 64-bit arithmetic on the carriers."""
    from h3_optimizations_b200 import ops

    sequence, heads = 1000, 2
    q, k, v = workloads.gaussian_qkv(workloads.small_spec("scale", heads, 0, sequence), seed=6, widen=True)
    q8, qs = oracle.quantize_blocks(q * scale ** 0.5, 128)
    k8, ks = oracle.quantize_blocks(k * scale ** 0.5, 64)
    vc, vs = oracle.v_fp8_carrier(v)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out = ops.sparse_attention(*(t.cuda() for t in (q8, k8, vc, qs, ks, vs)), status=status, out_dtype=torch.float32).cpu()
    assert status.tolist() == [0, 0, 0, 0] and bool(torch.isfinite(out).all())
    z = q8[0].double() @ k8[0].double().transpose(1, 2) * 128 ** -0.5
    z *= qs[0].double().repeat_interleave(128, 1)[:, :sequence, None] * ks[0].double().repeat_interleave(64, 1)[:, None, :sequence]
    want = torch.softmax(z, -1) @ (vc[0, :, :, :sequence].double() * vs[0].double()[:, :, None]).transpose(1, 2)
    # 2^-11 of each probability; 2^-24 * c * 12582912 bits of a tile that was not left out, where c is about 1e-4 * scale
    # and such tiles have weight at the smaller scales only
    assert float((out[0].double() - want).norm() / want.norm()) <= 1e-3
