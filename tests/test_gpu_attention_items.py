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


def _again(bits, sequence, gen):
    """Q and K of one head whose first tile, walked last, scores ``bits`` above the others: up to 21 bits nothing is left
    out, up to 128 the noted tiles are walked once more, beyond that twice."""
    q, k = torch.randn((2, sequence, 128), generator=gen)
    step = (bits / (2 * 128 * 128 ** -0.5 * 1.4426950408889634)) ** 0.5
    sign = -torch.ones(sequence)
    sign[:64] = 1.0
    return q + step, k + step * sign[:, None]


def test_results_do_not_depend_on_how_often_the_items_before_were_walked(native_lib):
    """Three kinds of heads, of one, two and three walks, in an order without a period: the same bits for every head of a kind."""
    from h3_optimizations_b200 import ops

    sequence, heads = 64 * 11 - 3, 180
    gen = torch.Generator().manual_seed(6)
    q, k = (torch.stack(t) for t in zip(*[_again(bits, sequence, gen) for bits in (0.0, 48.0, 300.0)]))
    v = torch.randn((3, sequence, 128), generator=gen)
    kind = torch.randint(0, 3, (heads,), generator=gen)
    q8, qs = oracle.quantize_blocks(q[None], 128)
    k8, ks = oracle.quantize_blocks(k[None], 64)
    vc, vs = oracle.v_fp8_carrier(v[None])
    args = [t.view(torch.uint8)[:, kind].view(t.dtype).contiguous().cuda() if t.dtype == torch.float8_e4m3fn else t[:, kind].contiguous().cuda()
            for t in (q8, k8, vc, qs, ks, vs)]
    geo = oracle.geometry(sequence, 0)
    out = ops.sparse_attention(*args, None, q_start=geo.pure_video_q_start, q_stop=geo.pure_video_q_stop, out_dtype=torch.float32).cpu()
    ref = oracle.sparse_attention_int8_fp8(q8, qs, k8, ks, vc, vs, geo, None)
    for i in range(3):
        mine = out[:, kind == i]
        assert torch.equal(mine, mine[:, :1].expand_as(mine)), i
        assert oracle.compare(mine[:, :1], ref[:, i:i + 1])["rel_max_abs"] <= 2.0 ** -8, i


@pytest.mark.parametrize("heads,sequence", [(2, 1601), (1, 5000)])
def test_parts_give_the_same_bits_every_time(native_lib, heads, sequence):
    from h3_optimizations_b200 import _native, ops

    assert _native.load().h3s_sparse_attn_half_workspace_bytes(heads, sequence, 0, 0, 0) > 0
    gen = torch.Generator().manual_seed(sequence)
    q, k = (torch.stack(t)[None] for t in zip(*[_again(48.0, sequence, gen) for _ in range(heads)]))
    v = torch.randn((1, heads, sequence, 128), generator=gen)
    args = [t.cuda() for t in (*oracle.quantize_blocks(q, 128), *oracle.quantize_blocks(k, 64), *oracle.v_fp8_carrier(v))]
    q8, qs, k8, ks, vc, vs = args
    run = lambda: ops.sparse_attention(q8, k8, vc, qs, ks, vs, None, q_start=0, q_stop=-(-sequence // 128), out_dtype=torch.float32)
    first = run()
    for _ in range(8):
        assert torch.equal(run(), first)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("heads,sequence", [(60, 541), (2, 1601)])  # more items than SMs; rows in parts
def test_further_outputs_hold_what_the_own_one_does(native_lib, heads, sequence, dtype):
    """A staged tile is still being copied to the other outputs when the CTA's next item is under way."""
    from h3_optimizations_b200 import ops

    spec = workloads.small_spec("items", heads, 0, sequence)
    q, k, v = (t.cuda() for t in workloads.gaussian_qkv(spec, seed=3))
    q8, qs, _ = ops.quant_qk_blocks(q, 128)
    k8, ks, _ = ops.quant_qk_blocks(k, 64)
    vs = ops.column_stats(None, v)[1]
    args = (q8, k8, ops.quant_v_fp8(v, vs)[0], qs, ks, vs, None)
    rows = {"q_start": 0, "q_stop": -(-sequence // 128)}
    plain = ops.sparse_attention(*args, **rows, out_dtype=dtype).contiguous()
    for _ in range(3):
        local, *others = (torch.full((1, heads, sequence, 128), float("nan"), dtype=dtype, device="cuda") for _ in range(8))
        ops.sparse_attention(*args, **rows, out=local, peer_out_ptrs=[t.data_ptr() for t in others])
        assert torch.equal(local, plain) and all(torch.equal(t, plain) for t in others)
