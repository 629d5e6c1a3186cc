"""Which item the status words name.  Needs a B200.

The last P.V of an item is waited for when its CTA has gone on to the next one, or has found that there is none.  The load
that it waits for is never issued (``H3S_ATTN_TEST_DROP_LAST_V_LOAD``, a budget of a millisecond as in
test_gpu_bounded_wait): the words must name the item whose load it was."""

import pytest
import torch

from h3_optimizations_b200 import workloads

from .test_gpu_bounded_wait import K_V_TILE_LOAD, short_budget  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,sequence", [(1, 64), (1, 128), (3, 300), (148, 64), (200, 64), (160, 400)])
@pytest.mark.parametrize("staged", [False, True], ids=["own_rows", "staged"])
def test_the_item_that_was_given_up(short_budget, heads, sequence, staged):  # noqa: F811
    ops = short_budget
    spec = workloads.small_spec("status", heads, 0, sequence)
    q, k, v = (t.cuda() for t in workloads.gaussian_qkv(spec, seed=1))
    k_mean, v_scale = ops.column_stats(k, v)
    q8, qs, _ = ops.quant_qk_blocks(q, 128)
    k8, ks, _ = ops.quant_qk_blocks(k, 64, mean=k_mean)
    vc, _ = ops.quant_v_fp8(v, v_scale)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    further = torch.empty((1, sequence, heads, 128), dtype=torch.bfloat16, device="cuda")
    peers = [further.data_ptr()] if staged else None
    ops.sparse_attention(q8, k8, vc, qs, ks, v_scale, status=status, peer_out_ptrs=peers, extra_flags=ops.ATTN_TEST_DROP_LAST_V_LOAD)
    torch.cuda.synchronize()
    code, item, head, tile = status.tolist()
    tiles = -(-sequence // 128)
    assert code == K_V_TILE_LOAD
    assert 0 <= head < heads and 0 <= tile < tiles and item == head * tiles + tile
    status.zero_()
    ops.sparse_attention(q8, k8, vc, qs, ks, v_scale, status=status)
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
