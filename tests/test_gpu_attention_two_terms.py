"""The tcgen05 kernel that reads the E4M3 carrier itself (``h3s_sparse_attn_fwd`` and ``_scatter``), with P as two
E4M3 terms or one.  Needs a B200.

The oracle rounds the probabilities as this kernel does, but for the lazily raised reference point: it shifts P by
a power of two, which matters only where P meets E4M3's smallest values.  Bounds are those of test_gpu_attention."""

import pytest
import torch

from h3_optimizations_b200 import workloads
from oracle import h3_oracle as oracle

from .test_gpu_attention import CASES, TIGHT_COS, TIGHT_REL, _carriers, _run

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


# and a list of one ragged tile, of one full tile, of an odd number
@pytest.mark.parametrize("sequence,video_start,heads,budget", CASES + [(40, 0, 1, 1.0), (64, 0, 2, 1.0), (2111, 0, 2, 1.0)])
def test_two_terms_against_the_oracle(ops, sequence, video_start, heads, budget):
    carriers, geo, route = _case(sequence, video_start, heads, budget, seed=sequence)
    out = _run(ops, carriers, route, geo, out_dtype=torch.float32, two_term_p=True)
    m = oracle.compare(out.cpu(), oracle.sparse_attention_int8_fp8(*carriers, geo, route, p_format="e4m3x2"))
    assert m["cosine"] >= TIGHT_COS and m["rel_max_abs"] <= TIGHT_REL, m
    assert torch.equal(_run(ops, carriers, route, geo, out_dtype=torch.float32, two_term_p=True), out)
    for dtype in (torch.bfloat16, torch.float16):
        assert torch.equal(_run(ops, carriers, route, geo, out_dtype=dtype, two_term_p=True), out.to(dtype))


@pytest.mark.parametrize("tiles", [2, 3, 8])
def test_scores_that_rise_by_hundreds_of_bits(ops, tiles):
    sequence = 64 * tiles - 5
    q, k, v = workloads.gaussian_qkv(workloads.small_spec("terms", 2, 0, sequence), seed=tiles, widen=True)
    sign = torch.ones(sequence)
    sign[:64] = -1.0
    q, k, geo = q + 3.0, k + 3.0 * sign[:, None], oracle.geometry(sequence, 0)
    carriers = _carriers(q, k, v)
    out = _run(ops, carriers, None, geo, out_dtype=torch.float32, two_term_p=True).cpu()
    ref = oracle.sparse_attention_int8_fp8(*carriers, geo, None)
    size = oracle.sparse_attention_int8_fp8(*_carriers(q, k, v.abs()), geo, None)
    # two terms of four significant bits: 2^-8 of P, but no less than half of E4M3's last unit, 2^-10, where the
    # largest P is 2^6 or more; a tenth for ex2.approx and the order of summation
    bound = 1.1 * 2.0 ** -8 * size + 2.0 ** -16 * v.abs().sum(dim=2, keepdim=True)
    assert bool(((out - ref).abs() <= bound).all()), float(((out - ref).abs() / bound).max())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_scatter_writes_every_extra_buffer(ops, dtype):
    carriers, geo, route = _case(541, 100, 2, 0.4, seed=7)
    plain = _run(ops, carriers, route, geo, out_dtype=dtype, two_term_p=True)
    peers = [torch.full((1, 5, 541, 128), float("nan"), dtype=dtype, device="cuda") for _ in range(3)]
    local = torch.empty((1, 2, 541, 128), dtype=dtype, device="cuda")
    got = _run(ops, carriers, route, geo, out=local, peer_out_ptrs=[p[:, 2:4].data_ptr() for p in peers], two_term_p=True)
    assert torch.equal(got, plain.contiguous())
    for p in peers:
        assert torch.equal(p[:, 2:4], plain.contiguous())
        assert bool(torch.isnan(p[:, :2].float()).all()) and bool(torch.isnan(p[:, 4:].float()).all())


def test_an_expired_wait_reports_and_leaves_the_device_usable(ops):
    """As in test_gpu_bounded_wait: the first K/V load is not issued, the wait for it runs out after 1 ms."""
    carriers, geo, _ = _case(128, 0, 1, 1.0, seed=5)
    args = [t.cuda() for t in carriers]
    args = [args[0], args[2], args[4], args[1], args[3], args[5]]
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    good = ops.sparse_attention(*args, out_dtype=torch.float32, status=status, two_term_p=True)
    previous = ops.set_wait_budget_ns(1_000_000)
    try:
        ops.sparse_attention(*args, out_dtype=torch.float32, status=status, two_term_p=True, extra_flags=ops.ATTN_TEST_DROP_KV_LOAD)
        torch.cuda.synchronize()
    finally:
        ops.set_wait_budget_ns(previous)
    assert status.tolist() == [2, 0, 0, 0]  # the K/V tile load, in the first CTA
    status.zero_()
    again = ops.sparse_attention(*args, out_dtype=torch.float32, status=status, two_term_p=True)
    assert status.tolist() == [0, 0, 0, 0] and torch.equal(again, good)
