"""Which memory the attention kernels write to.  Needs a B200.

An output that the device cannot reach is refused on the host, before anything is launched; pinned host memory gets what
device memory gets."""

import pytest
import torch

from h3_optimizations_b200 import B200SparseBackend, HybridSparseConfig, runtime_options, workloads

pytestmark = pytest.mark.gpu

KERNELS = {"half": {}, "two_terms": {"two_term_p": True}, "one_term": {"single_term_p": True}, "mma": {"legacy_mma": True}}


def _carriers(ops):
    spec = workloads.small_spec("memory", 2, 0, 200)
    q, k, v = (t.cuda() for t in workloads.gaussian_qkv(spec, seed=7))
    k_mean, v_scale = ops.column_stats(k, v)
    q8, qs, _ = ops.quant_qk_blocks(q, 128)
    k8, ks, _ = ops.quant_qk_blocks(k, 64, mean=k_mean)
    vc, _ = ops.quant_v_fp8(v, v_scale)
    return q8, k8, vc, qs, ks, v_scale


@pytest.mark.parametrize("kernel", list(KERNELS))
def test_pageable_memory_is_refused(native_lib, kernel):
    from h3_optimizations_b200 import _native, ops

    args = _carriers(ops)
    pageable = torch.full((1, 2, 200, 128), 77.0, dtype=torch.bfloat16)
    with pytest.raises(_native.NativeError, match="not memory that device"):
        ops.sparse_attention(*args, out=pageable, **KERNELS[kernel])
    torch.cuda.synchronize()
    assert bool((pageable == 77.0).all())
    pinned = pageable.pin_memory()
    ops.sparse_attention(*args, out=pinned, **KERNELS[kernel])
    out = ops.sparse_attention(*args, **KERNELS[kernel])
    torch.cuda.synchronize()
    assert torch.equal(pinned, out.cpu())


def test_execute_refuses_it_too(native_lib):
    from h3_optimizations_b200.errors import SparseSageError

    spec = workloads.small_spec("memory", 2, 64, 640)
    qkv = [t.cuda() for t in workloads.gaussian_qkv(spec, seed=3)]
    backend = B200SparseBackend(HybridSparseConfig(video_budget=0.3))
    options = runtime_options(spec.layout(), step_index=5, total_steps=30)
    for touched in (False, True):  # both ways through execute()
        prepared = backend.prepare(*qkv, layer_index=0, transformer_options=options)
        if touched:
            prepared.sparse.q_scale
        with pytest.raises(SparseSageError, match="not memory that device"):
            backend.execute(prepared, out=torch.empty_like(qkv[0], device="cpu"))
        pinned = torch.empty_like(qkv[0], device="cpu").pin_memory()
        backend.execute(prepared, out=pinned)
        out = backend.execute(prepared)
        torch.cuda.synchronize()
        assert torch.equal(pinned, out.cpu())
    backend.check_status()


def test_pinned_memory_in_a_capture(native_lib):
    """Asking where an output is does not disturb a capture of any mode."""
    from h3_optimizations_b200 import ops

    args = _carriers(ops)
    half = ops.v_half_copy(args[2])
    out = ops.sparse_attention(*args, v_half=half)
    for mode in ("global", "thread_local", "relaxed"):
        pinned = torch.zeros((1, 2, 200, 128), dtype=torch.bfloat16).pin_memory()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, capture_error_mode=mode):
            ops.sparse_attention(*args, out=pinned, v_half=half)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(pinned, out.cpu())
