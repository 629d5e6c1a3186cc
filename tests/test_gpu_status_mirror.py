"""The mirror of the status words in host memory.  Needs a B200.

The kernel that gives up writes both; the wait is made to run out as in test_gpu_bounded_wait (a load that is never
issued, a budget of a millisecond)."""

import pytest
import torch

from .test_gpu_bounded_wait import K_V_TILE_LOAD, _carriers, short_budget  # noqa: F401

pytestmark = pytest.mark.gpu


def test_the_mirror_holds_the_words(short_budget):  # noqa: F811
    ops = short_budget
    args = _carriers(ops)
    status, mirror = torch.zeros(4, dtype=torch.int32, device="cuda"), torch.zeros(4, dtype=torch.int32).pin_memory()
    ops.sparse_attention(*args, status=status, status_mirror=mirror)
    torch.cuda.synchronize()
    assert mirror.tolist() == [0, 0, 0, 0]
    ops.sparse_attention(*args, status=status, status_mirror=mirror, extra_flags=ops.ATTN_TEST_DROP_KV_LOAD)
    torch.cuda.synchronize()
    assert mirror.tolist() == status.tolist() and mirror[0] == K_V_TILE_LOAD


def test_the_next_prepare_raises_until_the_words_are_cleared(short_budget):  # noqa: F811
    from h3_optimizations_b200 import B200SparseBackend, HybridSparseConfig, runtime_options, workloads
    from h3_optimizations_b200.errors import SparseSageError

    ops = short_budget
    spec = workloads.small_spec("mirror", 1, 64, 192)
    qkv = [t.cuda() for t in workloads.gaussian_qkv(spec, seed=1)]
    options = runtime_options(spec.layout(), step_index=5, total_steps=20)
    backend = B200SparseBackend(HybridSparseConfig(video_budget=0.3))

    def prepare():
        return backend.prepare(*qkv, layer_index=0, transformer_options=options)

    backend.execute(prepare())
    word, mirror = backend._status_slot(qkv[0].device)
    ops.sparse_attention(*_carriers(ops), status=word, status_mirror=mirror, extra_flags=ops.ATTN_TEST_DROP_KV_LOAD)
    torch.cuda.synchronize()
    for _ in range(2):
        with pytest.raises(SparseSageError, match="K/V tile load.*reported by an earlier launch"):
            prepare()
    with pytest.raises(SparseSageError, match="found by check_status"):
        backend.check_status()
    backend.execute(prepare())
    backend.check_status()


def test_the_projected_way_looks_at_it_too(native_lib):
    from h3_optimizations_b200 import B200SparseBackend, HybridSparseConfig, runtime_options, workloads
    from h3_optimizations_b200.errors import SparseSageError
    from h3_optimizations_b200.projector import run_chunked_sparse_qkv

    spec = workloads.small_spec("mirror", 1, 64, 192)
    options = runtime_options(spec.layout(), step_index=5, total_steps=20)
    x = torch.ones((256, 256), dtype=torch.bfloat16, device="cuda")
    w = torch.ones((384, 256), dtype=torch.int8, device="cuda")
    projected = run_chunked_sparse_qkv(x, w, torch.full((384,), 0.01, device="cuda"), heads=1)
    backend = B200SparseBackend(HybridSparseConfig(video_budget=0.3))
    backend.execute(backend.prepare_projected(projected, layer_index=0, transformer_options=options))
    torch.cuda.synchronize()
    backend._status_slot(x.device)[1].copy_(torch.tensor([K_V_TILE_LOAD, 0, 0, 1], dtype=torch.int32))
    with pytest.raises(SparseSageError, match="K/V tile load.*reported by an earlier launch"):
        backend.prepare_projected(projected, layer_index=0, transformer_options=options)
    with pytest.raises(SparseSageError, match="found by check_status"):
        backend.check_status()
    backend.execute(backend.prepare_projected(projected, layer_index=0, transformer_options=options))
    backend.check_status()
