"""Host calls whose outputs are copied out in pieces.  Needs a B200."""

import pytest
import torch

from h3_optimizations_b200 import B200SparseBackend, HybridSparseConfig, runtime_options, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [1, 7000, 10**9])
@pytest.mark.parametrize("heads,chunk", [(1, 1), (3, 1), (5, 2), (4, 4)])
def test_pieces_change_nothing(native_lib, monkeypatch, heads, chunk, size):
    from h3_optimizations_b200 import backend as module

    spec = workloads.small_spec("pieces", heads, 64, 333)
    host = [t.pin_memory() for t in workloads.gaussian_qkv(spec, seed=heads)]
    options = runtime_options(spec.layout(), step_index=5, total_steps=30)
    backend = B200SparseBackend(HybridSparseConfig(video_budget=0.3))
    prepared = backend.prepare(*(t.cuda() for t in host), layer_index=0, transformer_options=options)
    expected = backend.execute(prepared).cpu()  # lists too short to be cut, so the same sums for any number of heads
    monkeypatch.setattr(module, "COPY_OUT_BYTES", size)
    for _ in range(2):
        out = backend.forward_host(*host, layer_index=0, transformer_options=options, heads_per_chunk=chunk)
        assert torch.equal(out, expected)
