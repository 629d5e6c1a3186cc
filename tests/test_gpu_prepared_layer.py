"""What ``prepare`` hands to ``execute``: carriers by address until somebody looks at them.  Needs a B200."""

import copy
import dataclasses

import pytest
import torch

from h3_optimizations_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture()
def layer(native_lib):
    from h3_optimizations_b200 import B200SparseBackend, HybridSparseConfig, runtime_options

    def make(heads=2, video=1500, budget=0.3, **kwargs):
        spec = workloads.small_spec("layer", heads, 192, video)
        qkv = [t.cuda() for t in workloads.gaussian_qkv(spec, seed=heads)]
        backend = B200SparseBackend(HybridSparseConfig(video_budget=budget), **kwargs)
        options = runtime_options(spec.layout(), step_index=5, total_steps=20)
        return backend, lambda: backend.prepare(*qkv, layer_index=0, transformer_options=options)

    return make


@pytest.mark.parametrize("budget", [0.3, 1.0])
def test_looking_at_the_carriers_changes_nothing(layer, budget):
    backend, prepare = layer(budget=budget)
    prepared = prepare()
    assert prepared.sparse.untouched() is not None
    expected = backend.execute(prepared)
    for names in (["q_int8"], ["v_scale", "k_scale"], ["v_carrier"], ["q_int8", "k_int8", "q_scale", "k_scale", "v_scale", "v_carrier"]):
        prepared = prepare()
        tensors = [getattr(prepared.sparse, name) for name in names]
        assert all(t.is_contiguous() and t.is_cuda for t in tensors) and prepared.sparse.untouched() is None
        if "v_carrier" in names:
            assert prepared.sparse._buffers.v_half is None  # dropped: whoever holds the codes may write to them
        assert torch.equal(backend.execute(prepared), expected)


def test_copies_and_replacements(layer):
    backend, prepare = layer()
    expected = backend.execute(prepare())
    prepared = prepare()
    for other in (copy.copy(prepare().sparse), copy.deepcopy(prepare().sparse), dataclasses.replace(prepare().sparse, layer_index=3)):
        assert torch.equal(backend.execute(dataclasses.replace(prepared, sparse=other)), expected)
    twin = copy.copy(prepared.sparse)  # a copy's codes are the same memory: neither may go by an older copy of V
    twin.v_carrier.zero_()
    assert not backend.execute(prepared).any()
    prepared = prepare()
    prepared.sparse.v_scale = prepared.sparse.v_scale * 2
    assert torch.equal(backend.execute(prepared), (expected.float() * 2).to(expected.dtype))
    with pytest.raises(AttributeError):
        prepared.sparse.no_such_field


@pytest.mark.parametrize("smooth_k", [False, True])
@pytest.mark.parametrize("budget", [0.3, 1.0])
def test_one_stream_and_two_prepare_the_same(layer, monkeypatch, budget, smooth_k):
    from h3_optimizations_b200 import backend as module

    results = []
    for rows in (0, 10**9):
        monkeypatch.setattr(module, "ONE_STREAM_ROWS", rows)
        backend, prepare = layer(heads=3, video=1333, budget=budget, smooth_k=smooth_k)
        sparse = prepare().sparse
        results.append([sparse.q_int8, sparse.k_int8, sparse.q_scale, sparse.k_scale, sparse.v_scale, sparse.v_carrier.view(torch.uint8)]
                       + ([] if sparse.route.indices is None else [sparse.route.indices]))
        graph = torch.cuda.CUDAGraph()
        expected = backend.execute(prepare())
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, capture_error_mode="thread_local"):
            out = backend.execute(prepare())
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, expected)
    assert all(torch.equal(a, b) for a, b in zip(*results))


def test_a_short_call_leaves_nothing_to_a_capture(layer, monkeypatch):
    """The second stream is there before a capture, which uses it, although the calls before it did not."""
    from h3_optimizations_b200 import ops

    taken = []
    for name in ("prepare_layer", "quant_qkv"):
        real = getattr(ops, name)
        monkeypatch.setattr(ops, name, lambda *args, _name=name, _real=real, **kwargs: taken.append(_name) or _real(*args, **kwargs))
    backend, prepare = layer(heads=4, video=5808)
    expected = backend.execute(prepare())
    assert taken == ["prepare_layer"] and len(backend._side_streams) == 1
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        out = backend.execute(prepare())
    assert taken == ["prepare_layer", "quant_qkv"] and len(backend._side_streams) == 1
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        # the K mean's FP64 sum is gathered with atomics, in any order: its rounding is the same but for ties
        assert (out.float() - expected.float()).abs().max() <= 2.0 ** -8 * expected.float().abs().max()
