"""Kernels that are launched before the one in front of them has ended.  Needs a B200.

Calls issued back to back, over scratch memory that the allocator hands from one to the next, give the same bits as calls
with the device idle before each of them, and so does a captured graph of them."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _mlp():
    from h3_optimizations_b200.mlp import ChunkedFP8MLP

    gen = torch.Generator(device="cuda").manual_seed(0)
    w1, w2 = (torch.randn(s, generator=gen, device="cuda") * 0.05 for s in ((1024, 256), (256, 1024)))
    mlp = ChunkedFP8MLP(w1, None, w2, None, chunk_rows=128)
    return mlp, [torch.randn((n, 256), generator=gen, device="cuda").bfloat16() for n in (300, 1, 517, 128, 2000, 129)]


def _layer(heads=2):
    from h3_optimizations_b200 import B200SparseBackend, HybridSparseConfig, runtime_options, workloads

    spec = workloads.small_spec("chain", heads, 192, 1500)
    options = runtime_options(spec.layout(), step_index=5, total_steps=20)
    backend = B200SparseBackend(HybridSparseConfig(video_budget=0.3), smooth_k=False)  # no sums whose order is free
    inputs = [[t.cuda() for t in workloads.gaussian_qkv(spec, seed=s)] for s in range(6)]
    return lambda x: backend.execute(backend.prepare(*x, layer_index=0, transformer_options=options)), inputs


@pytest.mark.parametrize("make", [_mlp, _layer], ids=["mlp", "layer"])
def test_back_to_back_is_the_same_as_one_by_one(native_lib, make):
    call, inputs = make()
    one_by_one = []
    for x in inputs:
        torch.cuda.synchronize()
        one_by_one.append(call(x).clone())
        torch.cuda.synchronize()
    for _ in range(3):
        outputs = [call(x) for x in inputs]
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(outputs, one_by_one))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        outputs = [call(x) for x in inputs]
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(outputs, one_by_one))


@pytest.mark.parametrize("heads", [2, 24])  # 24: more items than SMs
@pytest.mark.parametrize("one_stream_rows", [0, 10**9], ids=["two_streams", "one_stream"])
def test_layers_back_to_back_on_one_stream_and_on_two(native_lib, monkeypatch, heads, one_stream_rows):
    """Calls of their own take one stream or two by their length; here both, whatever it is."""
    from h3_optimizations_b200 import backend

    monkeypatch.setattr(backend, "ONE_STREAM_ROWS", one_stream_rows)
    call, inputs = _layer(heads)
    one_by_one = []
    for x in inputs:
        torch.cuda.synchronize()
        one_by_one.append(call(x).clone())
        torch.cuda.synchronize()
    assert not any(torch.equal(a, b) for a, b in zip(one_by_one, one_by_one[1:]))
    for _ in range(6):
        outputs = [call(x) for x in inputs]
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(outputs, one_by_one))
        del outputs  # the next calls get the same memory
