"""What the projector hands to the backend: carriers by address until somebody looks at them.  Needs a B200, but for the first test."""

import copy
import dataclasses
from types import SimpleNamespace

import pytest
import torch

from h3_optimizations_b200 import workloads
from h3_optimizations_b200.carriers import PreparedFusedQKV, PreparedLayer, ProjectedLayer, VCarrier, validate_prepared_fused_qkv

CARRIERS = ["q_int8", "k_int8", "q_scale", "k_scale", "v_scale", "v_carrier"]


def test_both_ends_share_the_pair_of_v():
    tensors = {"v_carrier": torch.ones((1, 2, 128, 128)).to(torch.float8_e4m3fn), "v_scale": torch.ones((1, 2, 128))}
    buffers = SimpleNamespace(heads=2, sequence=100, device=torch.device("cpu"), tensor=tensors.__getitem__, v_half=torch.ones(1))
    means = {"q_summary": torch.zeros((1, 2, 1, 128)), "k_summary": torch.zeros((1, 2, 2, 128))}
    projected = ProjectedLayer.over(buffers, head_dim=128, v=None, **means)
    prepared = PreparedLayer.over(buffers, route=None)
    assert projected.untouched() is buffers and prepared.untouched() is buffers and isinstance(projected, PreparedFusedQKV)
    half = VCarrier.of(prepared).half
    assert half is not None and VCarrier.of(projected).half is half
    projected.v_carrier  # whoever holds the codes may write to them: gone for both
    assert VCarrier.of(prepared).half is None and prepared.untouched() is None and projected.untouched() is None
    assert projected.v_scale is tensors["v_scale"]
    for other in ({"sequence": 101}, {"heads": 3}, {"head_dim": 64}, {"q_summary": means["k_summary"]}, {"v_scale": None}):
        again = ProjectedLayer.over(SimpleNamespace(**dict(vars(buffers), v_half=half, v_pair=None)), head_dim=128, v=None, **means)
        assert again.untouched() is not None
        for name, value in other.items():
            setattr(again, name, value)
        assert again.untouched() is None, other


@pytest.fixture()
def block(native_lib):
    from h3_optimizations_b200 import B200SparseBackend, ChunkedSparseQKVProjector, HybridSparseConfig, runtime_options

    spec = workloads.small_spec("block", 2, 192, 1300)
    x, w, w_scale = workloads.projection_inputs(spec.sequence, hidden=256, heads=2, seed=3)
    module = SimpleNamespace(heads=2, head_dim=128, qkv_weight_int8=w.cuda(), qkv_weight_scale=w_scale.cuda())
    x, options = x.cuda(), runtime_options(spec.layout(), step_index=5, total_steps=20)
    backend = B200SparseBackend(HybridSparseConfig(video_budget=0.4))
    project = lambda: ChunkedSparseQKVProjector().project(module, x, None, layer_index=1, transformer_options=options)
    finish = lambda projected: backend.execute(backend.prepare_projected(projected, layer_index=1, transformer_options=options))
    return project, finish


@pytest.mark.gpu
def test_looking_copying_and_replacing_change_nothing(block):
    project, finish = block
    projected = project()
    assert projected.untouched() is not None
    expected = finish(projected)
    assert projected.untouched() is not None and torch.equal(finish(projected), expected)  # and once more from the same carriers
    for names in ([name] for name in CARRIERS):
        projected = project()
        tensors = [getattr(projected, name) for name in names]
        assert all(t.is_cuda and t.is_contiguous() for t in tensors) and projected.untouched() is None
        assert torch.equal(finish(validate_prepared_fused_qkv(projected)), expected), names
    for other in (copy.copy(project()), copy.deepcopy(project()), dataclasses.replace(project(), layer_index=2)):
        assert torch.equal(finish(other), expected)
    assert type(copy.copy(project())) is PreparedFusedQKV


@pytest.mark.gpu
def test_what_is_written_or_put_in_their_place_counts(block):
    from h3_optimizations_b200 import SparseSageError

    project, finish = block
    expected = finish(project())
    projected = project()
    projected.v_scale.mul_(2)  # a power of two
    assert torch.equal(finish(projected).float(), expected.float() * 2)
    projected = project()
    projected.v_carrier.zero_()
    assert not finish(projected).any()
    projected = project()
    projected.v_carrier = torch.zeros_like(projected.v_carrier)
    assert not finish(projected).any()
    for name, value, text in (("sequence", 1, "Q/K carrier shape"), ("head_dim", 64, "head_dim 128"), ("v_scale", None, "requires V scale"),
                              ("q_summary", projected.k_summary, "Q router summary shape")):
        wrong = project()
        setattr(wrong, name, value)
        with pytest.raises(SparseSageError, match=text):
            finish(wrong)
