"""The FP16 copy of the V codes never outlives the codes it was made from.  Needs a B200.

``v_carrier`` of prepared carriers is the caller's to read, replace or write to; the attention
call then uses what it holds."""

import dataclasses
from types import SimpleNamespace

import pytest
import torch

from h3_optimizations_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["prepare", "prepare_projected"])
def made(request, native_lib):
    """(backend, prepared, projected or None)"""
    from h3_optimizations_b200 import B200SparseBackend, ChunkedSparseQKVProjector, HybridSparseConfig, runtime_options

    heads, hidden = 2, 512
    spec = workloads.small_spec("copy", heads, 100, 900)
    options = runtime_options(spec.layout())
    backend = B200SparseBackend(HybridSparseConfig(video_budget=0.4))
    if request.param == "prepare":
        q, k, v = (t.cuda() for t in workloads.gaussian_qkv(spec, seed=3))
        return backend, backend.prepare(q, k, v, layer_index=0, transformer_options=options), None
    x, w, w_scale = workloads.projection_inputs(spec.sequence, hidden=hidden, heads=heads, seed=1)
    module = SimpleNamespace(heads=heads, head_dim=128, qkv_weight_int8=w.cuda(), qkv_weight_scale=w_scale.cuda())
    projected = ChunkedSparseQKVProjector().project(module, x.cuda(), None, layer_index=0, transformer_options=options)
    return backend, backend.prepare_projected(projected, layer_index=0, transformer_options=options), projected


def _with(prepared, codes):
    from h3_optimizations_b200 import ops

    s, geo = prepared.sparse, prepared.sparse.route.geometry
    return ops.sparse_attention(s.q_int8, s.k_int8, codes, s.q_scale, s.k_scale, s.v_scale, s.route.indices,
                                q_start=geo.pure_video_q_start, q_stop=geo.pure_video_q_stop, out_dtype=s.output_dtype)


def _other(codes):
    return (-codes.float()).to(torch.float8_e4m3fn)


@pytest.mark.parametrize("how", ["untouched", "read", "assigned", "written", "replaced", "written through the projection"])
def test_the_codes_are_what_counts(made, how):
    backend, prepared, projected = made
    sparse = prepared.sparse
    if how == "untouched":
        got = backend.execute(prepared)
        assert torch.equal(got, _with(prepared, sparse.v_carrier))
        return
    codes = sparse.v_carrier
    if how == "written through the projection":
        if projected is None:
            pytest.skip("no projection here")
        codes = projected.v_carrier
    want = _with(prepared, codes if how == "read" else _other(codes))
    if how == "assigned":
        sparse.v_carrier = _other(codes)
    elif how.startswith("written"):
        codes.copy_(_other(codes))
    elif how == "replaced":
        prepared = dataclasses.replace(prepared, sparse=dataclasses.replace(sparse, v_carrier=_other(codes)))
    assert torch.equal(backend.execute(prepared), want)


def test_written_through_the_projection_without_a_look_at_the_prepared_codes(made):
    backend, prepared, projected = made
    if projected is None:
        pytest.skip("no projection here")
    codes = projected.v_carrier
    codes.copy_(_other(codes))
    assert torch.equal(backend.execute(prepared), _with(prepared, codes))


def test_carriers_of_another_class_need_no_copy(made):
    """A projector's own record of the same fields, without ``v_half``."""
    backend, prepared, projected = made
    if projected is None:
        pytest.skip("no projection here")
    from h3_optimizations_b200 import runtime_options

    spec = workloads.small_spec("copy", 2, 100, 900)
    record = SimpleNamespace(**{f.name: getattr(projected, f.name) for f in dataclasses.fields(projected)})
    again = backend.prepare_projected(record, layer_index=0, transformer_options=runtime_options(spec.layout()))
    assert torch.equal(backend.execute(again), backend.execute(prepared))
