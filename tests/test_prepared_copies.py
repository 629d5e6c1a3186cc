"""Copies of a prepared layer keep the FP16 copy of V (CPU)."""

import copy
import io
from types import SimpleNamespace

import pytest
import torch

from h3_optimizations_b200.carriers import PreparedLayer, PreparedSparse, VCarrier


def _layer():
    tensors = {"q_int8": torch.ones((1, 2, 100, 128), dtype=torch.int8), "k_int8": torch.ones((1, 2, 100, 128), dtype=torch.int8),
               "v_carrier": torch.ones((1, 2, 128, 128)).to(torch.float8_e4m3fn), "q_scale": torch.ones((1, 2, 1)),
               "k_scale": torch.ones((1, 2, 2)), "v_scale": torch.ones((1, 2, 128))}
    buffers = SimpleNamespace(heads=2, sequence=100, device=torch.device("cpu"), tensor=tensors.__getitem__,
                              v_half=torch.ones((1, 2, 128, 128), dtype=torch.float16))
    return PreparedLayer.over(buffers, route=None, output_dtype=torch.bfloat16, output_shape=(1, 2, 100, 128), layer_index=4,
                              metadata={"layer": 4}), buffers


@pytest.mark.parametrize("looked_at", [(), ("q_int8",), ("k_scale", "v_scale")])
def test_a_shallow_copy_shares_it(looked_at):
    layer, buffers = _layer()
    for name in looked_at:
        getattr(layer, name)
    half = buffers.v_half
    twin = copy.copy(layer)
    assert type(twin) is PreparedSparse and twin.layer_index == 4 and twin.metadata is layer.metadata and twin.q_int8 is layer.q_int8
    assert VCarrier.of(layer) is VCarrier.of(twin) and VCarrier.of(twin).half is half
    twin.v_carrier  # whoever holds the codes may write to them: gone for both
    assert VCarrier.of(layer).half is None and layer.untouched() is None


def _saved(layer):
    file = io.BytesIO()
    torch.save(layer, file)
    file.seek(0)
    return torch.load(file, weights_only=False)


@pytest.mark.parametrize("copied", [copy.deepcopy, _saved])
def test_a_copy_of_its_own_has_its_own(copied):
    layer, buffers = _layer()
    half = buffers.v_half
    twin = copied(layer)
    mine = VCarrier.of(twin).half
    assert type(twin) is PreparedSparse and mine is not half and torch.equal(mine, half)
    twin.v_carrier.zero_()
    assert VCarrier.of(layer).half is half and bool((VCarrier.of(layer).codes.float() == 1).all())
    assert twin.sequence == 100 and twin.heads == 2 and torch.equal(twin.k_scale, layer.k_scale)
