"""The heads that a call on host memory takes through at a time (CPU)."""

import pytest
import torch

from h3_optimizations_b200 import backend as module
from h3_optimizations_b200.backend import B200SparseBackend


@pytest.mark.parametrize("heads", [1, 2, 7, 8, 9, 24, 25])
@pytest.mark.parametrize("asked", [None, 1, 2, 3, 100])
def test_chunks_cover_the_heads_once(heads, asked):
    chunks = B200SparseBackend._head_chunks(heads, asked)
    assert [h for a, b in chunks for h in range(a, b)] == list(range(heads))
    sizes = [b - a for a, b in chunks]
    if asked is not None:
        assert sizes[:-1] == [min(asked, heads)] * (len(sizes) - 1)
    else:
        assert max(sizes) == (2 if heads >= 8 else 1) and sizes[-1] == 1


@pytest.mark.parametrize("heads", [1, 2, 7, 8, 9, 24, 25])
@pytest.mark.parametrize("asked", [None, 1, 3])
def test_short_heads_stay_in_pairs(heads, asked):
    chunks = B200SparseBackend._head_chunks(heads, asked, module.LONE_HEAD_BYTES - 1)
    assert [h for a, b in chunks for h in range(a, b)] == list(range(heads))
    size = min(heads, asked or (2 if heads >= 8 else 1))
    assert [b - a for a, b in chunks] == [size] * (heads // size) + [heads % size] * (heads % size > 0)


@pytest.mark.parametrize("size", [1, 512, 5000, 10**9])
@pytest.mark.parametrize("heads,sequence", [(1, 1), (1, 7), (2, 13), (3, 64)])
def test_the_output_arrives_whole(monkeypatch, heads, sequence, size):
    monkeypatch.setattr(module, "COPY_OUT_BYTES", size)
    slot = torch.randn((1, 3, sequence, 128)).bfloat16()
    out = torch.full((1, 5, sequence, 128), 77.0, dtype=torch.bfloat16)
    B200SparseBackend._copy_out(out[:, 1:1 + heads], slot[:, :heads])
    assert torch.equal(out[:, 1:1 + heads], slot[:, :heads])
    assert bool((out[:, :1] == 77.0).all()) and bool((out[:, 1 + heads:] == 77.0).all())
