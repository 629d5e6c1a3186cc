"""The heads that a call on host memory takes through at a time (CPU)."""

import pytest

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
