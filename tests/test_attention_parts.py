"""Which dense rows the attention call cuts into parts (host arithmetic, no GPU): the workspace it asks for says so."""

import pytest


def _parts(native_lib, heads, sequence, context=0, density=1.0):
    q_tiles, kv_tiles = -(-sequence // 128), -(-sequence // 64)
    q_start = kv_start = route_len = 0
    if density < 1.0:
        q_start, kv_start = -(-context // 128), -(-context // 64)
        route_len = kv_start + max(1, int(-(-density * (kv_tiles - kv_start) // 1)))
    rows = heads * (q_start if density < 1.0 else q_tiles)
    size = native_lib.h3s_sparse_attn_half_workspace_bytes(heads, sequence, route_len, q_start, q_tiles if route_len else 0)
    return size // (rows * 128 * 130 * 4) or 1  # a part's sums; the counters are less than one


@pytest.mark.parametrize("heads,sequence", [(2, 9000), (2, 16000), (3, 8000), (3, 12000), (4, 2742), (4, 9000), (6, 1545), (6, 4000),
                                            (8, 3000), (12, 2000), (24, 9872)])
def test_rows_that_fill_the_processors_in_rounds_stay_whole(native_lib, heads, sequence):
    """In parts these took 1.1 to 1.8 times as long."""
    assert _parts(native_lib, heads, sequence) == 1


@pytest.mark.parametrize("heads,sequence,context,density", [(24, 5000, 300, 0.1), (24, 2362, 488, 0.2), (12, 4540, 545, 0.2),
                                                            (12, 10000, 600, 0.1), (8, 3205, 192, 0.5)])
def test_rows_that_end_with_the_routed_ones_stay_whole(native_lib, heads, sequence, context, density):
    assert _parts(native_lib, heads, sequence, context, density) == 1


@pytest.mark.parametrize("heads,sequence,context,density", [(1, 5000, 0, 1.0), (1, 20000, 0, 1.0), (1, 3137, 0, 1.0), (1, 33272, 512, 0.1),
                                                            (1, 33272, 512, 0.3), (3, 6404, 812, 0.1), (4, 7511, 193, 0.3)])
def test_rows_that_outlast_everything_else_are_cut(native_lib, heads, sequence, context, density):
    assert 2 <= _parts(native_lib, heads, sequence, context, density) <= 16


@pytest.mark.parametrize("heads,sequence,context,density", [(1, 2304, 256, 0.3), (4, 2304, 256, 0.3), (6, 4256, 512, 0.3), (3, 2103, 813, 0.3),
                                                            (7, 1594, 234, 0.15), (4, 29543, 451, 0.15), (4, 9000, 978, 0.3)])
def test_rows_whose_parts_cost_more_than_they_even_out_stay_whole(native_lib, heads, sequence, context, density):
    """With the cost of a part underestimated these were cut, and took up to 1.4 times as long."""
    assert _parts(native_lib, heads, sequence, context, density) == 1


@pytest.mark.parametrize("heads,sequence,context,density,parts", [(1, 12512, 512, 0.3, 6), (3, 6512, 512, 0.3, 2), (1, 5000, 512, 0.15, 5),
                                                                  (2, 15000, 512, 0.15, 3), (1, 33272, 512, 0.1, 5), (1, 9400, 0, 1.0, 2)])
def test_the_number_of_parts(native_lib, heads, sequence, context, density, parts):
    assert _parts(native_lib, heads, sequence, context, density) == parts
