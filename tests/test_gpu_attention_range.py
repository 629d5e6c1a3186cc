"""Finite inputs give finite outputs, whatever the scale of V.  Needs a B200.

Row sums may reach 2^16 a tile, the accumulators 448 times that: dequantising them before the
division would overflow where a row runs ahead of its reference tiles and V is large.  Oracle and
bound are those of test_gpu_attention_tiles."""

import pytest
import torch

from h3_optimizations_b200 import workloads
from oracle import h3_oracle as oracle

from .test_gpu_attention_tiles import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sequence", [187, 1601])  # whole lists; lists cut into two parts
def test_a_large_v_in_rows_that_run_ahead(native_lib, sequence):
    spec = workloads.small_spec("range", 2, 0, sequence)
    q, k, v = workloads.gaussian_qkv(spec, seed=sequence, widen=True)
    sign = -torch.ones(sequence)
    sign[:64] = 1.0
    q, k, v = q + 0.75, k + 0.75 * sign[:, None], v * 2.0 ** 114                   # about 18 bits ahead, V up to 2^116
    _check(native_lib, q, k, v, oracle.geometry(sequence, 0), None)
