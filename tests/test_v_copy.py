"""What is asked of the FP16 copy of the V codes before anything is launched."""

import pytest
import torch

from h3_optimizations_b200 import PreparedFusedQKV, ops
from h3_optimizations_b200._native import NativeError
from h3_optimizations_b200.carriers import validate_prepared_fused_qkv
from h3_optimizations_b200.errors import FusedQKVError

SHAPE = (1, 2, 128, 256)
GOOD = torch.zeros(SHAPE, dtype=torch.float16)
BAD = {
    "type": torch.zeros(SHAPE, dtype=torch.bfloat16),
    "short": torch.zeros((1, 2, 128, 128), dtype=torch.float16),
    "heads": torch.zeros((1, 1, 128, 256), dtype=torch.float16),
    "strided": torch.zeros((1, 2, 256, 128), dtype=torch.float16).transpose(2, 3),
    "device": torch.zeros(SHAPE, dtype=torch.float16, device="meta"),
}


def _projected(v_half):
    sequence, heads = 200, 2
    rows = torch.zeros((1, heads, sequence, 128), dtype=torch.int8)
    return PreparedFusedQKV(
        q_int8=rows, k_int8=rows, q_scale=torch.zeros((1, heads, 2)), k_scale=torch.zeros((1, heads, 4)), v=None,
        q_summary=torch.zeros((1, heads, 2, 128)), k_summary=torch.zeros((1, heads, 4, 128)), output_dtype=torch.bfloat16,
        sequence=sequence, heads=heads, head_dim=128, layer_index=0,
        v_carrier=torch.zeros(SHAPE, dtype=torch.float8_e4m3fn), v_scale=torch.zeros((1, heads, 128)), v_half=v_half)


@pytest.mark.parametrize("good", [None, GOOD])
def test_a_fitting_copy_or_none_passes(good):
    validate_prepared_fused_qkv(_projected(good))
    if good is not None:
        ops.check_v_half(good, _projected(None).v_carrier)


@pytest.mark.parametrize("what", BAD)
def test_a_copy_that_does_not_fit_is_refused(what):
    with pytest.raises(FusedQKVError):
        validate_prepared_fused_qkv(_projected(BAD[what]))
    with pytest.raises(NativeError, match="v_half"):
        ops.check_v_half(BAD[what], torch.zeros(SHAPE, dtype=torch.float8_e4m3fn))


@pytest.mark.parametrize("carrier", [torch.zeros(SHAPE, dtype=torch.uint8), torch.zeros(SHAPE, dtype=torch.float8_e4m3fn)])
def test_the_copy_is_made_of_a_carrier_on_the_gpu(carrier):
    with pytest.raises(NativeError, match="carrier"):
        ops.v_half_copy(carrier)
