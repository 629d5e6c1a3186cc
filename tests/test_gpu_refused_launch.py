"""A launch that the runtime refuses.  Needs a B200.

More than 65535 heads do not fit a grid's second dimension: the runtime refuses the launch on the host and nothing runs.
The call raises, and its error is not left behind for the next one."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_the_error_is_not_taken_for_the_next_calls(native_lib):
    from h3_optimizations_b200 import _native, ops

    x = torch.ones((1, 65536, 1, 128), dtype=torch.bfloat16, device="cuda")
    lut = torch.empty((1, 1, 1, 2), dtype=torch.int32, device="cuda")
    valid = torch.empty((1, 1, 1), dtype=torch.int32, device="cuda")
    with pytest.raises(_native.NativeError, match="invalid"):
        ops.quant_qk_blocks(x, 64)
    # this one asks for the last error behind its launch
    _native.check(native_lib.h3s_route_to_delta_lut(None, 1, 1, 2, 0, 0, 0, lut.data_ptr(), valid.data_ptr(), _native.stream_ptr()),
                  "h3s_route_to_delta_lut")
    torch.cuda.synchronize()
    assert lut.flatten().tolist() == [0, 1] and valid.item() == 2
    codes, _, _ = ops.quant_qk_blocks(x[:, :3], 64)
    assert bool((codes == 127).all())
