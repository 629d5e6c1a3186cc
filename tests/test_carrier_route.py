"""Which layers have their carriers made by one kernel (CPU)."""

import pytest
import torch

from h3_optimizations_b200 import backend


@pytest.mark.parametrize("heads,sequence,size,called,replayed", [
    (1, 64, 2, True, True), (4, 2304, 4, True, True), (4, 5000, 2, True, True), (1, 12000, 4, True, True),
    # V beside the router in a replay; the host's time decides in a call
    (4, 6000, 2, True, False), (24, 2304, 2, True, False), (3, 10500, 4, True, False), (16, 4500, 2, True, False),
    (4, 11912, 2, False, False), (4, 11912, 4, False, False), (7, 10384, 2, False, False), (6, 9000, 4, False, False),
    # the router fills the chip
    (24, 6112, 2, True, True), (24, 6112, 4, False, True), (12, 11912, 2, True, True), (24, 4374, 2, False, False), (24, 4375, 2, True, True),
    # long
    (4, 13512, 2, False, False), (24, 6251, 2, False, False), (24, 33272, 2, False, False)])
def test_route(monkeypatch, heads, sequence, size, called, replayed):
    for capturing, one in ((False, called), (True, replayed)):
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing)
        assert backend.one_carrier_kernel(heads, sequence, size) is one
