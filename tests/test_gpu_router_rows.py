"""Router with sixteen and with eight query tiles a CTA, at the edges of its blocks.  Needs a B200.

Summaries of small integers: every score is exact in any order of the additions, and there are many ties, of
which the lower indices win."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,rows,tiles", [
    (300, 1, 3), (150, 17, 64), (150, 16, 65), (20, 121, 130),  # sixteen rows
    (2, 15, 63), (1, 17, 129),                                  # too few for sixteen
    (30, 90, 1232), (30, 90, 1233),                             # the last that fits, the first that does not
])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_selection_is_exact(native_lib, heads, rows, tiles, dtype):
    from h3_optimizations_b200 import ops

    gen = torch.Generator().manual_seed(rows + tiles)
    q = torch.randint(-3, 4, (1, heads, rows + 2, 128), generator=gen).to(dtype)
    k = torch.randint(-3, 4, (1, heads, tiles + 3, 128), generator=gen).to(dtype)
    retained = max(1, tiles * 3 // 10)
    got = ops.route_topk(q.cuda(), k.cuda(), q_start=1, q_stop=rows + 1, kv_start=2, kv_stop=tiles + 2, retained=retained).cpu()
    scores = (q[0, :, 1:rows + 1].float() @ k[0, :, 2:tiles + 2].float().transpose(1, 2)).to(torch.int32)
    order = scores.sort(dim=-1, descending=True, stable=True).indices[..., :retained] + 2
    want = torch.cat([torch.tensor([0, 1, tiles + 2]).expand(heads, rows, 3), order], dim=-1).sort(dim=-1).values
    assert torch.equal(got[0].long(), want)
