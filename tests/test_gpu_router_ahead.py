"""The router's CTAs of eight rows with and without a block of means ahead.  Needs a B200.

One CTA an SM has the next block's loads in flight, several have not: sizes around that line, blocks of 64 tiles with all kinds of
ends, rows that do not fill a CTA.  Scores are sums of random products, so there are no ties, and the selection is
that of 64-bit matrix products."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,rows,tiles,q_start,kv_start,after", [
    (1, 1, 1, 0, 0, 0), (1, 9, 63, 1, 2, 1), (2, 8, 64, 0, 0, 0), (3, 17, 65, 2, 1, 0), (4, 40, 128, 0, 3, 2), (5, 61, 129, 1, 0, 0),
    (148, 8, 70, 0, 1, 0), (149, 8, 70, 0, 1, 0), (37, 25, 191, 0, 0, 3), (37, 33, 193, 1, 1, 0), (1, 591, 1181, 1, 8, 0)])
def test_selection(native_lib, heads, rows, tiles, q_start, kv_start, after, dtype):
    from h3_optimizations_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(rows * tiles)
    q = torch.randn((1, heads, q_start + rows, 128), generator=gen, device="cuda").to(dtype)
    k = torch.randn((1, heads, kv_start + tiles + after, 128), generator=gen, device="cuda").to(dtype)
    retained = max(1, tiles * 3 // 10)
    route = ops.route_topk(q, k, q_start=q_start, q_stop=q_start + rows, kv_start=kv_start, kv_stop=kv_start + tiles, retained=retained)
    scores = q[0, :, q_start:].double() @ k[0, :, kv_start:kv_start + tiles].double().transpose(1, 2)
    chosen = scores.topk(retained, dim=-1).indices.sort(dim=-1).values + kv_start
    around = [torch.arange(kv_start, device="cuda"), kv_start + tiles + torch.arange(after, device="cuda")]
    before, behind = (a.expand(heads, rows, -1) for a in around)
    assert torch.equal(route[0].long(), torch.cat([before, chosen, behind], dim=-1))
