"""Norm weights of the projection in the types a model holds them in.  Needs a B200.

bf16 weights go to the kernel as they are; they are the same numbers in fp32, so every carrier is the same."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float16, torch.float16)])
@pytest.mark.parametrize("rows,heads,rope", [(130, 1, None), (500, 3, torch.bfloat16), (300, 2, torch.float32)])
def test_the_same_carriers(native_lib, rows, heads, rope, types):
    from h3_optimizations_b200.projector import run_chunked_sparse_qkv

    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn((rows, 256), generator=gen, device="cuda").bfloat16()
    w = torch.randint(-127, 128, (3 * heads * 128, 256), generator=gen, device="cuda", dtype=torch.int8)
    w_scale = torch.rand(3 * heads * 128, generator=gen, device="cuda") / 2000
    table = None if rope is None else torch.randn((1, rows, 1, 48, 2, 2), generator=gen, device="cuda").to(rope)
    # a view that begins at an odd element: the weights have no alignment but their own
    norms = [(torch.rand(129, generator=gen, device="cuda") + 0.5).to(t)[1:] for t in types]

    def carriers(q_norm, k_norm):
        p = run_chunked_sparse_qkv(x, w, w_scale, heads=heads, chunk_rows=128, norm=(q_norm, k_norm, 1e-6), rope_freqs=table, smooth_k=False)
        return [t.view(torch.uint8) for t in (p.q_int8, p.k_int8, p.q_scale, p.k_scale, p.q_summary, p.k_summary, p.v_scale, p.v_carrier)]

    expected = carriers(*[n.float() for n in norms])
    assert all(torch.equal(a, b) for a, b in zip(carriers(*norms), expected))
