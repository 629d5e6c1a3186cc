"""Where the attention kernel's output tiles go.  Needs a B200.

Without further outputs every warp stores its rows through a tensor map of the output; with one, the
tile is staged as a whole and written as lines.  Both write the same bits, for every order and stride of the output
that the call takes, and leave alone what lies between its rows."""

import pytest
import torch

from h3_optimizations_b200 import workloads

pytestmark = pytest.mark.gpu

LAYOUTS = {  # (heads, sequence) -> elements, head stride, row stride
    "token_major": lambda h, s: (s * h * 128, 128, h * 128),
    "head_major": lambda h, s: (h * s * 128, s * 128, 128),
    "padded_rows": lambda h, s: (h * s * 144, s * 144, 144),
    "padded_heads": lambda h, s: (s * h * 152, 152, h * 152),
    "one_heads_stride_is_free": lambda h, s: (s * 136 + h * 8, 8, 136),
}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("layout", list(LAYOUTS))
@pytest.mark.parametrize("sequence", [1, 33, 97, 160, 700])
def test_stores_are_the_same(native_lib, layout, sequence, dtype):
    from h3_optimizations_b200 import ops

    heads = 1 if layout == "one_heads_stride_is_free" else 3
    spec = workloads.small_spec("output", heads, 0, sequence)
    q, k, v = (t.cuda() for t in workloads.gaussian_qkv(spec, seed=sequence))
    k_mean, v_scale = ops.column_stats(k, v)
    q8, qs, _ = ops.quant_qk_blocks(q, 128)
    k8, ks, _ = ops.quant_qk_blocks(k, 64, mean=k_mean)
    vc, _ = ops.quant_v_fp8(v, v_scale)
    elements, stride_h, stride_s = LAYOUTS[layout](heads, sequence)
    whole = [torch.full((elements,), 77.0, dtype=dtype, device="cuda") for _ in range(3)]
    out, staged, further = (w.as_strided((1, heads, sequence, 128), (elements, stride_h, stride_s, 1)) for w in whole)
    ops.sparse_attention(q8, k8, vc, qs, ks, v_scale, out=out)
    ops.sparse_attention(q8, k8, vc, qs, ks, v_scale, out=staged, peer_out_ptrs=[further.data_ptr()])
    torch.cuda.synchronize()
    assert torch.isfinite(out).all() and not (out == 77.0).all(dim=-1).any()
    assert torch.equal(whole[0], whole[1]) and torch.equal(whole[0], whole[2])


def test_an_output_in_pinned_host_memory(native_lib):
    from h3_optimizations_b200 import ops

    spec = workloads.small_spec("output", 2, 0, 200)
    q, k, v = (t.cuda() for t in workloads.gaussian_qkv(spec, seed=7))
    k_mean, v_scale = ops.column_stats(k, v)
    q8, qs, _ = ops.quant_qk_blocks(q, 128)
    k8, ks, _ = ops.quant_qk_blocks(k, 64, mean=k_mean)
    vc, _ = ops.quant_v_fp8(v, v_scale)
    host = torch.zeros((1, 2, 200, 128), dtype=torch.bfloat16).pin_memory()
    ops.sparse_attention(q8, k8, vc, qs, ks, v_scale, out=host)
    out = ops.sparse_attention(q8, k8, vc, qs, ks, v_scale)
    torch.cuda.synchronize()
    assert torch.equal(host, out.cpu())
