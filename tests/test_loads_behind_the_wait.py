"""Kernels that start before the one in front of them has ended read global memory only behind their wait (CPU, from the sources).

`__ldg`, `ld.global.nc` and loads through `const __restrict__` parameters may be moved up by the compiler, so straight-line code behind
`wait_for_previous` uses none of them; what is left stands in the roles of a kernel, behind barriers and loops."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "h3_optimizations_b200" / "csrc"
FILES = ("common.cuh", "quant.cu", "router.cu", "attn_half.cu")


def _code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def test_row_kernels_router_and_attention_have_none():
    for name in FILES:
        code = _code(name)
        assert "__ldg" not in code and "ld.global.nc" not in code, name


def test_what_a_kernel_is_handed_is_not_read_directly():
    """Inputs of the kernels that are read element by element go through one of the two ways."""
    quant = _code("quant.cu")
    for name in ("k_sum", "v_amax_bits", "mean", "v_scale"):
        body = re.sub(r"load_written\([^;]*", "", quant)
        assert not re.search(r"=\s*%s\[|\(\s*%s\[" % (name, name), body), name
    router = _code("router.cu")
    assert "q_summary = written_before(q_summary);" in router and "k_summary = written_before(k_summary);" in router
    assert not re.search(r"__restrict__ [qk]_summary", router)


def test_the_projection_reads_scales_and_norm_weights_so():
    gemm = _code("qkv_gemm.cu")
    kernel = gemm[gemm.index("wait_for_previous();", gemm.index("qkv_gemm_kernel(const")):]
    assert "__ldg" not in kernel[:kernel.index("if (warp == W::kLoad)")]
    assert "__ldg(prm.x_scale" not in gemm and "__ldg" not in gemm[gemm.index("float rope_load"):gemm.index("bf16_lo(uint32_t")]
