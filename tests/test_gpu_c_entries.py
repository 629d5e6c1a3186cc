"""C entry points that the package itself does not call: those with fewer arguments do what the longer ones do, and the
copy of the status words.  Needs a B200."""

import pytest
import torch

from h3_optimizations_b200 import workloads

pytestmark = pytest.mark.gpu


def test_attention_without_a_mirror(native_lib, monkeypatch):
    from h3_optimizations_b200 import ops

    spec = workloads.small_spec("entries", 2, 0, 500)
    q, k, v = (t.cuda() for t in workloads.gaussian_qkv(spec, seed=2))
    k_mean, v_scale = ops.column_stats(k, v)
    q8, qs, _ = ops.quant_qk_blocks(q, 128)
    k8, ks, _ = ops.quant_qk_blocks(k, 64, mean=k_mean)
    vc, _ = ops.quant_v_fp8(v, v_scale)
    expected = ops.sparse_attention(q8, k8, vc, qs, ks, v_scale)
    calls = []
    monkeypatch.setattr(native_lib, "h3s_sparse_attn_half_fwd_mirrored",
                        lambda *args: calls.append(1) or native_lib.h3s_sparse_attn_half_fwd(*args[:-2], args[-1]))
    assert torch.equal(ops.sparse_attention(q8, k8, vc, qs, ks, v_scale), expected) and calls


def test_projection_with_fp32_norms(native_lib, monkeypatch):
    from h3_optimizations_b200.projector import run_chunked_sparse_qkv

    gen = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn((300, 256), generator=gen, device="cuda").bfloat16()
    w = torch.randint(-127, 128, (3 * 2 * 128, 256), generator=gen, device="cuda", dtype=torch.int8)
    w_scale = torch.rand(3 * 2 * 128, generator=gen, device="cuda") / 2000
    norm = (*(torch.rand(128, generator=gen, device="cuda") + 0.5 for _ in range(2)), 1e-6)

    def carriers():
        p = run_chunked_sparse_qkv(x, w, w_scale, heads=2, chunk_rows=128, norm=norm)
        return [p.q_int8, p.k_int8, p.q_scale, p.k_scale, p.v_scale, p.q_summary, p.v_carrier.view(torch.uint8)]

    expected = carriers()
    calls = []
    monkeypatch.setattr(native_lib, "h3s_project_qkv_norms",
                        lambda *args: calls.append(1) or native_lib.h3s_project_qkv(*args[:16], *args[17:]))
    assert all(torch.equal(a, b) for a, b in zip(carriers(), expected)) and calls


def test_copy_of_the_status_words(native_lib):
    from h3_optimizations_b200 import _native

    word = torch.tensor([2, 5, 1, 3], dtype=torch.int32, device="cuda")
    mirror = torch.zeros(4, dtype=torch.int32).pin_memory()
    event = torch.cuda.Event()
    event.record()
    _native.check(native_lib.h3s_status_mirror(word.data_ptr(), mirror.data_ptr(), event.cuda_event, _native.stream_ptr()), "h3s_status_mirror")
    event.synchronize()
    assert mirror.tolist() == [2, 5, 1, 3]


@pytest.mark.parametrize("smooth_k", [True, False])
@pytest.mark.parametrize("v_after_k", [True, False])
def test_carriers_by_kernels_of_their_own_on_one_stream(native_lib, smooth_k, v_after_k):
    from h3_optimizations_b200 import _native, ops

    gen = torch.Generator(device="cuda").manual_seed(6)
    qkv = [torch.randn((1, 3, 1100, 128), generator=gen, device="cuda").bfloat16() for _ in range(3)]
    stream, second = _native.stream_ptr(qkv[0].device), ops.SideStream(qkv[0].device)
    results = []
    for side in (second, None):
        buffers = ops.LayerBuffers(3, 1100, qkv[0].device, smooth_k=smooth_k, summary_dtype=torch.float32)
        ops.quant_qkv(*qkv, buffers, side, stream, smooth_k=smooth_k, v_after_k=v_after_k)
        if side is not None:
            side.join(stream)
        names = ("q_int8", "k_int8", "v_carrier", "q_scale", "k_scale", "v_scale")
        results.append([buffers.tensor(name).view(torch.uint8) for name in names] + [buffers.v_half, buffers.q_summary, buffers.k_summary])
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("heads", [1, 5, 600])
def test_layer_carriers_with_counters_of_their_own(native_lib, heads):
    import ctypes

    from h3_optimizations_b200 import _native, ops

    gen = torch.Generator(device="cuda").manual_seed(heads)
    qkv = [torch.randn((1, heads, 150, 128), generator=gen, device="cuda").bfloat16() for _ in range(3)]
    strides = (ctypes.c_int64 * 6)(*(150 * 128, 128) * 3)
    guard = torch.full((heads + 9,), 7, dtype=torch.int32, device="cuda")
    results = []
    for own in (False, True):
        buffers = ops.LayerBuffers(heads, 150, qkv[0].device, smooth_k=True, summary_dtype=torch.float64)
        buffers._call.fill_(91)
        counters = guard.data_ptr() + 4 * 5 if own else buffers.native.scratch + buffers.counters_at
        _native.check(native_lib.h3s_prepare_layer(
            buffers.native, *(t.data_ptr() for t in qkv), strides, _native.H3S_BF16, heads, 150, 1, 448.0, counters, None, None,
            _native.stream_ptr(qkv[0].device)), "h3s_prepare_layer")
        names = ("q_int8", "k_int8", "v_carrier", "q_scale", "k_scale", "v_scale")
        results.append([buffers.tensor(name).view(torch.uint8) for name in names] + [buffers.v_half, buffers.q_summary, buffers.k_summary])
    assert all(torch.equal(a, b) for a, b in zip(*results))
    assert guard[:5].tolist() + guard[heads + 6:].tolist() == [7] * 8
    assert native_lib.h3s_prepare_layer_counter_bytes(heads) == 4 * (heads + 1)
    assert native_lib.h3s_prepare_layer(buffers.native, *(t.data_ptr() for t in qkv), strides, _native.H3S_BF16, heads, 150, 1, 448.0,
                                        counters + 2, None, None, None) == -1
