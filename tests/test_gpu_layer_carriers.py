"""The carriers of a layer from one kernel against the kernels of their own, bit for bit.  Needs a B200."""

import pytest
import torch

from oracle import h3_oracle as oracle

pytestmark = pytest.mark.gpu

CARRIERS = ("q_int8", "k_int8", "v_carrier", "q_scale", "k_scale", "v_scale")


# one row; a K block and its first row more; a last step without a second K block; as many statistics jobs as fit one wave and more; heads of
# one short block each
@pytest.mark.parametrize("heads,sequence,dtype", [
    (2, 1, torch.bfloat16), (3, 64, torch.float32), (1, 65, torch.float16), (2, 129, torch.bfloat16), (5, 1100, torch.float32),
    (4, 2304, torch.bfloat16), (7, 10384, torch.float16), (3, 33272, torch.bfloat16), (200, 70, torch.bfloat16)])
@pytest.mark.parametrize("token_major", [False, True])
@pytest.mark.parametrize("smooth_k,means", [(True, True), (False, True), (True, False)])
def test_one_kernel_gives_what_the_others_give(native_lib, heads, sequence, dtype, token_major, smooth_k, means):
    from h3_optimizations_b200 import _native, ops

    gen = torch.Generator(device="cuda").manual_seed(heads * sequence)
    qkv = []
    for offset in (0.0, 0.7, -0.2):
        x = (torch.randn((1, heads, sequence, 128), generator=gen, device="cuda") + offset).to(dtype)
        qkv.append(x.transpose(1, 2).contiguous().transpose(1, 2) if token_major else x)
    device = qkv[0].device
    stream, side = _native.stream_ptr(device), ops.SideStream(device)
    word, mirror = torch.zeros(4, dtype=torch.int32, device="cuda"), torch.zeros(4, dtype=torch.int32).pin_memory()
    results = []
    for one in (False, True, True):
        buffers = ops.LayerBuffers(heads, sequence, device, smooth_k=smooth_k, summary_dtype=torch.float64 if means else None)
        buffers._carriers.fill_(77)
        buffers.v_half.fill_(3.0)
        buffers._call.fill_(91)  # scratch and counters come as they are
        if one:
            ops.prepare_layer(*qkv, buffers, stream, smooth_k=smooth_k, status=word, status_mirror=mirror)
        else:
            ops.quant_qkv(*qkv, buffers, side, stream, smooth_k=smooth_k, v_after_k=True)
            side.join(stream)
        torch.cuda.synchronize()
        tensors = [buffers.tensor(name) for name in CARRIERS] + [buffers.v_half]
        results.append([t.view(torch.uint8).clone() for t in tensors + ([buffers.q_summary, buffers.k_summary] if means else [])])
    assert word.tolist() == mirror.tolist() == [0, 0, 0, 0]
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))


def test_what_the_kernel_cannot_take_is_refused(native_lib):
    from h3_optimizations_b200 import _native, ops

    q, k, v = (torch.zeros((1, 2, 128, 136), device="cuda", dtype=torch.bfloat16)[..., :128] for _ in range(3))
    buffers = ops.LayerBuffers(2, 128, q.device, smooth_k=True, summary_dtype=None)
    word, mirror = torch.zeros(4, dtype=torch.int32, device="cuda"), torch.zeros(4, dtype=torch.int32).pin_memory()
    call = lambda *qkv: ops.prepare_layer(*qkv, buffers, _native.stream_ptr(q.device), smooth_k=True, status=word, status_mirror=mirror)
    call(q, k, v)
    odd = torch.zeros((2 * 128 * 132 + 4,), device="cuda", dtype=torch.bfloat16)
    with pytest.raises(_native.NativeError, match="multiples of 8"):
        call(q, odd[: 2 * 128 * 132].view(1, 2, 128, 132)[..., :128], v)
    with pytest.raises(_native.NativeError, match="aligned"):
        call(q, k, odd[4:].view(-1)[: 2 * 128 * 128].view(1, 2, 128, 128))


def _one_zero(codes):
    """E4M3 codes with -0, which the quantiser writes as 0, as 0."""
    return torch.where(codes == 0x80, torch.zeros_like(codes), codes)


UNUSUAL = ["zeros", "zero column", "equal rows", "tiny", "huge", "steps", "infinity", "NaN"]


@pytest.mark.parametrize("how", UNUSUAL)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("one", [True, False])
@pytest.mark.parametrize("heads,sequence", [(2, 300), (1, 1)])
def test_unusual_values_against_the_oracle(native_lib, heads, sequence, one, dtype, how):
    """K mean, codes, scales and tile means by plain torch.  A NaN counts as nothing where a maximum is taken; codes of it are 0 in
    Q and K and NaN in V, as are those of an infinity by an infinite scale."""
    from h3_optimizations_b200 import _native, ops

    gen = torch.Generator().manual_seed(sequence)
    q, k, v = ((torch.randn((1, heads, sequence, 128), generator=gen) + offset).to(dtype) for offset in (0.0, 0.7, -0.2))
    row = sequence // 2
    for x in (q, k, v):
        if how == "zeros":
            x.zero_()
        elif how == "zero column":
            x[:, 0, :, 9] = 0.0
            x[:, -1, :, 70] = -0.0
        elif how == "equal rows":
            x[:] = x[:, :, :1].clone()
        elif how == "tiny":
            x *= 2.0 ** -125
        elif how == "huge":
            x *= 2.0 ** 120
        elif how == "steps":
            x[:, :, ::7] *= 2.0 ** 20
    plain = [x.clone() for x in (q, k, v)]
    bad = {"infinity": float("inf"), "NaN": float("nan")}.get(how)
    if bad is not None:  # not in K, whose mean would be so
        q[0, 0, row, 3] = v[0, 0, row, 5] = bad
    device = torch.device("cuda", torch.cuda.current_device())
    stream, side = _native.stream_ptr(device), ops.SideStream(device)
    word, mirror = torch.zeros(4, dtype=torch.int32, device="cuda"), torch.zeros(4, dtype=torch.int32).pin_memory()
    buffers = ops.LayerBuffers(heads, sequence, device, smooth_k=True, summary_dtype=torch.float64)
    inputs = [x.cuda() for x in (q, k, v)]
    if one:
        ops.prepare_layer(*inputs, buffers, stream, smooth_k=True, status=word, status_mirror=mirror)
    else:
        ops.quant_qkv(*inputs, buffers, side, stream, smooth_k=True, v_after_k=True)
        side.join(stream)
    got = {name: buffers.tensor(name).cpu() for name in CARRIERS}
    q_means, k_means = buffers.q_summary.cpu(), buffers.k_summary.cpu()

    mean = k.double().mean(dim=2).to(torch.float32).to(dtype).float()
    k_codes, k_scale = oracle.quantize_blocks(k, 64, mean=mean)
    assert torch.equal(got["k_int8"], k_codes) and torch.equal(got["k_scale"], k_scale)
    q_codes, q_scale = oracle.quantize_blocks(plain[0], 128)
    v_codes, v_scale = oracle.v_fp8_carrier(plain[2])
    v_codes = v_codes.view(torch.uint8)
    if how == "infinity":
        block = slice(row // 128 * 128, row // 128 * 128 + 128)
        q_codes[0, 0, block], q_scale[0, 0, row // 128] = 0, bad
        v_codes[0, 0, 5, :sequence] = 0
        v_scale[0, 0, 5] = bad
    if how == "NaN":
        for x, tile in ((plain[0], 128), (plain[2], None)):
            x[0, 0, row, 3 if tile else 5] = 0.0  # counts as nothing
        q_codes, q_scale = oracle.quantize_blocks(plain[0], 128)
        v_codes, v_scale = oracle.v_fp8_carrier(plain[2])
        v_codes = v_codes.view(torch.uint8)
    if bad is not None:
        assert got["v_carrier"].view(torch.uint8)[0, 0, 5, row] & 0x7F == 0x7F  # NaN
        v_codes[0, 0, 5, row] = got["v_carrier"].view(torch.uint8)[0, 0, 5, row]
    assert torch.equal(got["q_int8"], q_codes) and torch.equal(got["q_scale"], q_scale)
    assert torch.equal(_one_zero(got["v_carrier"].view(torch.uint8)), _one_zero(v_codes)) and torch.equal(got["v_scale"], v_scale)
    half = buffers.v_half.cpu()
    want_half = got["v_carrier"].to(torch.float16)
    assert torch.equal(torch.isnan(half), torch.isnan(want_half)) and torch.equal(half.nan_to_num(0.0), want_half.nan_to_num(0.0))
    for x, means, tile in ((q, q_means, 128), (k, k_means, 64)):
        want = oracle.mean_pool(x.double(), tile)
        largest = oracle.mean_pool(x.double().abs(), tile)
        fine = torch.isfinite(want)
        # up to eight rows are added up in fp32
        assert bool(((means - want).abs()[fine] <= 8 * 2.0 ** -24 * largest[fine]).all()) and not bool(torch.isfinite(means[~fine]).any())
    assert word.tolist() == [0, 0, 0, 0]


# fewer jobs than blocks, and more than twice as many
@pytest.mark.parametrize("heads,sequence,dtype", [(2, 200, torch.bfloat16), (1, 1, torch.float32), (24, 2304, torch.bfloat16), (9, 5000, torch.float32)])
@pytest.mark.parametrize("smooth_k", [True, False])
def test_statistics_that_do_not_come_are_given_up(native_lib, heads, sequence, dtype, smooth_k):
    """The wait expects a statistics job that nobody does, with a limit of 1 ms: the launch says so and ends, every block with one wait,
    all jobs are done (the statistics are there by then, so with the right result), and the next launch is as ever."""
    from h3_optimizations_b200 import _native, ops

    gen = torch.Generator(device="cuda").manual_seed(heads)
    qkv = [torch.randn((1, heads, sequence, 128), generator=gen, device="cuda").to(dtype) for _ in range(3)]
    device = qkv[0].device
    word, mirror = torch.zeros(4, dtype=torch.int32, device="cuda"), torch.zeros(4, dtype=torch.int32).pin_memory()
    start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def carriers(flags):
        buffers = ops.LayerBuffers(heads, sequence, device, smooth_k=smooth_k, summary_dtype=torch.float64)
        buffers._carriers.fill_(77)
        buffers.v_half.fill_(3.0)
        buffers._call.fill_(91)
        torch.cuda.synchronize()
        start.record()
        ops.prepare_layer(*qkv, buffers, _native.stream_ptr(device), smooth_k=smooth_k, status=word, status_mirror=mirror, extra_flags=flags)
        stop.record()
        torch.cuda.synchronize()  # returns: the kernel ended by itself
        return [t.view(torch.uint8).clone() for t in [buffers.tensor(name) for name in CARRIERS] + [buffers.v_half, buffers.q_summary, buffers.k_summary]]

    good = carriers(0)
    assert word.tolist() == mirror.tolist() == [0, 0, 0, 0]
    previous = ops.set_wait_budget_ns(1_000_000)
    try:
        late = carriers(ops.PREPARE_TEST_MISSING_STATISTICS)
    finally:
        ops.set_wait_budget_ns(previous)
    assert 0.9 < start.elapsed_time(stop) < 50.0
    code, job, head, step = word.tolist()
    assert code == 15 and mirror.tolist() == [code, job, head, step]
    steps = -(-sequence // 128)
    job -= _early_jobs(heads, sequence, smooth_k)
    assert 0 <= job < heads * 2 * steps and (head, step) == (job // (2 * steps), job % steps)
    assert all(torch.equal(a, b) for a, b in zip(good, late))
    word.zero_()
    mirror.zero_()
    assert all(torch.equal(a, b) for a, b in zip(good, carriers(0)))
    assert word.tolist() == mirror.tolist() == [0, 0, 0, 0]


def _early_jobs(heads, sequence, smooth_k):
    """Jobs that wait for nothing: statistics, of as many rows a job as leave 380 of them where there are so many, and Q blocks."""
    rows = 1024
    while rows > 64 and heads * -(-sequence // rows) * (2 if smooth_k else 1) < 380:
        rows //= 2
    return heads * (-(-sequence // rows) * (2 if smooth_k else 1) + -(-sequence // 128))
