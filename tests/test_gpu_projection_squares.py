"""The sum of squares of the RMS norm in the carrier epilogue, to its last bit.  Needs a B200.

An FP32 sum that is off by a unit in the last place, and the reciprocal square root with it, hardly ever shows behind the
rounding to bf16.  Here it does: the norm's weights put every channel's product halfway between two bf16 values
if the reciprocal were off by half a unit, the even channels on one side, the odd ones on the other.  The
rows marked NEAR_TIES have totals within 2^-42 of themselves of the middle between two floats, which sums of fewer
bits take for the other side; the others have sizes as rows have them."""

import numpy as np
import pytest
import torch

from oracle import h3_oracle as oracle

pytestmark = pytest.mark.gpu

# per row: two hex digits a channel, (|m| - 129) / 2 and 64 for a minus sign; a letter a channel, -exponent
NEAR_TIES = [
    ("61765d2f53350f2456645121116f4e15001f405e362a610d77010c05160b4936226d612f301c75463c1d09776a601168331709493268505f4a5673107d6c0354"
     "13243f504b7027176c1e783b146d602f575541752158623f7539186a61756e221e2e2007037f10334709014f3e6400707b49637d1556273f7b70121f4b17262d",
     "ahnlmgjgmfhijdhelhggjkkdlggejkndjmniimeljfjngjflhelnikhedgdgddlnngkfefjggnnnifehdllnmifnefmkgfemnilmjfihhlgdngjkmejjddmkkdnnefpq"),
    ("43474d410e09517e0f2624322c6518285d56732a6e1103621a614222264734207511714111306247623c4620195715026800426b6e6c351634764c5232615d49"
     "5e566a2e725b221160206e353d6508112f79420711301b1c36210b103f5056095262106e504026125e1f0e7e6c205d2327627f0a2f616b4a4072463120311a3f",
     "ajlmmjemghhggijjlldggmddiijiielmedkehjimlfnnhffgemenfmkghjjdkmididdkendengnggmfnmkgedngfkllkdheelhghdfngeekkidldjgnnhjnfdlkimkmq"),
]


def _near_tie(text, letters):
    code = [int(text[i:i + 2], 16) for i in range(0, 256, 2)]
    return [(2 * (c & 63) + 129) * (-1 if c & 64 else 1) for c in code], [97 - ord(c) for c in letters]


def _drawn(kind, seed):
    rng = np.random.default_rng(seed)
    m = rng.integers(64, 128, 128) * 2 + 1
    e = {"flat": np.zeros(128), "outlier": np.where(np.arange(128) == seed, 8, 0), "wide": rng.integers(-30, 1, 128),
         "small": np.full(128, -50), "tiny": np.full(128, -70), "tiny beside small": np.where(np.arange(128) % 48 < 24, -70, -40)}[kind]
    return (m * rng.choice([-1, 1], 128)).tolist(), e.astype(int).tolist()


def _weights(row, inverse):
    """Weights whose products with ``row * inverse`` change their bf16 value half an FP32 unit of ``inverse`` further up
    (even channels) or down (odd channels)."""
    step = np.where(np.arange(128) % 2 == 0, np.nextafter(inverse, np.float32(np.inf)), np.nextafter(inverse, np.float32(0)))
    here, there = (row * inverse).astype(np.float64), (row * step.astype(np.float32)).astype(np.float64)
    return ((1 + 2.0 ** -8) / np.abs((here + there) / 2)).astype(np.float32)


def _normed(native_lib, m, exponent):
    """The kernel's normed row of one token, and the oracle's."""
    from h3_optimizations_b200 import ops

    row = (np.array(m) * 2.0 ** np.array(exponent)).astype(np.float32)
    total = np.float32((row.astype(np.longdouble) ** 2).sum())
    inverse = np.float32(1.0 / np.sqrt(np.float64(total * np.float32(1 / 128))))
    weight = torch.from_numpy(_weights(row, inverse))
    x = torch.zeros((1, 128), dtype=torch.int8)
    x[0, :3] = 1
    w = torch.zeros((384, 128), dtype=torch.int8)
    for part in range(3):  # |m| <= 255 as three weights
        left = torch.tensor(m).repeat(2) - w.sum(1, dtype=torch.int32)[:256]
        w[:256, part] = left.clamp(-127, 127).to(torch.int8)
    w_scale = torch.ones(384)
    w_scale[:256] = (2.0 ** torch.tensor(exponent, dtype=torch.float64)).float().repeat(2)
    empty = lambda *shape, dtype=torch.float32: torch.empty(shape, dtype=dtype, device="cuda")
    q_mean, k_mean = empty(1, 1, 1, 128), empty(1, 1, 1, 128)
    ops.qkv_gemm_chunk_carriers(
        x.cuda(), torch.ones(1).cuda(), w.cuda(), w_scale.cuda(), heads=1, row_start=0, q_int8=empty(1, 1, 1, 128, dtype=torch.int8),
        q_scale=empty(1, 1, 1), q_summary=q_mean, k_summary=k_mean, v_stage=empty(1, 1, 1, 128, dtype=torch.bfloat16),
        stats=ops.column_stats_scratch(1, "cuda"), k_stage=empty(1, 1, 1, 128, dtype=torch.bfloat16), q_norm=weight.cuda(),
        k_norm=weight.cuda(), epsilon=0.0)
    y = torch.cat([torch.from_numpy(row), torch.from_numpy(row), torch.zeros(128)])[None]
    want = oracle.rms_norm_rope_split_half(y, 1, weight, weight, 0.0)[0, :128].float()
    return want, q_mean.cpu().flatten(), k_mean.cpu().flatten()  # the mean of one row is the row


@pytest.mark.parametrize("text,letters", NEAR_TIES)
def test_totals_close_to_the_middle_between_two_floats(native_lib, text, letters):
    want, q, k = _normed(native_lib, *_near_tie(text, letters))
    assert torch.equal(q, want) and torch.equal(k, want)


@pytest.mark.parametrize("kind", ["flat", "outlier", "wide", "small", "tiny", "tiny beside small"])
def test_rows_of_all_shapes(native_lib, kind):
    for seed in range(8):
        want, q, k = _normed(native_lib, *_drawn(kind, seed))
        assert torch.equal(q, want) and torch.equal(k, want), seed
