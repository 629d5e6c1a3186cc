"""Accesses to tensor memory behind a wait, in the sources of the tcgen05 attention kernels (CPU).

A thread learns through an mbarrier that an MMA is complete; only ``tcgen05.fence::after_thread_sync``
orders its own loads and stores of tensor memory behind that.  No run on a GPU shows a missing one for certain,
so the text is checked: of the waits and fences above an access, the nearest one is a fence."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "h3_optimizations_b200" / "csrc"
ACCESS = re.compile(r"H3S_TMEM_(?:LD|ST)\d+\(")
EVENT = re.compile(r"(tc_fence_after\(\))|(?:warp_wait|mbar_wait|mbar_test_wait)\(&")


def _unordered(text):
    """Line numbers of accesses whose nearest event above is a wait."""
    text = re.sub(r"//[^\n]*", "", text)
    lines = []
    for access in ACCESS.finditer(text):
        events = list(EVENT.finditer(text, 0, access.start()))
        if not events or events[-1].group(1) is None:
            lines.append(text.count("\n", 0, access.start()) + 1)
    return lines


def test_the_check_sees_a_missing_fence():
    wait, fence, access = "if (!warp_wait(&sh.s_full, 0)) break;\n", "ptx::tc_fence_after();\n", "H3S_TMEM_LD32(t, r);\n"
    assert _unordered(wait + fence + access) == []
    assert _unordered(wait + access) == [2] and _unordered(fence + wait + access) == [3]


@pytest.mark.parametrize("name", ["attn_half.cu", "attn_tc.cu"])
def test_a_fence_stands_between_wait_and_access(name):
    assert _unordered((CSRC / name).read_text()) == []
