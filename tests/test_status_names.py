"""What the status word of an attention launch says (CPU, from the sources): one code, one kind of wait, one text."""

import re
from pathlib import Path

from h3_optimizations_b200.backend import B200SparseBackend

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "h3_optimizations_b200" / "csrc"
# K and V have a ring each, filled and freed alike
SAME = {"k_full": "full", "v_full": "full", "kv_full": "full", "kv_empty": "empty"}


def _codes():
    body = re.search(r"enum AbortCode \{(.*?)\}", (CSRC / "attn_common.cuh").read_text(), re.S).group(1)
    return {name: number for number, name in enumerate(re.findall(r"kAbort\w+", body), start=1)}


def test_a_code_names_one_kind_of_wait():
    text = (CSRC / "attn_half.cu").read_text()
    waits = {}
    for barrier, code in re.findall(r"(?:warp_wait|mbar_wait)\(&(?:sh\.)?(\w+)[^;]*?(kAbort\w+)", text):
        waits.setdefault(code, set()).add(SAME.get(barrier, barrier))
    assert waits and all(len(barriers) == 1 for barriers in waits.values()), waits
    assert set(waits) <= set(_codes())


def test_every_code_has_its_text():
    assert sorted(_codes().values()) == sorted(B200SparseBackend.ABORT_NAMES)
    header = " ".join((ROOT / "include" / "h3sparse.h").read_text().replace("*", " ").split())
    for number, name in B200SparseBackend.ABORT_NAMES.items():
        assert "%d %s" % (number, name) in header, name
