"""What the status word of an attention launch says (CPU, from the sources): one code, one kind of wait, one text."""

import re
from pathlib import Path

import pytest

from h3_optimizations_b200.backend import B200SparseBackend
from h3_optimizations_b200.errors import SparseSageError

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


def test_the_words_name_the_kernel_that_waited():
    def text(*words):
        with pytest.raises(SparseSageError) as caught:
            B200SparseBackend._raise_for(words, "here")
        return str(caught.value)

    assert text(2, 7, 1, 3) == ("Sparse attention kernel gave up waiting for K/V tile load (code 2) in CTA 7, head 1, query tile 3 (here); "
                                "the output of that launch is invalid")
    assert text(15, 90, 2, 4) == ("Layer carrier kernel gave up waiting for whole-sequence statistics (code 15) in job 90, head 2, "
                                  "block 4 of 128 rows (here); the output of that launch is invalid")
    assert "an unknown event (code 19) in CTA 0, head 0, query tile 0" in text(19, 0, 0, 0)
