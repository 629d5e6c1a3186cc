"""The status words and their mirror as the host sees them (CPU, with tensors in place of the device's)."""

import pytest
import torch

from h3_optimizations_b200 import B200SparseBackend
from h3_optimizations_b200.errors import SparseSageError

NOTHING, GAVE_UP = [0, 0, 0, 0], [2, 5, 1, 3]
DEVICE = torch.device("cuda", 0)


@pytest.mark.parametrize("word", [NOTHING, GAVE_UP], ids=["word_clear", "word_set"])
@pytest.mark.parametrize("mirror", [NOTHING, GAVE_UP], ids=["mirror_clear", "mirror_set"])
def test_whatever_is_set_is_reported_once_and_cleared(word, mirror):
    backend = B200SparseBackend(check_device=False)
    slot = backend._status[0] = tuple(torch.tensor(words, dtype=torch.int32) for words in (word, mirror))
    if word[0] or mirror[0]:
        with pytest.raises(SparseSageError, match="K/V tile load.*CTA 5, head 1, query tile 3"):
            backend.check_status(DEVICE)
    backend.check_status(DEVICE)
    backend._poll_status(DEVICE)
    assert all(not words.any() for words in slot)
