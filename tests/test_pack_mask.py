"""Filter words of boolean masks at the edges of the kernel that makes them: partial words, masks that do not begin on a
16-byte boundary, rows of masks, bytes other than 0 and 1."""

import numpy as np
import pytest
import torch

from libcertex_b200.index import pack_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 1000, 8192, 100_003])
@pytest.mark.parametrize("offset", [0, 1, 16])
def test_words_hold_the_mask(n, offset):
    rng = np.random.default_rng(n + offset)
    m = rng.random(n + offset) < 0.5
    words = pack_mask(torch.from_numpy(m).cuda()[offset:]).cpu().numpy().view(np.uint8)
    bits = np.unpackbits(words, bitorder="little")
    assert len(words) == 4 * ((n + 31) // 32)
    assert np.array_equal(bits[:n].astype(bool), m[offset:]) and not bits[n:].any()


def test_rows_and_other_bytes():
    rng = np.random.default_rng(0)
    m = rng.random((7, 45)) < 0.3
    words = pack_mask(torch.from_numpy(m)).cpu().numpy().view(np.uint8)
    assert np.array_equal(np.unpackbits(words, bitorder="little")[: 7 * 45].astype(bool), m.ravel())
    raw = rng.choice(np.array([0, 1, 2, 128, 255], dtype=np.uint8), 500)
    words = pack_mask(torch.from_numpy(raw).cuda().view(torch.bool)).cpu().numpy().view(np.uint8)
    assert np.array_equal(np.unpackbits(words, bitorder="little")[:500].astype(bool), raw != 0)
    assert pack_mask(torch.zeros(0, dtype=torch.bool)).numel() == 0
