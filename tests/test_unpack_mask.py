"""Verdict words as bools: the first n bits, and no more than the words hold."""
import numpy as np
import pytest

import golaypair_gb300 as gp


@pytest.mark.parametrize("words,n", [(0, 0), (1, 0), (1, 1), (1, 32), (2, 33), (3, 96), (1, 40), (0, 5), (2, -3)])
def test_unpack_mask(words, n):
    mask = np.random.default_rng(words).integers(0, 1 << 32, words, dtype=np.uint32)
    bits = [bool(int(w) >> k & 1) for w in mask for k in range(32)]
    got = gp.unpack_mask(mask, n)
    assert got.dtype == np.bool_ and got.tolist() == bits[:n]
