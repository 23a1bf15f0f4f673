"""The enumerator's blocks: alphabets of 2 to 9 values, lengths below and above
the one from which a block has all its digits, 64- and 128-bit words, windows
that begin and end inside blocks.  Bar: the oracle's files and necklace count."""
import pytest

import golaypair_gb300 as gp
from conftest import GenStats

import ctypes

pytestmark = pytest.mark.gpu

WHOLE = [(8, 2), (10, 1), (18, 3), (20, 4), (40, 8), (26, 1), (34, 2), (2, 1), (4, 1), (4, 2)]
PARTS = [(26, 1), (34, 2), (45, 3), (40, 5), (80, 2), (68, 1), (90, 3)]


def _windows():
    for order, compress in WHOLE:
        yield order, compress, 0, (compress + 1) ** (order // compress)
    for order, compress in PARTS:
        k, L = compress + 1, order // compress
        for lo, size in ((0, 1), (1, 62), (63, 2), (k ** 3 - 1, 5003), (k ** (L - 4) // 3 + 17, 99991),
                         (k ** (L - 2) + k ** (L // 2) - 7, 70001), (k ** L - 4099, 4099)):
            yield order, compress, lo, lo + size


@pytest.mark.parametrize("order,compress,lo,hi", list(_windows()))
def test_window_in_blocks(oracle_lib, tmp_path, order, compress, lo, hi):
    m = 2**64 - 1
    oa, ob = tmp_path / "oa", tmp_path / "ob"
    ost = GenStats()
    rc = oracle_lib.gpo_generate_window(order, compress, 0, str(oa).encode(), str(ob).encode(), lo >> 64, lo & m,
                                        hi >> 64, hi & m, ctypes.byref(ost))
    assert rc == 0
    with gp.Context(0) as ctx:
        st = ctx.generate_window(order, compress, 0, lo, hi, tmp_path / "a", tmp_path / "b")
    assert st.necklaces == ost.necklaces
    assert (tmp_path / "a").read_bytes() == oa.read_bytes()
    assert (tmp_path / "b").read_bytes() == ob.read_bytes()
