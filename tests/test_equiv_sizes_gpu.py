"""Pair files on both sides of the size from which the device parses and sorts
them, equal pairs included, and every layout of test_equiv_text_gpu past it.
Bar: the oracle's output file."""
import numpy as np
import pytest

import golaypair_gb300 as gp
from test_equiv_text_gpu import _cases, _pairs, _text

pytestmark = pytest.mark.gpu
LINE = 40 << 10  # bytes


def _check(oracle_lib, d, L, compress, text):
    src, got, want = (str(d / x) for x in ("in", "got", "want"))
    with open(src, "wb") as f:
        f.write(text.encode())
    order = L * compress
    with gp.Context(0) as ctx:
        for _ in range(2):  # the second call finds the first one's buffers
            ctx.check(ctx._lib.gp_equiv_filter(ctx.handle, order, compress, src.encode(), got.encode()), "gp_equiv_filter")
    assert oracle_lib.gpo_equiv_filter(order, compress, src.encode(), want.encode()) == 0
    with open(got, "rb") as f, open(want, "rb") as g:
        assert f.read() == g.read()


@pytest.mark.parametrize("L,compress,values", [(1, 1, [-1, 1]), (2, 1, [-1, 1]), (3, 1, [-1, 1]), (6, 1, [-1, 1]),
                                               (9, 15, [-128, -11, -1, 0, 3, 127]), (15, 3, [-3, -1, 1, 3]),
                                               (24, 1, [-1, 1])])
@pytest.mark.parametrize("size", [LINE - 1, LINE, LINE + 1, 2 * LINE])
def test_sizes_at_the_line(oracle_lib, tmp_path, L, compress, values, size):
    lines = _text(_pairs(L, 60, values, L), L).splitlines(True)
    rng = np.random.default_rng(size)
    text = ""
    while len(text) < size - 4000:  # each pair a few times, in any order
        text += "".join(lines[i] for i in rng.permutation(len(lines)))
    text = text[:text.rfind("\n", 0, size - 3) + 1]
    _check(oracle_lib, tmp_path, L, compress, text + "\n" * (size - len(text)))


@pytest.mark.parametrize("name,L,compress,text", [pytest.param(*c, id=c[0].replace(" ", "_")) for c in _cases()
                                                  if c[1] <= 64])
def test_layouts_past_the_line(oracle_lib, tmp_path, name, L, compress, text):
    _check(oracle_lib, tmp_path, L, compress, "\n" * LINE + " " + text)
