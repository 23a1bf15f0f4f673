"""Pair files as the equivalence filter reads and writes them: layouts the
device parser takes, and those it leaves to strtol (signs, large values, a
token that ends the values).  Bar: the oracle's output file."""
import numpy as np
import pytest

import golaypair_gb300 as gp

pytestmark = pytest.mark.gpu


def _pairs(L, n, values, seed):
    rng = np.random.default_rng(seed)
    p = rng.choice(values, size=(n, 2 * L))
    i = np.arange(L)
    shifted = np.concatenate([p[:, :L], p[:, L:][:, (i + 1) % L]], axis=1)   # images of the first ones
    swapped = np.concatenate([p[:, L:], p[:, :L]], axis=1)
    return np.concatenate([p, shifted, swapped[: n // 2], p[: n // 3]])


def _text(p, L, sep=" ", mid="  ", end=" \n"):
    return "".join(sep.join(map(str, r[:L])) + mid + sep.join(map(str, r[L:])) + end for r in p)


def _cases():
    one, wide = [-1, 1], [-11, -1, 0, 3, 127]
    yield "plain", 5, 1, _text(_pairs(5, 400, one, 1), 5)
    yield "no newline at the end", 4, 1, _text(_pairs(4, 300, one, 2), 4).rstrip()
    yield "tabs and CRLF", 7, 1, _text(_pairs(7, 200, one, 3), 7, "\t", "\t\t", "\r\n")
    yield "all on one line", 6, 2, _text(_pairs(6, 500, [-2, 0, 2], 4), 6, end=" ")
    yield "several digits", 9, 15, _text(_pairs(9, 700, wide, 5), 9)
    yield "a partial pair at the end", 8, 1, _text(_pairs(8, 150, one, 6), 8) + "1 -1 1\n"
    yield "plus signs", 5, 1, _text(_pairs(5, 100, one, 7), 5).replace(" 1", " +1")
    yield "leading zeros", 5, 1, _text(_pairs(5, 100, one, 8), 5).replace(" 1", " 0001")
    yield "values end at a word", 6, 1, _text(_pairs(6, 90, one, 9), 6) + "end " + _text(_pairs(6, 9, one, 10), 6)
    yield "values end inside a token", 6, 1, _text(_pairs(6, 90, one, 11), 6) + "1-1 1x " + "1 " * 30
    yield "empty", 5, 1, ""
    yield "blanks only", 5, 1, " \n\t \n"
    yield "blocks of text", 3, 1, "\n" * 4095 + _text(_pairs(3, 5000, one, 12), 3) + " " * 4097
    yield "long rows", 128, 1, _text(_pairs(128, 40, one, 13), 128)


@pytest.mark.parametrize("name,L,compress,text", [pytest.param(*c, id=c[0].replace(" ", "_")) for c in _cases()])
def test_pair_text_matches_oracle(oracle_lib, tmp_path, name, L, compress, text):
    src, got, want = (str(tmp_path / x) for x in ("in", "got", "want"))
    with open(src, "wb") as f:
        f.write(text.encode())
    order = L * compress
    with gp.Context(0) as ctx:
        ctx.check(ctx._lib.gp_equiv_filter(ctx.handle, order, compress, src.encode(), got.encode()), "gp_equiv_filter")
    if L > 64:  # the oracle's table of the group is too large: every pair's lines, once a class at most
        lines = open(got).read().splitlines()
        assert 0 < len(lines) <= 40 and len(set(lines)) == len(lines)
        return
    assert oracle_lib.gpo_equiv_filter(order, compress, src.encode(), want.encode()) == 0
    with open(got, "rb") as f, open(want, "rb") as g:
        assert f.read() == g.read()
