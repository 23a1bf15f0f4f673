"""Uncompressed pairs as the device sorts and writes them: several matches per
pair, pairs that repeat and come in any order, two-level chains, values of one
and two characters.  Bar: the oracle's files."""
import ctypes

import numpy as np
import pytest

import golaypair_gb300 as gp

pytestmark = pytest.mark.gpu


def _pairs(ctx, tmp_path, order, compress, paf):
    """The compressed pairs of an order, shuffled, some twice."""
    space = (compress + 1) ** (order // compress)
    ctx.generate_window(order, compress, paf, 0, space, tmp_path / "a", tmp_path / "b")
    for n in "ab":
        arr = (ctypes.c_char_p * 1)(str(tmp_path / n).encode())
        ctx.check(ctx._lib.gp_sort(ctx.handle, ctypes.cast(arr, ctypes.c_void_p), 1, str(tmp_path / f"{n}s").encode()),
                  "gp_sort")
    found = ctypes.c_int64()
    ctx.check(ctx._lib.gp_match(ctx.handle, order, compress, paf, str(tmp_path / "as").encode(),
                                str(tmp_path / "bs").encode(), str(tmp_path / "pairs").encode(), 0,
                                ctypes.byref(found)), "gp_match")
    lines = (tmp_path / "pairs").read_text().splitlines(True)
    rng = np.random.default_rng(order)
    lines = [lines[i] for i in rng.permutation(len(lines))[:60]]
    return lines + lines[:7]


@pytest.mark.parametrize("order,compress,new,paf", [(16, 2, 1, 0), (20, 2, 1, 0), (26, 2, 1, 0), (27, 3, 1, -2),
                                                    (36, 6, 3, 0), (40, 4, 2, 0), (34, 2, 1, 0)])
def test_uncompressed_pairs_match_oracle(oracle_lib, tmp_path, order, compress, new, paf):
    got, want = tmp_path / "got", tmp_path / "want"
    with gp.Context(0) as ctx:
        lines = _pairs(ctx, tmp_path, order, compress, paf)
        (tmp_path / "in").write_text("".join(lines))
        ctx.check(ctx._lib.gp_uncompress(ctx.handle, order, compress, new, paf, str(tmp_path / "in").encode(),
                                         str(got).encode(), str(tmp_path).encode(), b"d"), "gp_uncompress")
    assert lines
    assert oracle_lib.gpo_uncompress(order, compress, new, paf, str(tmp_path / "in").encode(), str(want).encode(),
                                     str(tmp_path).encode(), b"o") == 0
    assert got.read_bytes() == want.read_bytes()
