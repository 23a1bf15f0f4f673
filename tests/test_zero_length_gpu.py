"""Orders that leave a sequence no entries: the stages that take them write
the same lines, or none, whichever path reads the text."""
import ctypes

import pytest

import golaypair_gb300 as gp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lines", [1, 40, 700])
def test_match_of_sequences_without_entries(tmp_path, lines):
    # every line is its token alone, and equal tokens are a pair: a blank
    # between two empty sequences, and the newline
    text = "".join(f"PSD{1000 + k}\n" for k in range(lines))
    (tmp_path / "a").write_text(text)
    (tmp_path / "b").write_text(text)
    n = ctypes.c_int64(-1)
    with gp.Context(0) as ctx:
        rc = ctx._lib.gp_match(ctx.handle, 0, 1, 0, str(tmp_path / "a").encode(), str(tmp_path / "b").encode(),
                               str(tmp_path / "out").encode(), 0, ctypes.byref(n))
    assert rc == 0 and n.value == lines
    assert (tmp_path / "out").read_text() == " \n" * lines


@pytest.mark.parametrize("order", [0, -4])
@pytest.mark.parametrize("values", ["", "1 -1 1 -1 \n", "1 1  -1 1 \n" * 300])
def test_equivalence_of_pairs_without_entries(tmp_path, order, values):
    (tmp_path / "in").write_text(values)
    (tmp_path / "out").write_text("an older file")
    with gp.Context(0) as ctx:
        rc = ctx._lib.gp_equiv_filter(ctx.handle, order, 1, str(tmp_path / "in").encode(), str(tmp_path / "out").encode())
    assert rc == 0
    assert (tmp_path / "out").read_bytes() == b""  # no pair to write
