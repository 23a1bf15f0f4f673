"""Inputs that the sort and the match refuse."""
import ctypes

import pytest

import golaypair_gb300 as gp

pytestmark = pytest.mark.gpu


def test_sort_refuses_a_directory(tmp_path):
    (tmp_path / "in").write_text("b\na\n")
    (tmp_path / "dir").mkdir()
    for names in (["dir"], ["in", "dir"]):
        arr = (ctypes.c_char_p * len(names))(*[str(tmp_path / x).encode() for x in names])
        with gp.Context(0) as ctx:
            rc = ctx._lib.gp_sort(ctx.handle, ctypes.cast(arr, ctypes.c_void_p), len(names),
                                  str(tmp_path / "out").encode())
        assert rc < 0
        assert not (tmp_path / "out").exists()


@pytest.mark.parametrize("a,b", [("dir", "f"), ("f", "dir")])
def test_match_refuses_a_directory(tmp_path, a, b):
    (tmp_path / "f").write_text("PSD1 1 1 1 1 \n")
    (tmp_path / "dir").mkdir()
    n = ctypes.c_int64()
    with gp.Context(0) as ctx:
        rc = ctx._lib.gp_match(ctx.handle, 4, 1, 0, str(tmp_path / a).encode(), str(tmp_path / b).encode(),
                               str(tmp_path / "out").encode(), 0, ctypes.byref(n))
    assert rc < 0


def _lines(n):
    return "".join(f"PSD{100000 + k} 1 1 1 -1 \n" for k in range(n))


# below a stream's buffer only the close fails, above it a write does and the
# close may not; "!" is left to the sort's host path, "+1" to the match's
@pytest.mark.parametrize("n,extra", [(3, ""), (20000, ""), (20000, "!\n")])
def test_sort_onto_a_full_disk(tmp_path, n, extra):
    (tmp_path / "in").write_text(_lines(n) + extra)
    arr = (ctypes.c_char_p * 1)(str(tmp_path / "in").encode())
    with gp.Context(0) as ctx:
        assert ctx._lib.gp_sort(ctx.handle, ctypes.cast(arr, ctypes.c_void_p), 1, b"/dev/full") == -6  # GP_ERR_IO


@pytest.mark.parametrize("n,plus", [(3, False), (20000, False), (20000, True)])
def test_match_onto_a_full_disk(tmp_path, n, plus):
    # x = + + + -: PAF(1) + PAF(1) = 0 and PAF(2) + PAF(2) = 0, so every line meets its own
    text = _lines(n).replace(" 1 ", " +1 ") if plus else _lines(n)
    (tmp_path / "a").write_text(text)
    m = ctypes.c_int64()
    with gp.Context(0) as ctx:
        args = (ctx.handle, 4, 1, 0, str(tmp_path / "a").encode(), str(tmp_path / "a").encode())
        assert ctx._lib.gp_match(*args, str(tmp_path / "out").encode(), 0, ctypes.byref(m)) == 0 and m.value == n
        assert ctx._lib.gp_match(*args, b"/dev/full", 0, ctypes.byref(m)) == -6
