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
