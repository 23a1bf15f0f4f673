"""The match past the sizes of its device path: 2^32 candidate pairs, and a
text of more than 4 GiB (a sparse file)."""
import ctypes
import shutil

import pytest

import golaypair_gb300 as gp

pytestmark = pytest.mark.gpu


def _match(d, a, b):
    n = ctypes.c_int64()
    with gp.Context(0) as ctx:
        ctx.check(ctx._lib.gp_match(ctx.handle, 4, 1, 0, str(d / a).encode(), str(d / b).encode(),
                                    str(d / "out").encode(), 0, ctypes.byref(n)), "gp_match")
    return n.value, (d / "out").read_text()


def _line(a, b):
    return a + "  " + b + " \n"


@pytest.mark.parametrize("na,nb", [(65537, 65537), (65536, 65535), (40000, 110000)])
def test_match_of_four_billion_candidate_pairs(tmp_path, na, nb):
    # one token, so every a line meets every b line.  PAF(1), PAF(2) of + + + +
    # are 4, 4 and of any rotation of + + + - 0, 0: only these match, each other
    common = "1 1 1 1"
    special = ["1 1 1 -1", "1 1 -1 1", "1 -1 1 1", "-1 1 1 1"]
    at_a, at_b = {0: special[0], na // 2: special[1], na - 1: special[2]}, {1: special[3], nb - 1: special[1]}
    for name, n, at in (("a", na, at_a), ("b", nb, at_b)):
        (tmp_path / name).write_text("".join(f"PSD0 {at.get(k, common)} \n" for k in range(n)))
    assert na * nb >= 1 << 31  # more than the device path takes
    n, out = _match(tmp_path, "a", "b")
    assert n == 6
    assert out == "".join(_line(x, y) for x in at_a.values() for y in at_b.values())


def test_match_of_a_text_past_four_gib(tmp_path):
    # values after the first L are not read: the first line goes on past 2^32 bytes
    with open("/proc/meminfo") as f:
        free = int(next(x for x in f if x.startswith("MemAvailable")).split()[1]) << 10
    if free < 24 << 30 or shutil.disk_usage(tmp_path).free < 8 << 30:
        pytest.skip("no room for a text of 4 GiB")
    with open(tmp_path / "a", "wb") as f:
        f.write(b"PSD1 1 1 1 -1 ")
        f.seek((1 << 32) + 100)
        f.write(b"\nPSD2 1 1 -1 1 \nPSD4 1 -1 1 1 \n")
    (tmp_path / "b").write_text("PSD1 1 1 1 -1 \nPSD2 1 -1 1 1 \nPSD3 1 1 1 -1 \nPSD4 -1 1 1 1 \n")
    n, out = _match(tmp_path, "a", "b")
    (tmp_path / "a").unlink()
    assert n == 3
    assert out == (_line("1 1 1 -1", "1 1 1 -1") + _line("1 1 -1 1", "1 -1 1 1") + _line("1 -1 1 1", "-1 1 1 1"))
