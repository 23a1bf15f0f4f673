"""Sorts of lines whose keys have more words than the digit totals are held for at once."""
import ctypes
import random
import subprocess
import sys

import pytest

import golaypair_gb300 as gp

pytestmark = pytest.mark.gpu

WORDS = 1024  # of a key: 8 characters each of candidate lines, 4 of others


def _sort(ctx, src, dst):
    arr = (ctypes.c_char_p * 1)(str(src).encode())
    ctx.check(ctx._lib.gp_sort(ctx.handle, ctypes.cast(arr, ctypes.c_void_p), 1, str(dst).encode()), "gp_sort")


@pytest.mark.parametrize("chars,per", [("0123456789-", 8), ("abcxyz!", 4)])
@pytest.mark.parametrize("same", [0, WORDS - 1, WORDS, WORDS + 1, 3 * WORDS])
def test_lines_around_a_slice_of_totals(tmp_path, chars, per, same):
    """Lines that agree in their first `same` words: few, and more than a run that is ranked."""
    rng = random.Random(same)
    word = lambda n: "".join(rng.choice(chars) for _ in range(n))
    with gp.Context(0) as ctx:
        for n in (2, 40, 700):
            head = word(same * per)
            lines = [head + word(rng.choice([0, 1, per, 2 * WORDS * per])) for _ in range(n)]
            tail = word(2 * WORDS * per)
            lines += [lines[0] + tail + x for x in sorted(chars)] * 4 + lines[: n // 2]
            rng.shuffle(lines)
            (tmp_path / "in").write_text("\n".join(lines) + "\n")
            _sort(ctx, tmp_path / "in", tmp_path / "out")
            assert (tmp_path / "out").read_text().split("\n")[:-1] == sorted(set(lines))


def test_lines_of_megabytes_take_no_gigabytes(tmp_path):
    """The totals of every digit of an 8 MB line would take 8 GB of host memory."""
    code = """if True:
        import ctypes, random, resource, sys
        import golaypair_gb300 as gp
        rng = random.Random(1)
        lines = [bytes(rng.choices(b"abcdefgh", k=8 << 20)) for _ in range(3)]
        open(sys.argv[1], "wb").write(b"\\n".join(lines) + b"\\n")
        with gp.Context(0) as ctx:
            before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
            arr = (ctypes.c_char_p * 1)(sys.argv[1].encode())
            ctx.check(ctx._lib.gp_sort(ctx.handle, ctypes.cast(arr, ctypes.c_void_p), 1, sys.argv[2].encode()), "gp_sort")
            grown = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before
        assert open(sys.argv[2], "rb").read().split(b"\\n")[:-1] == sorted(lines)
        print(grown)
    """
    r = subprocess.run([sys.executable, "-c", code, str(tmp_path / "in"), str(tmp_path / "out")], capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    assert int(r.stdout) < 1 << 20  # KB; the file and its copies are some 100 MB
