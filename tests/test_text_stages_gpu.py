"""Sort and match on texts at the edges of their device paths, and on texts
they leave to the host's line index and parser.  Bar: the oracle's files."""
import ctypes

import numpy as np
import pytest

import golaypair_gb300 as gp

pytestmark = pytest.mark.gpu


def _candidates(n, L, seed, tokens=40):
    """Lines of few distinct first tokens over +-1, so that tokens repeat."""
    rng = np.random.default_rng(seed)
    x = rng.choice([-1, 1], size=(n, L))
    t = rng.integers(0, tokens, n)
    return [f"PSD{10 ** int(k % 5)}{k} " + " ".join(map(str, r)) + " \n" for k, r in zip(t, x)]


def _sort_texts():
    lines = _candidates(3000, 9, 1)
    yield "candidates", ["".join(lines)]
    yield "two files, duplicates", ["".join(lines[:2000]), "".join(lines[1000:])]
    yield "no newline at the end", ["".join(lines[:50]).rstrip("\n"), "".join(lines[40:90]).rstrip("\n")]
    yield "empty lines", ["\n\n" + "".join(lines[:20]) + "\n" + "".join(lines[10:20]) + "\n\n"]
    yield "other characters", ["b\na\n\tz\n" + "".join(lines[:30]) + "A\r\n\xff\xfe\n~\n"]
    yield "one line", ["PSD1 1 \n"]
    yield "one newline", ["\n"]
    yield "an empty file among others", ["", "".join(lines[:10]), ""]
    yield "nothing", ["", ""]
    yield "text of whole blocks", ["1" * 4095 + "\n" + "2" * 8191 + "\n" + "1" * 4094 + "\n"]
    yield "a long line", ["9" * 70000 + "\n" + "9" * 69999 + "\n" + "1\n"]
    yield "prefixes", ["1\n11\n111\n1 \n1-\n11 \n"]


@pytest.mark.parametrize("name,texts", [pytest.param(*c, id=c[0].replace(" ", "_")) for c in _sort_texts()])
def test_sort_matches_oracle(oracle_lib, tmp_path, name, texts):
    paths = []
    for i, t in enumerate(texts):
        p = tmp_path / f"in{i}"
        p.write_bytes(t.encode("latin-1"))
        paths.append(str(p).encode())
    arr = (ctypes.c_char_p * len(paths))(*paths)
    got, want = str(tmp_path / "got").encode(), str(tmp_path / "want").encode()
    with gp.Context(0) as ctx:
        for _ in range(2):
            ctx.check(ctx._lib.gp_sort(ctx.handle, ctypes.cast(arr, ctypes.c_void_p), len(paths), got), "gp_sort")
    assert oracle_lib.gpo_sort(ctypes.cast(arr, ctypes.c_void_p), len(paths), want) == 0
    assert (tmp_path / "got").read_bytes() == (tmp_path / "want").read_bytes()


def test_sort_onto_its_input(tmp_path):
    p = tmp_path / "f"
    p.write_text("b\na\nb\n")
    arr = (ctypes.c_char_p * 1)(str(p).encode())
    with gp.Context(0) as ctx:
        ctx.check(ctx._lib.gp_sort(ctx.handle, ctypes.cast(arr, ctypes.c_void_p), 1, str(p).encode()), "gp_sort")
    assert p.read_text() == "a\nb\n"


def _match_texts():
    def srt(n, seed, tokens=40):
        return "".join(sorted(set(_candidates(n, 4, seed, tokens))))
    a, b = srt(400, 2), srt(900, 3)
    yield "sorted", a, b
    yield "one token", srt(60, 4, 1), srt(64, 5, 1)
    yield "no common token", "PSD1 1 1 1 1 \n", "PSD2 1 1 1 -1 \n"
    yield "no newline at the end", a.rstrip("\n"), b.rstrip("\n")
    yield "unsorted", "".join(_candidates(200, 4, 6)), b
    yield "unsorted b", a, "".join(_candidates(200, 4, 7))
    yield "lines of blanks", a + "   \n\n" + " " * 3, "\n" + b
    yield "leading blanks", "".join("  " + x for x in a.splitlines(True)), b
    yield "more values than L", "".join(x[:-2] + " 1 1 \n" for x in a.splitlines(True)), b
    # a sign joined to the first token leaves a line one value short: refused
    yield "signs without blanks", a.replace(" -1", "-1").replace("PSD-1", "PSD -1"), b
    parts = [x.split(" ", 1) for x in a.splitlines(True)]
    yield "values without blanks", "".join(t + " " + v.replace("1 -1", "1-1") for t, v in parts), b
    yield "CRLF", a.replace("\n", "\r\n"), b
    yield "plus signs", a.replace(" 1", " +1"), b


@pytest.mark.parametrize("name,a,b", [pytest.param(*c, id=c[0].replace(" ", "_")) for c in _match_texts()])
def test_match_matches_oracle(oracle_lib, tmp_path, name, a, b):
    pa, pb = str(tmp_path / "a"), str(tmp_path / "b")
    for p, t in ((pa, a), (pb, b)):
        with open(p, "wb") as f:
            f.write(t.encode())
    got, want = str(tmp_path / "got"), str(tmp_path / "want")
    n, m = ctypes.c_int64(), ctypes.c_int64()
    with gp.Context(0) as ctx:
        rc = ctx._lib.gp_match(ctx.handle, 4, 1, 0, pa.encode(), pb.encode(), got.encode(), 0, ctypes.byref(n))
    orc = oracle_lib.gpo_match(4, 1, 0, pa.encode(), pb.encode(), want.encode(), 0, ctypes.byref(m))
    if name == "signs without blanks":
        assert rc == -7  # GP_ERR_FORMAT
        return
    assert rc == orc == 0 and n.value == m.value
    with open(got, "rb") as f, open(want, "rb") as g:
        assert f.read() == g.read()


@pytest.mark.parametrize("rows,run,chars", [
    (2, 2, "09"), (31, 1, "0123456789"), (4096, 31, "0123456789"), (4096, 32, "0123456789"),
    (4100, 33, "0123456789"), (4096, 1024, "-0123456789"), (6000, 32, "abcdefghAB"), (20000, 2, " 1"),
    (2**19 + 5, 1, "0123456789"), (2**19, 2, "0123456789"),
])
def test_sort_of_lines_with_equal_starts(oracle_lib, tmp_path, rows, run, chars):
    """Runs of lines whose first 24 characters agree, a quarter of them whole."""
    rng = np.random.default_rng(rows + run)
    c = np.frombuffer(chars.encode(), np.uint8)
    lead = np.repeat(rng.choice(c, (-(-rows // run), 24)), run, axis=0)[:rows]
    tail = rng.choice(c, (rows, 17))
    same = rng.random(rows) < 0.25
    tail[same] = tail[0]
    rng.shuffle(text := np.concatenate([lead, tail, np.full((rows, 1), 10, np.uint8)], axis=1))
    (tmp_path / "in").write_bytes(text.tobytes())
    arr = (ctypes.c_char_p * 1)(str(tmp_path / "in").encode())
    got, want = str(tmp_path / "got").encode(), str(tmp_path / "want").encode()
    with gp.Context(0) as ctx:
        ctx.check(ctx._lib.gp_sort(ctx.handle, ctypes.cast(arr, ctypes.c_void_p), 1, got), "gp_sort")
    assert oracle_lib.gpo_sort(ctypes.cast(arr, ctypes.c_void_p), 1, want) == 0
    assert (tmp_path / "got").read_bytes() == (tmp_path / "want").read_bytes()
