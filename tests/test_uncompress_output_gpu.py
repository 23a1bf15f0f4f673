"""The uncompression's output file and buffers."""
import ctypes
import threading

import pytest

import golaypair_gb300 as gp

pytestmark = pytest.mark.gpu


def _pairs(ctx, d, order, compress, paf):
    """The pair lines of a whole order at a compression."""
    ctx.generate_window(order, compress, paf, 0, (compress + 1) ** (order // compress), d / "a", d / "b")
    for n in "ab":
        arr = (ctypes.c_char_p * 1)(str(d / n).encode())
        ctx.check(ctx._lib.gp_sort(ctx.handle, ctypes.cast(arr, ctypes.c_void_p), 1, str(d / f"{n}s").encode()), "gp_sort")
    ctx.check(ctx._lib.gp_match(ctx.handle, order, compress, paf, str(d / "as").encode(), str(d / "bs").encode(),
                                str(d / "pairs").encode(), 0, ctypes.byref(ctypes.c_int64())), "gp_match")
    return (d / "pairs").read_text().splitlines(True)


def _uncompress(ctx, d, order, compress, new, paf, out):
    return ctx._lib.gp_uncompress(ctx.handle, order, compress, new, paf, str(d / "in").encode(), str(out).encode(),
                                  str(d).encode(), b"d")


@pytest.mark.parametrize("whole", [False, True])
def test_uncompress_onto_a_full_disk(tmp_path, whole):
    with gp.Context(0) as ctx:
        lines = _pairs(ctx, tmp_path, 16, 2, 0)
        for n in [len(lines)] if whole else range(1, len(lines)):
            (tmp_path / "in").write_text("".join(lines[:n]) * (2000 if whole else 1))
            assert _uncompress(ctx, tmp_path, 16, 2, 1, 0, tmp_path / "out") == 0
            if (tmp_path / "out").stat().st_size:
                break
        size = (tmp_path / "out").stat().st_size
        # the first pairs' lines stay in the stream's buffer until it is closed
        assert size > 1 << 16 if whole else 0 < size < 4096
        assert _uncompress(ctx, tmp_path, 16, 2, 1, 0, "/dev/full") == -6  # GP_ERR_IO


def test_many_matches_leave_no_buffers_of_theirs(tmp_path):
    # a match of this order takes 260 bytes of sort key alone; a call's match
    # buffers are there while it runs, and those above 64 MB gone after it
    torch = pytest.importorskip("torch")
    with gp.Context(0) as ctx:
        lines = _pairs(ctx, tmp_path, 39, 3, -2)
        (tmp_path / "in").write_text("".join(lines))
        assert _uncompress(ctx, tmp_path, 39, 3, 1, -2, tmp_path / "out") == 0
        per_copy = (tmp_path / "out").read_text().count("\n")
        copies = -(-(1 << 20) // per_copy)
        (tmp_path / "in").write_text("".join(lines) * copies)
        assert _uncompress(ctx, tmp_path, 39, 3, 1, -2, tmp_path / "out") == 0  # every other buffer has its size
        after, least = torch.cuda.mem_get_info()[0], []
        done = threading.Event()

        def watch():
            while not done.is_set():
                least.append(torch.cuda.mem_get_info()[0])

        t = threading.Thread(target=watch)
        t.start()
        try:
            assert _uncompress(ctx, tmp_path, 39, 3, 1, -2, tmp_path / "out") == 0
        finally:
            done.set()
            t.join()
        assert (tmp_path / "out").stat().st_size > 1 << 26
        assert after - min(least) >= 260 << 20
        assert torch.cuda.mem_get_info()[0] >= after - (1 << 20)
