"""Generation when the host has no room: for the text made on the device (the
records are then formatted on the host, into the same files), for the records
and their lines as well (GP_ERR_NOMEM).  No exception crosses the C ABI or
ends a thread."""
import os
import subprocess

import pytest

import golaypair_gb300 as gp

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("alloc_limit") / "alloc_limit"
    where = os.path.dirname(gp.LIB_PATH)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(os.path.dirname(HERE), "include"),
                    os.path.join(HERE, "alloc_limit.cpp"), gp.LIB_PATH, f"-Wl,-rpath,{where}", "-o", str(exe)],
                   check=True)
    return exe


def _run(program, entry, d, first, count):
    d.mkdir(exist_ok=True)
    r = subprocess.run([str(program), entry, str(d), str(first), str(count)], stdout=subprocess.PIPE, timeout=100)
    assert r.returncode == 0, {2: "an exception crossed the C ABI", 3: "an exception ended a thread"}.get(r.returncode, r)
    return int(r.stdout), {p.name: p.read_bytes() for p in sorted(d.iterdir())}


@pytest.mark.parametrize("entry", ["generate", "window", "batch"])
def test_generation_without_room_on_the_host(program, tmp_path, entry):
    rc, want = _run(program, entry, tmp_path / "want", 0, 0)
    assert rc == 0 and len(want) == (4 if entry == "batch" else 2) and len(want["a"]) > 100000
    # the first large allocation is the (first job's) text
    assert _run(program, entry, tmp_path / "host", 0, 1) == (0, want)
    assert _run(program, entry, tmp_path / "none", 0, 1 << 40)[0] == -4  # GP_ERR_NOMEM
    for first in range(1, 8):  # room for some of the text, records or lines
        for count in (1, 1 << 40):
            rc, got = _run(program, entry, tmp_path / f"{first}_{count}", first, count)
            assert rc == -4 or (rc == 0 and got == want)
