"""Host threads that run out of memory: the calling thread learns of it, and
the text export of binary survivor files (host only) returns GP_ERR_NOMEM."""
import os
import struct
import subprocess

import numpy as np

import golaypair_gb300 as gp

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)


def test_exceptions_of_host_threads_reach_the_caller(tmp_path):
    (tmp_path / "t.cpp").write_text("""
#include <atomic>
#include <cstdio>
#include <stdexcept>
#include "host_par.h"
int main() {
    for (size_t blocks : {1, 2, 100}) {
        std::atomic<int> ran{0};
        bool caught = false;
        try {
            gp::par_for(blocks, [&](size_t b) { ++ran; if (b + 1 == blocks) throw std::runtime_error("last"); });
        } catch (const std::runtime_error&) { caught = true; }
        if (!caught || ran != (int)blocks) return 1;
    }
    int left = 0;
    try {
        gp::Workers w;
        for (int t = 0; t < 8; ++t) w.run([&left, t] { if (t % 2) throw std::runtime_error("odd"); });
        w.join();
    } catch (const std::runtime_error&) { left = 1; }
    return left == 1 ? 0 : 2;
}
""")
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", os.path.join(REPO, "golaypair_gb300", "csrc"),
                    str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0


def test_export_without_room_on_the_host(tmp_path):
    L, n = 16, 40000  # several blocks of records, +-1, 2 bytes of word, 1 of each signature value
    body = np.random.default_rng(1).integers(0, 256, (n, 2 + L - 1), dtype=np.uint8)
    hdr = b"GPSURV01" + struct.pack("<I9iQ", 1, L, 1, 0, L, 2, 1, 0, 1, 2, n)
    (tmp_path / "in").write_bytes(hdr + struct.pack("<16b", -1, 1, *[0] * 14) + bytes(8) + body.tobytes())
    exe = tmp_path / "alloc_limit"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(REPO, "include"), os.path.join(HERE, "alloc_limit.cpp"),
                    gp.LIB_PATH, f"-Wl,-rpath,{os.path.dirname(gp.LIB_PATH)}", "-o", str(exe)], check=True)

    def run(first, count):
        r = subprocess.run([str(exe), "export", str(tmp_path), str(first), str(count)], stdout=subprocess.PIPE)
        assert r.returncode == 0, {2: "an exception crossed the C ABI", 3: "an exception ended a thread"}.get(r.returncode, r)
        return int(r.stdout)

    assert run(0, 0) == 0
    want = (tmp_path / "a").read_bytes()
    assert want.count(b"\n") == n
    for first in range(12):
        rc = run(first, 1)
        assert rc == -4 or (rc == 0 and (tmp_path / "a").read_bytes() == want)
    assert run(0, 1 << 40) == -4
