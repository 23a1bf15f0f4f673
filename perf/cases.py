"""What the framework's users have it do, as timed cases through its public entry points.

The framework runs one search path: candidate generation, PSD filter, sort and match,
uncompression, equivalence filter.  A user calls the batched filter on rows in device
or host memory, or the stages on the files of the path.  Each case below is one such
call (sort and match are two, always run together), over the range of orders, lengths
and sizes that searches use: the smallest calls, where launches and host work count,
and the largest, where the kernels do.

`prepare` makes what the user's program has before the call: rows of a length and
compression with a permitted row sum, or the files that the stage before would have
written (by running that stage).  `run` is the call.  Stage outputs are files; `run`
reads them whole into a buffer of a size fixed by the case (zeros after the end), as
the next program on the path would.
"""
import ctypes
import functools
import math
import os
import shutil
import tempfile

import numpy as np
import torch

import golaypair_gb300 as gp
from golaypair_gb300 import workloads

MIB = 1 << 20


# ------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest batch a caller bothers the GPU with: the survivors of one
        # search step at the benchmark's order (latency: launches, not rows)
        dict(name="filter_small_n90", kind="filter", order=90, compress=2, paf=0, rows=4096, mode="tc"),
        # an ordinary batch of uncompressed Legendre-type rows (length 57), not a
        # multiple of the 128-row tile
        dict(name="filter_n57_c1", kind="filter", order=57, compress=1, paf=-2, rows=1_000_003, mode="tc"),
        # the benchmark's own workload: 2^28 rows of length 45, larger than the L2
        dict(name="filter_large_n90", kind="filter", order=90, compress=2, paf=0, rows=1 << 28, mode="tc"),
        # long rows (length 98, compression 1): the widest padded lengths
        dict(name="filter_long_n98", kind="filter", order=98, compress=1, paf=0, rows=(1 << 24) + 77, mode="tc"),
        # the plain FP64 mode, which users take to check the fast one
        dict(name="filter_fp64_n90", kind="filter", order=90, compress=2, paf=0, rows=1 << 20, mode="fp64"),
        # rows that live in host memory (candidate files of another program)
        dict(name="filter_host_n68", kind="host", order=68, compress=2, paf=0, rows=(1 << 22) + 1),
        # one order, one window: a shard of the order-57 search
        dict(name="generate_n57", kind="generate", order=57, compress=3, paf=-2, words=1 << 32, out_mib=256),
        # the uneven batch of five orders, 2^32-word windows, one engine call
        dict(name="generate_batch", kind="batch", words=1 << 32, out_mib=256),
        # candidate files of a whole order (compression 3) sorted and matched
        dict(name="sort_match_n51", kind="match", order=51, compress=3, paf=-2, keep=0.9, out_mib=64),
        # a handful of small pairs: one uncompression call's fixed cost
        dict(name="uncompress_n39", kind="uncompress", order=39, compress=3, new_compress=1, paf=-2, pairs=200,
             out_mib=2),
        # a slice of the order-57 pairs, the stage that dominates that search
        dict(name="uncompress_n57", kind="uncompress", order=57, compress=3, new_compress=1, paf=-2, pairs=4000,
             out_mib=4),
        # equivalence classes among uncompressed pairs
        dict(name="equivalence_n57", kind="equivalence", length=57, pairs=30_000, out_mib=16),
    ]


# (order, compress, paf) with a permitted row sum, over the lengths the filter takes
FILTER_ORDERS = [(16, 2, 0), (26, 2, 0), (34, 2, 0), (50, 2, 0), (57, 3, -2), (58, 2, 0), (68, 2, 0), (90, 5, 0),
                 (82, 2, 0), (90, 2, 0), (57, 1, -2), (52, 1, 0), (61, 1, -2), (65, 1, -2), (74, 1, 0), (80, 1, 0),
                 (85, 1, -2), (90, 1, 0), (98, 1, 0), (106, 1, 0), (117, 1, -2), (122, 1, 0), (164, 2, 0),
                 (180, 2, 0)]
GENERATE_ORDERS = [(34, 2, 0), (50, 2, 0), (58, 2, 0), (68, 2, 0), (90, 5, 0), (57, 3, -2), (63, 3, -2)]
PAIR_ORDERS = [(26, 2, 1, 0), (34, 2, 1, 0), (33, 3, 1, -2), (39, 3, 1, -2), (45, 3, 1, -2), (51, 3, 1, -2),
               (57, 3, 1, -2)]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["filter", "filter", "filter", "fp64", "host", "generate", "batch", "match", "uncompress",
                       "uncompress", "equivalence"])
    if kind in ("filter", "fp64", "host"):
        order, c, paf = rng.choice(FILTER_ORDERS)
        length = order // c
        if kind == "fp64":
            return dict(kind="filter", order=order, compress=c, paf=paf, mode="fp64",
                        rows=_log(rng, 1000, (1 << 26) // length))
        if kind == "host":
            return dict(kind="host", order=order, compress=c, paf=paf, rows=_log(rng, 1000, (1 << 28) // length))
        return dict(kind="filter", order=order, compress=c, paf=paf, mode="tc",
                    rows=_log(rng, 1000, (1 << 31) // length))
    if kind == "generate":
        order, c, paf = rng.choice(GENERATE_ORDERS)
        return dict(kind="generate", order=order, compress=c, paf=paf, words=_log(rng, 1 << 22, 1 << 31),
                    out_mib=192)
    if kind == "batch":
        return dict(kind="batch", words=_log(rng, 1 << 22, 1 << 31), out_mib=192)
    if kind == "match":
        order = rng.choice([39, 45, 51])
        return dict(kind="match", order=order, compress=3, paf=-2, keep=round(rng.uniform(0.3, 0.95), 3), out_mib=64)
    if kind == "uncompress":
        order, c, cn, paf = rng.choice(PAIR_ORDERS)
        return dict(kind="uncompress", order=order, compress=c, new_compress=cn, paf=paf,
                    pairs=_log(rng, 100, 2000), out_mib=8)
    return dict(kind="equivalence", length=rng.randrange(20, 91), pairs=_log(rng, 100, 20_000), out_mib=16)


# ------------------------------------------------------------ shared pieces

@functools.lru_cache(maxsize=1)
def _context():
    """The one context a program keeps."""
    return gp.Context(0)


class _Folder:
    """A working folder, gone with the state that holds it."""

    def __init__(self):
        self.path = tempfile.mkdtemp(prefix="golay_", dir="/dev/shm" if os.path.isdir("/dev/shm") else None)

    def __del__(self):
        shutil.rmtree(self.path, ignore_errors=True)

    def __truediv__(self, name):
        return os.path.join(self.path, name)


class _Output:
    """The bytes of one stage's files, one after another, in a buffer of fixed size."""

    def __init__(self, mib):
        self.buf = np.zeros(mib * MIB, dtype=np.uint8)
        self.used = 0

    def read(self, paths):
        at = 0
        for p in paths:
            with open(p, "rb", buffering=0) as f:
                size = os.fstat(f.fileno()).st_size
                if at + size > len(self.buf):
                    raise RuntimeError(f"{p}: the output of this case needs more than {len(self.buf)} bytes")
                while size:
                    got = f.readinto(memoryview(self.buf)[at:at + size])
                    if not got:
                        raise RuntimeError(f"{p}: short read")
                    at += got
                    size -= got
        self.buf[at:self.used] = 0
        self.used = at
        return self.buf


def _row_sums(order, paf, length, compress):
    """The row sums a side of a pair can have: x with x^2 + y^2 = 2n + (n - 1) paf."""
    total = 2 * order + (order - 1) * paf
    out = [x for x in range(-length * compress, length * compress + 1)
           if x * x <= total and math.isqrt(total - x * x) ** 2 == total - x * x]
    assert out, (order, paf)
    return out


def _rows(order, compress, paf, n, seed):
    """n rows over the compression's alphabet, uniform but for a permitted row sum, on the GPU."""
    length = order // compress
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    sums = torch.zeros(2 * length * compress + 1, dtype=torch.bool, device="cuda")
    sums[torch.tensor(_row_sums(order, paf, length, compress), device="cuda") + length * compress] = True
    out = torch.empty((n, length), dtype=torch.int8, device="cuda")
    have = 0
    chunk = min(max(8 * n, 4096), (1 << 30) // length)
    while have < n:
        s = torch.randint(0, compress + 1, (chunk, length), generator=g, device="cuda", dtype=torch.int8)
        s.mul_(2).sub_(compress)
        s = s[sums[s.sum(1, dtype=torch.int32).long() + length * compress]]
        take = min(n - have, s.shape[0])
        out[have:have + take] = s[:take]
        have += take
    return out


def _call(name, *args):
    ctx = _context()
    ctx.check(getattr(gp.lib(), name)(ctx.handle, *args), name)


def _sort(inp, out):
    paths = (ctypes.c_char_p * 1)(inp.encode())
    _call("gp_sort", ctypes.cast(paths, ctypes.c_void_p), 1, out.encode())


@functools.lru_cache(maxsize=8)
def _whole_order(order, compress, paf):
    """The candidate lines (A, B) and the pair lines of a whole order's search at a compression."""
    d = _Folder()
    a, b, sa, sb, pairs = (d / x for x in ("a", "b", "sa", "sb", "pairs"))
    _context().generate_window(order, compress, paf, 0, (compress + 1) ** (order // compress), a, b)
    _sort(a, sa)
    _sort(b, sb)
    n = ctypes.c_int64()
    _call("gp_match", order, compress, paf, sa.encode(), sb.encode(), pairs.encode(), 0, ctypes.byref(n))
    got = []
    for p in ([a, b] if order <= 51 else []) + [pairs]:
        with open(p, "rb") as f:
            got.append(f.read().splitlines(keepends=True))
    return ([None, None] if order > 51 else []) + got


def _pair_text(a, b):
    """Pair lines of +-1 sequences: the values of a, two blanks, the values of b."""
    n, length = a.shape
    cells = np.zeros((n, 2 * length + 2, 3), dtype=np.uint8)  # zero bytes are dropped
    for at, x in ((0, a), (length + 1, b)):
        cells[:, at:at + length, 0] = np.where(x < 0, ord("-"), 0)
        cells[:, at:at + length, 1] = ord("1")
        cells[:, at:at + length, 2] = ord(" ")
    cells[:, length, 0] = ord(" ")
    cells[:, -1, 0] = ord("\n")
    flat = cells.reshape(-1)
    return flat[flat != 0].tobytes()


def _equivalent_pairs(length, pairs, seed):
    """Pairs in classes of about four: random pairs and images of them under shifts,
    reversal, negation, decimation and the swap, in random order."""
    rng = np.random.default_rng(seed)
    classes = (pairs + 3) // 4
    units = np.array([u for u in range(1, length) if math.gcd(u, length) == 1])
    base = rng.choice(np.array([-1, 1], dtype=np.int8), size=(classes, 2, length))
    pick = rng.integers(0, classes, pairs)
    x = base[pick]
    i = np.arange(length)
    rows = np.arange(pairs)[:, None]
    u = units[rng.integers(0, len(units), pairs)][:, None]
    half = []
    for h in (0, 1):
        shift = rng.integers(0, length, pairs)[:, None]
        turn = rng.choice([-1, 1], pairs)[:, None]
        sign = rng.choice(np.array([-1, 1], dtype=np.int8), pairs)[:, None]
        half.append(x[rows, h, (turn * u * i + shift) % length] * sign)
    swap = rng.integers(0, 2, pairs).astype(bool)[:, None]
    return np.where(swap, half[1], half[0]), np.where(swap, half[0], half[1])


# --------------------------------------------------------- prepare and run

def prepare(case, seed):
    k = case["kind"]
    st = dict(case, ctx=_context())
    if k == "filter":
        st["x"] = _rows(case["order"], case["compress"], case["paf"], case["rows"], seed)
        st["mask"] = torch.zeros((case["rows"] + 31) // 32, dtype=torch.int32, device="cuda")
    elif k == "host":
        st["x"] = _rows(case["order"], case["compress"], case["paf"], case["rows"], seed).cpu().numpy()
    else:
        st["dir"] = _Folder()
        st["out"] = _Output(case["out_mib"])
    if k == "generate":
        order, c = case["order"], case["compress"]
        space = (c + 1) ** (order // c)
        lo = min(workloads.necklace_anchor(order, c, seed), max(space - case["words"], 0))
        st["window"] = (lo, min(lo + case["words"], space))
    elif k == "batch":
        st["jobs"] = []
        for order, c in workloads.BATCH_ORDERS:
            space = (c + 1) ** (order // c)
            lo = 0 if space <= case["words"] else min(workloads.necklace_anchor(order, c, seed + order), space -
                                                      case["words"])
            st["jobs"].append((order, c, 0, lo, min(lo + case["words"], space), st["dir"] / f"{order}_{c}_a",
                               st["dir"] / f"{order}_{c}_b"))
    elif k == "match":
        rng = np.random.default_rng(seed)
        for name, lines in zip("ab", _whole_order(case["order"], case["compress"], case["paf"])):
            with open(st["dir"] / name, "wb") as f:
                f.writelines(x for x, r in zip(lines, rng.random(len(lines))) if r < case["keep"])
    elif k == "uncompress":
        lines = _whole_order(case["order"], case["compress"], case["paf"])[2]
        at = int(np.random.default_rng(seed).integers(0, len(lines)))
        with open(st["dir"] / "in", "wb") as f:  # consecutive pairs, as a split of the file gives them
            f.writelines((lines + lines)[at:at + min(case["pairs"], len(lines))])
    elif k == "equivalence":
        with open(st["dir"] / "in", "wb") as f:
            f.write(_pair_text(*_equivalent_pairs(case["length"], case["pairs"], seed)))
    return st


def run(st):
    k, ctx = st["kind"], st["ctx"]
    if k == "filter":
        mode = gp.GP_PSD_FP64 if st["mode"] == "fp64" else gp.GP_PSD_TC_GUARDED
        ctx.psd_filter_device(st["x"].data_ptr(), st["rows"], st["x"].shape[1], st["order"], st["paf"], mode,
                              st["mask"].data_ptr())
        return st["mask"]
    if k == "host":
        verdicts, stats = ctx.psd_filter(st["x"], st["order"], st["paf"])
        return {"verdicts": verdicts, "passes": stats.n_pass}
    d = st["dir"]
    if k == "generate":
        s = ctx.generate_window(st["order"], st["compress"], st["paf"], *st["window"], d / "a", d / "b")
        return {"files": st["out"].read([d / "a", d / "b"]), "necklaces": s.necklaces, "candidates": s.candidates,
                "pass": s.psd_pass, "a": s.written_a, "b": s.written_b}
    if k == "batch":
        stats, _ = ctx.generate_batch(st["jobs"])
        return {"files": st["out"].read([p for j in st["jobs"] for p in j[5:]]),
                "counts": np.array([[s.necklaces, s.candidates, s.psd_pass, s.written_a, s.written_b]
                                    for s in stats], dtype=np.int64)}
    if k == "match":
        _sort(d / "a", d / "sa")
        _sort(d / "b", d / "sb")
        n = ctypes.c_int64()
        _call("gp_match", st["order"], st["compress"], st["paf"], (d / "sa").encode(), (d / "sb").encode(),
              (d / "pairs").encode(), 0, ctypes.byref(n))
        return {"files": st["out"].read([d / "sa", d / "sb", d / "pairs"]), "pairs": n.value}
    if k == "uncompress":
        _call("gp_uncompress", st["order"], st["compress"], st["new_compress"], st["paf"], (d / "in").encode(),
              (d / "out").encode(), d.path.encode(), b"uncompress")
        return st["out"].read([d / "out"])
    _call("gp_equiv_filter", st["length"], 1, (d / "in").encode(), (d / "out").encode())
    return st["out"].read([d / "out"])


def work(case):
    """Bytes in and out once, and the operations of the plain algorithm.  Where the output's
    size depends on the data, the mean over these orders' searches stands for it."""
    k = case["kind"]
    if k in ("filter", "host"):
        length, n = case["order"] // case["compress"], case["rows"]
        h = length // 2
        return {"bytes": n * length + n / 8, "flops": n * (4 * length * h + 3 * h)}
    if k in ("generate", "batch"):
        jobs = [(case["order"], case["compress"])] if k == "generate" else workloads.BATCH_ORDERS
        ops = 0
        for order, c in jobs:
            length = order // c
            words = min(case["words"], (c + 1) ** length)
            # every length-th word a necklace (one successor each, length operations),
            # every tenth of those through the PSD filter
            ops += words + words / length / 10 * (4 * length * (length // 2))
        return {"bytes": 1 * MIB, "flops": ops}
    if k == "match":
        lines = {39: 9e3, 45: 7e4, 51: 4.8e5}[case["order"]] * case["keep"]
        return {"bytes": 2 * 80 * lines, "flops": lines * 20}
    if k == "uncompress":
        length = case["order"] // case["compress"]
        r = case["compress"] // case["new_compress"]
        # about 3/4 of the letters have r choices each; the bins that vary, five operations each
        return {"bytes": case["pairs"] * 4 * length,
                "flops": case["pairs"] * 2 * r ** (0.75 * length) * 5 * (case["order"] / case["new_compress"] / 2)}
    n, length = case["pairs"], case["length"]
    return {"bytes": n * 2 * 2.5 * length * 1.25, "flops": n * 4 * length * length * length / 2}
