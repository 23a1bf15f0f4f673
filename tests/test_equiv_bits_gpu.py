"""Least images of +-1 pairs as words of bits, lengths up to 64, against the
same pairs with every entry doubled, which take the general path (the group acts
on positions and signs only, so the classes are the same), and against the
oracle where its table of the group is small."""
import numpy as np
import pytest

import golaypair_gb300 as gp

pytestmark = pytest.mark.gpu


def _pairs(L):
    rng = np.random.default_rng(L)
    i = np.arange(L)
    rows = [rng.choice([-1, 1], 2 * L) for _ in range(40)]
    one = np.ones(L, int)
    alt = 1 - 2 * (i % 2)
    third = np.where(i % 3 == 0, 1, -1)
    for a in (one, alt, third):          # many elements fix these
        for b in (one, -alt, third):
            rows.append(np.concatenate([a, b]))
    units = [u for u in range(1, L) if np.gcd(u, L) == 1]
    for r in list(rows):
        a, b = r[:L], r[L:]
        u, s, t = units[rng.integers(len(units))], rng.integers(L), rng.integers(L)
        a2, b2 = a[(u * i + s) % L], b[(u * i + t) % L]
        if L % 2 == 0:
            a2, b2 = a2 * alt, b2 * alt
        rows.append(np.concatenate([b2, a2] if rng.integers(2) else [a2, b2]))
    return np.array(rows)


def _classes(tmp_path, L, p, name):
    src, dst = tmp_path / f"{name}.in", tmp_path / f"{name}.out"
    src.write_text("".join(" ".join(map(str, r[:L])) + "  " + " ".join(map(str, r[L:])) + " \n" for r in p))
    with gp.Context(0) as ctx:
        ctx.check(ctx._lib.gp_equiv_filter(ctx.handle, L, 1, str(src).encode(), str(dst).encode()), "gp_equiv_filter")
    return src, dst.read_text()


@pytest.mark.parametrize("L", [3, 4, 5, 8, 15, 16, 31, 32, 33, 34, 45, 57, 62, 63, 64, 65])
def test_bits_equal_general_path(oracle_lib, tmp_path, L):
    p = _pairs(L)
    src, got = _classes(tmp_path, L, p, "one")
    _, doubled = _classes(tmp_path, L, 2 * p, "two")
    assert got == doubled.replace("2", "1")
    if L <= 34:
        want = tmp_path / "want"
        assert oracle_lib.gpo_equiv_filter(L, 1, str(src).encode(), str(want).encode()) == 0
        assert got == want.read_text()
