"""The tensor-core filter where many rows lie near the bound: lengths at the
edges of every padded length above 48 (the accumulator holds the high twiddle
halves alone there, and a row inside that band is decided again in fp32, then
in FP64).  Bar: the oracle's verdicts and files."""
import ctypes

import numpy as np
import pytest

import golaypair_gb300 as gp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [47, 48, 57, 62, 63, 64, 79, 80, 95, 96, 111, 112, 127])
def test_bound_amid_the_row_maxima(oracle_lib, L):
    rng = np.random.default_rng(L)
    n = 20_000 + 45
    seqs = rng.choice(np.array([-1, 1], dtype=np.int8), size=(n, L))
    # the median of the row maxima: (1 - exp(-T / L))^(L / 2) = 1 / 2
    order = int(-L * np.log(1 - 0.5 ** (2 / L)) / 2)
    want = np.zeros(n, dtype=np.uint8)
    oracle_lib.gpo_psd_filter_batch(seqs.ctypes.data, n, L, order, 0, want.ctypes.data, 4)
    with gp.Context(0) as ctx:
        got, st = ctx.psd_filter(seqs, order, 0, gp.GP_PSD_TC_GUARDED)
    assert 0.2 * n < want.sum() < 0.8 * n
    assert np.array_equal(got, want.astype(bool))
    assert 0 < st.n_unsure < 0.2 * n


def _passing_word(oracle_lib, order):
    """Rank of the least dihedral image of a +-1 word that passes the filter
    and has a b-side row sum (the oracle writes it: the window holds a line)."""
    x, y = (ctypes.c_int * 64)(), (ctypes.c_int * 64)()
    sums = list(y[:oracle_lib.gpo_decomps(2 * order, x, y, 64)])
    rng = np.random.default_rng(order)
    while True:
        x = rng.choice(np.array([-1, 1]), size=(1 << 17, order))
        psd = np.abs(np.fft.rfft(x, axis=1)[:, 1:]) ** 2
        s = x.sum(1)
        ok = (psd.max(1) <= 2 * order) & np.isin(s, sums)
        if ok.any():
            d = ((x[np.argmax(ok)] + 1) // 2).tolist()
            images = [r[i:] + r[:i] for r in (d, d[::-1]) for i in range(order)]
            return int("".join(map(str, min(images))), 2)


@pytest.mark.parametrize("order", [52, 58, 74])
def test_packed_long_words_match_oracle(oracle_lib, tmp_path, order):
    at = _passing_word(oracle_lib, order)
    lo, hi = max(at - (1 << 12), 0), at + (1 << 12)
    m = (1 << 64) - 1
    a, b, oa, ob = (str(tmp_path / x) for x in ("a", "b", "oa", "ob"))
    with gp.Context(0) as ctx:
        ctx.generate_window(order, 1, 0, lo, hi, a, b)
    assert oracle_lib.gpo_generate_window(order, 1, 0, oa.encode(), ob.encode(), lo >> 64, lo & m, hi >> 64, hi & m,
                                          None) == 0
    lines = 0
    for x, y in ((a, oa), (b, ob)):
        with open(x, "rb") as f, open(y, "rb") as g:
            got = f.read()
            assert got == g.read()
            lines += got.count(b"\n")
    assert lines > 0
