"""The plain FP64 filter at the edges of its blocks: row counts around the
rows of a block (128 to 1024, by batch size and length), lengths with and
without a middle entry, bin counts that are not a multiple of a round's four,
the whole int8 range.  Bar: the oracle's verdicts, bit for bit."""
import numpy as np
import pytest

import golaypair_gb300 as gp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,n", [(1, 40), (2, 33), (3, 1), (3, 31), (4, 129), (9, 128), (10, 127), (16, 1025),
                                 (5, 152 * 2048 + 1), (12, 152 * 1024 + 31), (45, 152 * 512 + 513), (127, 700),
                                 (200, 300), (333, 257), (512, 131)])
def test_fp64_filter_block_edges(oracle_lib, L, n):
    rng = np.random.default_rng(L * 1000 + n)
    small = rng.choice(np.array([-3, -1, 1, 3], dtype=np.int8), size=(n, L))
    wide = rng.integers(-128, 128, size=(n, L)).astype(np.int8)
    with gp.Context(0) as ctx:
        for seqs, power in ((small, 5.0), (wide, 5461.0)):
            # bound at three times the mean bin power: rows leave at every
            # bin and some pass (below length 100)
            order = int(1.5 * L * power)
            want = np.zeros(n, dtype=np.uint8)
            oracle_lib.gpo_psd_filter_batch(seqs.ctypes.data, n, L, order, 0, want.ctypes.data, 4)
            got, st = ctx.psd_filter(seqs, order, 0, gp.GP_PSD_FP64)
            assert np.array_equal(got, want.astype(bool))
            assert st.n_pass == int(want.sum())
