"""Which rows spg_report.bin_rows counts under which index."""
import numpy as np
import pytest

from rtspmspm_b200 import Engine, gen

pytestmark = pytest.mark.gpu

HEAVY, EMPTY, FOLD = 10, 11, 12


def test_bin_rows():
    """7 empty rows, 5 of 4,000 entries, 20 of 100 distinct products, 30 of 8
    entries from 16 products."""
    rng = np.random.default_rng(0)
    cols = 5000
    # B: rows 0 to 9 of 4,000 columns, 10 to 19 of 10, 20 and 21 the same 8
    n = np.array([4000] * 10 + [10] * 10 + [8, 8])
    bc = [rng.choice(cols, 4000, replace=False) for _ in range(10)]
    bc += [np.arange(10) + 450 * i for i in range(10)] + [np.arange(8) * 100] * 2
    B = gen.coo_to_csr(22, cols, np.repeat(np.arange(22), n), np.concatenate(bc),
                       rng.uniform(-1, 1, n.sum()).astype(np.float32))
    per = [[]] * 7 + [[i] for i in range(5)] + [list(range(10, 20))] * 20 + [[20, 21]] * 30
    A = gen.coo_to_csr(62, 22, np.repeat(np.arange(62), [len(p) for p in per]), np.concatenate(per).astype(int),
                       rng.uniform(-1, 1, sum(len(p) for p in per)).astype(np.float32))
    with Engine(0) as eng:
        eng.set_tuning(small_rows=-1)
        C, rep = eng.multiply(A, B, algo="plain", use_tuning=True)
        C.free()
        bins = rep["bin_rows"]
        assert rep["rows_heavy"] == 5
        assert (bins[HEAVY], bins[EMPTY], bins[FOLD], sum(bins[:8])) == (5, 7, 20, 30)
        assert sum(bins) == A.rows
        # folding off: those rows are hashed
        eng.set_tuning(esc_min_prod=-1)
        C, rep = eng.multiply(A, B, algo="plain", use_tuning=True)
        C.free()
        bins = rep["bin_rows"]
        assert (bins[HEAVY], bins[EMPTY], bins[FOLD], sum(bins[:8])) == (5, 7, 0, 50)
