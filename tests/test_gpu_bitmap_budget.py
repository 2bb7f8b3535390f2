"""Rows that leave the warp tables early (past 512 entries) and the stored
bitmaps they need."""
import numpy as np
import pytest

from oracle import oracle
from rtspmspm_b200 import DeviceCsr, Engine, gen

from helpers import assert_parity

pytestmark = pytest.mark.gpu

def test_no_second_binning_where_no_row_leaves_early():
    """Past 262,144 columns the limit does not matter, so a call without stored
    bitmaps (past 1,310,720) launches no more than one whose tables end at it."""
    rows, per, cols = 300, 1100, 1400000
    rng = np.random.default_rng(0)
    B = gen.coo_to_csr(64, cols, np.repeat(np.arange(64), per), rng.integers(0, cols, 64 * per),
                       np.ones(64 * per, np.float32))
    A = gen.coo_to_csr(rows, 64, np.repeat(np.arange(rows), 2), np.arange(2 * rows) % 64, np.ones(2 * rows, np.float32))
    R = oracle.spgemm(A, B)
    launches = []
    with Engine(0) as eng:
        for table in (4096, 1024):
            eng.set_tuning(small_rows=-1, warp_table_max=table)
            C, rep = eng.multiply(A, B, algo="plain", use_tuning=True)
            assert rep["rows_heavy"] == rows
            assert_parity(C.to_host(), R)
            launches.append(rep["kernel_launches"])
            C.free()
    assert launches[0] == launches[1]
