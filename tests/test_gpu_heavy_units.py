"""Heavy rows in units of consecutive column tiles, against the oracle: rows
cut into many units, tile counts past one 32-tile scan, empty tiles at the
ends and inside, both symbolic CTA sizes (up to and past 393,216 columns),
rows wider than one bitmap window (1,310,720 columns: no stored bitmaps), and
the value-only recompute, whose units find their columns themselves."""
import numpy as np
import pytest

from oracle import oracle
from rtspmspm_b200 import DeviceCsr, Engine, gen

from helpers import assert_parity

pytestmark = pytest.mark.gpu


def _pair(cols):
    """A: one full row and rows of 150 entries; B: rows of mixed lengths whose
    columns leave a band of the tiles empty."""
    rng = np.random.default_rng(cols)
    inner = 1500
    r = np.concatenate([np.zeros(inner, np.int64), np.repeat(np.arange(1, 40), 150)])
    c = np.concatenate([np.arange(inner), *[rng.choice(inner, 150, replace=False) for _ in range(39)]])
    A = gen.coo_to_csr(40, inner, r, c, rng.uniform(-1, 1, r.size).astype(np.float32))
    n = np.where(np.arange(inner) % 7 == 0, 700, rng.integers(0, 60, inner))
    br = np.repeat(np.arange(inner), n)
    bc = rng.integers(0, cols, br.size)
    keep = ~((bc > cols // 3) & (bc < cols // 2))  # empty tiles inside
    br, bc = br[keep], bc[keep]
    return A, gen.coo_to_csr(inner, cols, br, bc, rng.uniform(-1, 1, br.size).astype(np.float32))


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("cols", [4099, 33 * 2048 + 5, 393216, 393217, 1400000])
def test_heavy_units(cols, bits):
    A, B = _pair(cols)
    R = oracle.spgemm(A, B)
    with Engine(0) as eng:
        dA, dB = DeviceCsr.from_host(A, index_bits=bits), DeviceCsr.from_host(B, index_bits=bits)
        for algo in ("plain", "learned"):
            eng.set_tuning(small_rows=-1)
            C, rep = eng.multiply(dA, dB, algo=algo, use_tuning=True)
            assert rep["rows_heavy"] > 0 and rep["device_flags"] == 0
            assert_parity(C.to_host(), R)
        A2 = gen.Csr(A.rows, A.cols, A.row_ptr, A.col_idx, -A.val[::-1].copy())
        rep = eng.multiply_reuse(DeviceCsr.from_host(A2, index_bits=bits), dB, C)
        assert rep["rows_heavy"] > 0
        assert_parity(C.to_host(), oracle.spgemm(A2, B))
        C.free()


@pytest.mark.parametrize("entries", [9, 12, 20, 36])
def test_rows_leaving_the_warp_tables_early(entries):
    """540 to 2,160 products a row over 1,800 columns: 470 to 1,260 output
    entries, on both sides of the 512 past which rows go to the units and of
    the products up to which they are folded."""
    rng = np.random.default_rng(entries)
    A = gen.coo_to_csr(60, 90, np.repeat(np.arange(60), entries),
                       np.concatenate([rng.choice(90, entries, replace=False) for _ in range(60)]),
                       rng.uniform(-1, 1, 60 * entries).astype(np.float32))
    B = gen.coo_to_csr(90, 1800, np.repeat(np.arange(90), 60),
                       np.concatenate([rng.choice(1800, 60, replace=False) for _ in range(90)]),
                       rng.uniform(-1, 1, 90 * 60).astype(np.float32))
    R = oracle.spgemm(A, B)
    with Engine(0) as eng:
        eng.set_tuning(small_rows=-1)
        for algo in ("plain", "learned"):
            C, rep = eng.multiply(A, B, algo=algo, use_tuning=True)
            assert rep["device_flags"] == 0
            assert_parity(C.to_host(), R)
        eng.multiply_reuse(A, B, C)
        assert_parity(C.to_host(), R)
        C.free()
