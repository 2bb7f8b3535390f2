"""Value-only recompute with A and B whose structure is not the one C was
computed from: a row of another number of columns is refused wherever its new
columns lie, and what the recompute does not read (the columns that C holds,
for rows up to the warp tables' 2,048 entries) does not decide."""
import numpy as np
import pytest

from oracle import oracle
from rtspmspm_b200 import Engine, SpgError, gen

from helpers import assert_parity

pytestmark = pytest.mark.gpu

ROWS, INNER = 50, 40


def _pair(cols, where, per=400, extra=()):
    """A full; B's rows of `per` columns drawn from `where`, row 0 with the
    columns `extra` besides."""
    r = np.repeat(np.arange(ROWS), INNER)
    A = gen.coo_to_csr(ROWS, INNER, r, np.tile(np.arange(INNER), ROWS), np.linspace(-1, 1, r.size, dtype=np.float32))
    rng = np.random.default_rng(1)
    bc = np.concatenate([rng.choice(where, per, replace=False) for _ in range(INNER)] + [np.asarray(extra, int)])
    br = np.concatenate([np.repeat(np.arange(INNER), per), np.zeros(len(extra), int)])
    return A, gen.coo_to_csr(INNER, cols, br, bc, rng.uniform(-1, 1, br.size).astype(np.float32))


def _zero_columns(C):
    import ctypes

    import torch

    ptr = ctypes.cast(C.s.col_idx, ctypes.c_void_p).value

    class Raw:
        __cuda_array_interface__ = dict(shape=(C.nnz,), typestr="<i4", data=(ptr, False), version=3)

    torch.as_tensor(Raw(), device="cuda").zero_()
    torch.cuda.synchronize()


# C's columns: the first tiles, the last ones, and both ends with more empty
# tiles between than one unit of tiles spans
LOW, HIGH = np.arange(1200), np.arange(58800, 60000)
ENDS = np.concatenate([np.arange(600), np.arange(119400, 120000)])


@pytest.mark.parametrize("cols,where,extra", [
    (60000, LOW, [50000, 50001]), (60000, LOW, [59999]), (60000, HIGH, [3]), (60000, HIGH, [40000]),
    (120000, ENDS, [60000]), (120000, ENDS, [5000]), (120000, ENDS, [118000]), (60000, LOW, [1300])])
def test_columns_elsewhere_are_refused(cols, where, extra):
    A, B = _pair(cols, where)
    A2, B2 = _pair(cols, where, extra=extra)
    R = oracle.spgemm(A, B)
    with Engine(0) as eng:
        C, _ = eng.multiply(A, B, algo="plain")
        rep = eng.multiply_reuse(A, B, C)
        assert rep["rows_heavy"] == ROWS  # rows of 1,200 entries, in units
        with pytest.raises(SpgError) as e:
            eng.multiply_reuse(A2, B2, C)
        assert e.value.status == 1
        eng.multiply_reuse(A, B, C)
        assert_parity(C.to_host(), R)
        C.free()


def test_as_many_other_columns_are_accepted():
    A, B = _pair(60000, LOW)
    A2, B2 = _pair(60000, LOW + 30000)
    R2 = oracle.spgemm(A2, B2)
    with Engine(0) as eng:
        C, _ = eng.multiply(A, B, algo="plain")
        eng.multiply_reuse(A2, B2, C)
        assert_parity(C.to_host(), R2)
        C.free()


def test_columns_of_c_are_written_not_read():
    A, B = _pair(60000, LOW)
    R = oracle.spgemm(A, B)
    with Engine(0) as eng:
        C, _ = eng.multiply(A, B, algo="plain")
        _zero_columns(C)
        eng.multiply_reuse(A, B, C)
        assert_parity(C.to_host(), R)
        C.free()


def test_rows_past_the_tables_count_by_tile():
    """Rows of 4,000 entries: one column moved into a neighbouring tile, and a C
    that names one column 4,000 times."""
    where = np.arange(8000, 12000)
    A, B = _pair(60000, where, per=3000)
    other = where.copy()
    other[where == 10239] = 12001  # out of tile 4, into tile 5
    A2, B2 = _pair(60000, other, per=3000)
    R = oracle.spgemm(A, B)
    with Engine(0) as eng:
        C, _ = eng.multiply(A, B, algo="plain")
        assert C.nnz == ROWS * 4000
        with pytest.raises(SpgError) as e:
            eng.multiply_reuse(A2, B2, C)
        assert e.value.status == 1
        _zero_columns(C)
        with pytest.raises(SpgError) as e:
            eng.multiply_reuse(A, B, C)
        assert e.value.status == 1
        C.free()
        C, _ = eng.multiply(A, B, algo="plain")
        eng.multiply_reuse(A, B, C)
        assert_parity(C.to_host(), R)
        C.free()


def test_one_column_repeated_past_a_units_room():
    """A C of 8,000-entry rows that names one column throughout: refused."""
    where = np.arange(8000, 16000)
    A, B = _pair(60000, where, per=6000)
    with Engine(0) as eng:
        C, _ = eng.multiply(A, B, algo="plain")
        assert C.nnz == ROWS * 8000
        _zero_columns(C)
        with pytest.raises(SpgError) as e:
            eng.multiply_reuse(A, B, C)
        assert e.value.status == 1
        C.free()
