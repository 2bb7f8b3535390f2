"""Heavy rows whose rows of B are mostly short, and new values into a C whose
columns the heavy rows take as they are."""
import numpy as np
import pytest

from oracle import oracle
from rtspmspm_b200 import Engine, gen

from helpers import assert_parity

pytestmark = pytest.mark.gpu

def _csr(rows, cols, r, c, seed=0):
    rng = np.random.default_rng(seed)
    return gen.coo_to_csr(rows, cols, np.asarray(r), np.asarray(c), rng.uniform(-1, 1, len(r)).astype(np.float32))


def _all_ways(eng, A, B, want, **tuning):
    """Plain, learned and new values of A*B, each with the oracle's bits; the
    plain call's report."""
    eng.set_tuning(small_rows=-1, **tuning)
    C, rep = eng.multiply(A, B, algo="learned", use_tuning=True)
    assert_parity(C.to_host(), want)
    C.free()
    C, rep = eng.multiply(A, B, algo="plain", use_tuning=True)
    assert rep["device_flags"] == 0
    assert_parity(C.to_host(), want)
    reuse = eng.multiply_reuse(A, B, C, use_tuning=True)
    assert_parity(C.to_host(), want)
    C.free()
    return rep, reuse


@pytest.mark.parametrize("cols", [9000, 70000])
@pytest.mark.parametrize("long_every", [0, 5, 40])
def test_heavy_rows_of_small_segments(cols, long_every):
    """Rows of B of 0 to 9 entries, every long_every-th of 33, 129 or 700: runs
    of small segments on the same columns, broken by longer ones."""
    rng = np.random.default_rng(cols + long_every)
    inner, rows = 5000, 12
    size = rng.integers(0, 10, inner)
    if long_every:
        size[::long_every] = rng.choice([33, 129, 700], size[::long_every].size)
    hot = rng.choice(cols, cols // 3, replace=False)
    bc = np.concatenate([rng.choice(hot, n, replace=False) for n in size])
    B = _csr(inner, cols, np.repeat(np.arange(inner), size), bc, 10)
    per = np.array([5000, 4000, 3001, 1500, 700, 640, 129, 128, 127, 33, 32, 1])
    A = _csr(rows, inner, np.repeat(np.arange(rows), per),
             np.concatenate([rng.choice(inner, n, replace=False) for n in per]), 11)
    with Engine(0) as eng:
        rep, reuse = _all_ways(eng, A, B, oracle.spgemm(A, B))
        assert rep["rows_heavy"] > 0 and reuse["rows_heavy"] > 0


@pytest.mark.parametrize("value", [-0.0, 0.0, np.inf, -np.inf, np.nan])
def test_new_values_of_heavy_rows_with_special_values(value):
    """Every accumulator is told from one without a product by its bits alone."""
    rng = np.random.default_rng(3)
    inner, cols = 300, 50000
    B = _csr(inner, cols, np.repeat(np.arange(inner), 20), rng.integers(0, cols, inner * 20), 12)
    A = _csr(3, inner, np.repeat(np.arange(3), inner), np.tile(np.arange(inner), 3), 13)
    with Engine(0) as eng:
        C, rep = eng.multiply(A, B, algo="plain")
        assert rep["rows_heavy"] == 3
        B.val[::3] = value
        A.val[: inner // 2] = 1.0
        fresh, _ = eng.multiply(A, B, algo="plain")
        want = fresh.to_host()
        eng.multiply_reuse(A, B, C)
        got = C.to_host()
        np.testing.assert_array_equal(np.asarray(got.col_idx), np.asarray(want.col_idx))
        np.testing.assert_array_equal(got.val.view(np.uint32), want.val.view(np.uint32))
        fresh.free()
        C.free()
