"""Rows around the rules that send them to one kernel or another: folded or
hashed by products and distinct share, crowded folds, a few or many rows that
may leave the warp tables early, rows of many products on few columns."""
import numpy as np
import pytest

from oracle import oracle
from rtspmspm_b200 import DeviceCsr, Engine, gen

from helpers import assert_parity

pytestmark = pytest.mark.gpu

FOLD, HEAVY = 12, 10


def _csr(rows, cols, r, c, seed=0):
    rng = np.random.default_rng(seed)
    return gen.coo_to_csr(rows, cols, np.asarray(r), np.asarray(c), rng.uniform(-1, 1, len(r)).astype(np.float32))


def _rows_of(products, distinct, rows=40, spread=7):
    """Rows of `products` single-entry segments on `distinct` columns each."""
    rng = np.random.default_rng(products * 1000 + distinct)
    inner = 4 * products
    where = rng.choice(inner * spread, distinct, replace=False)
    owner = np.concatenate([np.arange(distinct), rng.integers(0, distinct, inner - distinct)])
    B = _csr(inner, inner * spread, np.arange(inner), where[owner], 1)
    c = []
    for _ in range(rows):
        first = np.arange(distinct)
        c.append(np.sort(np.concatenate([first, distinct + rng.choice(inner - distinct, products - distinct,
                                                                      replace=False)])))
    return _csr(rows, inner, np.repeat(np.arange(rows), products), np.concatenate(c), 2), B


def _share_limit(p):
    """Fewest distinct columns of a folded row of p products."""
    return p if p < 48 else -(-p * (256 - p) // 256) if p < 128 else (p + 1) // 2


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


@pytest.mark.parametrize("products", [31, 32, 47, 48, 64, 127, 128, 129, 320])
@pytest.mark.parametrize("off", [-1, 0])
def test_folded_by_share(products, off):
    distinct = min(products, _share_limit(products)) + off
    A, B = _rows_of(products, distinct)
    with Engine(0) as eng:
        rep, _ = _all_ways(eng, A, B, oracle.spgemm(A, B))
        assert rep["bin_rows"][FOLD] == (A.rows if off == 0 and products >= 32 else 0)
        dA, dB = DeviceCsr.from_host(A), DeviceCsr.from_host(B)
        for algo in ("plain", "learned"):
            for C in eng.multiply_batched([dA, dA], [dB, dB], algo=algo)[0]:
                assert_parity(C.to_host(), oracle.spgemm(A, B))


@pytest.mark.parametrize("products", [66, 320, 1152, 2048, 4010])
@pytest.mark.parametrize("many", [8, 700])
def test_crowded_folds(products, many):
    """Columns in one run and one far away: nearly all in one bucket."""
    rng = np.random.default_rng(products)
    inner = products + 200
    col = np.concatenate([np.arange(inner - 1), [5000000]])
    B = _csr(inner, 5000001, np.arange(inner), rng.permutation(col), 3)
    c = np.concatenate([np.sort(np.append(rng.choice(inner - 1, products - 1, replace=False), inner - 1))
                        for _ in range(many)])
    A = _csr(many, inner, np.repeat(np.arange(many), products), c, 4)
    with Engine(0) as eng:
        _all_ways(eng, A, B, oracle.spgemm(A, B))


@pytest.mark.parametrize("early,others,heavy", [(255, 0, False), (256, 0, True), (20, 1, True), (0, 30, True)])
def test_rows_that_may_leave_the_tables_early(early, others, heavy):
    """`early` rows of some 600 entries (short rows of B, so no bitmap of their
    span) beside `others` of some 1,500 and small ones."""
    rng = np.random.default_rng(early + others)
    sizes = np.array([70] * early + [190] * others + [4] * 300)
    rows, inner, cols = sizes.size, 3000, 60000
    r = np.repeat(np.arange(rows), sizes)
    A = _csr(rows, inner, r, np.concatenate([rng.choice(inner, n, replace=False) for n in sizes]), 5)
    B = _csr(inner, cols, np.repeat(np.arange(inner), 9), rng.integers(0, cols, inner * 9), 6)
    with Engine(0) as eng:
        rep, reuse = _all_ways(eng, A, B, oracle.spgemm(A, B), esc_min_prod=-1)
        want = early + others if heavy else 0
        assert rep["rows_heavy"] == want and reuse["rows_heavy"] == want
        assert sum(rep["bin_rows"][:8]) + rep["bin_rows"][HEAVY] == np.count_nonzero(sizes)


def test_rows_of_many_products_on_few_columns_stay():
    """Bounds past 512, some 300 columns each: counted and added in the tables."""
    rng = np.random.default_rng(9)
    rows, inner, cols = 600, 2000, 60000
    base = rng.integers(0, inner - 100, rows)
    A = _csr(rows, inner, np.repeat(np.arange(rows), 60), (base[:, None] + np.arange(60)).ravel(), 7)
    bc = (np.repeat(np.arange(inner), 12) * 5 + rng.integers(0, 60, inner * 12))
    B = _csr(inner, cols, np.repeat(np.arange(inner), 12), bc, 8)
    with Engine(0) as eng:
        rep, _ = _all_ways(eng, A, B, oracle.spgemm(A, B))
        assert rep["rows_heavy"] == 0
