"""Symbolic span bitmaps and expand-sort-fold bins of the plain method against
the oracle: spans at and past the bitmap classes' word counts (rows past the
last are hashed), products around the fold's bins, a bucket crowded past the
fold's limit, and rows of A longer than a warp."""
import numpy as np
import pytest

from oracle import oracle
from rtspmspm_b200 import DeviceCsr, Engine, gen

from helpers import assert_parity

pytestmark = pytest.mark.gpu


def _check(A, B):
    R = oracle.spgemm(A, B)
    with Engine(0) as eng:
        eng.set_tuning(small_rows=-1)
        for bits in (32, 64):
            dA, dB = DeviceCsr.from_host(A, index_bits=bits), DeviceCsr.from_host(B, index_bits=bits)
            for algo in ("plain", "learned"):
                C, rep = eng.multiply(dA, dB, algo=algo, use_tuning=True)
                assert rep["device_flags"] == 0
                assert_parity(C.to_host(), R)
                C.free()
            assert np.array_equal(eng.row_nnz(dA, dB).cpu().numpy(), np.diff(R.row_ptr))


def _rows(rows, cols, per_row, rng, ends=False):
    r = np.repeat(np.arange(rows), per_row)
    c = np.concatenate([rng.choice(cols, per_row, replace=False) for _ in range(rows)])
    if ends:  # every row reaches the first and the last column
        r = np.concatenate([r, np.repeat(np.arange(rows), 2)])
        c = np.concatenate([c, np.tile([0, cols - 1], rows)])
    return gen.coo_to_csr(rows, cols, r, c, rng.uniform(-1, 1, r.size).astype(np.float32))


@pytest.mark.parametrize("cols", [40, 576 * 32, 576 * 32 + 1, 1216 * 32, 1216 * 32 + 1, 2048 * 32, 2048 * 32 + 1])
@pytest.mark.parametrize("entries", [24, 40])
def test_span_classes(cols, entries):
    rng = np.random.default_rng(cols + entries)
    _check(_rows(60, 200, entries, rng), _rows(200, cols, min(24, cols), rng, ends=True))


@pytest.mark.parametrize("entries", [13, 16, 32, 33, 57, 58, 102, 103, 200])
def test_fold_bins(entries):
    """entries x 20 products a row: 260, 320 | 640, 660 | 1,140, 1,160 | 2,040,
    2,060 | 4,000, nearly all of distinct columns."""
    rng = np.random.default_rng(entries)
    _check(_rows(50, 300, entries, rng), _rows(300, 60000, 20, rng))


def test_fold_crowded_bucket():
    """Most of a row's columns in a few of its span's 256 ranges: sorted whole."""
    rng = np.random.default_rng(5)
    B = _rows(300, 700, 20, rng)
    c = B.col_idx.astype(np.int64)
    c[B.row_ptr[1:] - 1] = 100000 + np.arange(300)  # one far column a row stretches the span
    B = gen.coo_to_csr(300, 100300, np.repeat(np.arange(300), B.row_lengths()), c, B.val)
    _check(_rows(50, 300, 30, rng), B)
