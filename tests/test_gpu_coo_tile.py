"""COO -> CSR of entries that fill about one tile of the sort, which then needs no
counts of its digits: single entries, a tile and one more, entries outside."""
import numpy as np
import pytest

from rtspmspm_b200 import Engine, SpgError

pytestmark = pytest.mark.gpu

@pytest.mark.parametrize("n", [1, 2, 511, 512, 4095, 4096, 4097])
def test_coo_of_about_one_tile(n):
    rng = np.random.default_rng(n)
    rows, cols = 300, 5
    r, c = rng.integers(0, rows, n).astype(np.int32), rng.integers(0, cols, n).astype(np.int32)
    v = rng.uniform(-1, 1, n).astype(np.float32)
    with Engine(0) as eng:
        C = eng.coo_to_csr(rows, cols, r, c, v)
        got = C.to_host()
        C.free()
        key = r.astype(np.int64) * cols + c
        order = np.argsort(key, kind="stable")
        at, first = np.unique(key[order], return_index=True)
        want = []
        for b, e in zip(first, list(first[1:]) + [n]):
            s = v[order[b]]
            for i in order[b + 1:e]:
                s = np.float32(s + v[i])
            want.append(s)
        np.testing.assert_array_equal(np.asarray(got.row_ptr),
                                      np.searchsorted(at, np.arange(rows + 1, dtype=np.int64) * cols))
        np.testing.assert_array_equal(np.asarray(got.col_idx), at % cols)
        np.testing.assert_array_equal(got.val.view(np.uint32), np.array(want, np.float32).view(np.uint32))
        for bad in ((rows, 0), (-1, 0), (0, cols), (0, -1)):
            r2, c2 = r.copy(), c.copy()
            r2[n // 2], c2[n // 2] = bad
            with pytest.raises(SpgError):
                eng.coo_to_csr(rows, cols, r2, c2, v)
