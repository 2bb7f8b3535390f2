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
