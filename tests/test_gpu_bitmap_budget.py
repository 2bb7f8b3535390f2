"""Rows that leave the warp tables early (past 512 entries) and the stored
bitmaps they need: rows on both sides of the limit, more rows than the bitmaps'
budget holds, columns past which no row leaves early, and bitmaps given back
when C needs their memory."""
import ctypes

import numpy as np
import pytest

from oracle import oracle
from rtspmspm_b200 import DeviceCsr, Engine, gen

from helpers import assert_parity

pytestmark = pytest.mark.gpu

COLS = 70000  # spans more words than the bitmaps of narrow spans hold


def _pair(rows, entries, inner=24, per=90, distinct=1800):
    """`entries` rows of B a row of A, B's rows of `per` of `distinct` columns
    spread over COLS: many products share a column, so none of the rows is
    folded past 1,152 products."""
    rng = np.random.default_rng(entries)
    A = gen.coo_to_csr(rows, inner, np.repeat(np.arange(rows), entries),
                       np.concatenate([rng.choice(inner, entries, replace=False) for _ in range(rows)]),
                       rng.uniform(-1, 1, rows * entries).astype(np.float32))
    where = np.arange(distinct) * (COLS // distinct)
    B = gen.coo_to_csr(inner, COLS, np.repeat(np.arange(inner), per),
                       np.concatenate([rng.choice(where, per, replace=False) for _ in range(inner)]),
                       rng.uniform(-1, 1, inner * per).astype(np.float32))
    return A, B


@pytest.mark.parametrize("entries,heavy", [(6, False), (20, True)])
def test_rows_on_both_sides_of_the_limit(entries, heavy):
    A, B = _pair(300, entries)
    R = oracle.spgemm(A, B)
    longest = int(np.diff(R.row_ptr).max())
    assert (longest > 512) == heavy and longest < 2048
    with Engine(0) as eng:
        eng.set_tuning(small_rows=-1)
        for kw in (dict(algo="plain"), dict(algo="learned", force_overflow=True)):
            C, rep = eng.multiply(A, B, use_tuning=True, **kw)
            assert rep["rows_heavy"] == (A.rows if heavy else 0) and rep["device_flags"] == 0
            assert_parity(C.to_host(), R)
        rep = eng.multiply_reuse(A, B, C)
        assert rep["rows_heavy"] == (A.rows if heavy else 0)
        assert_parity(C.to_host(), R)
        C.free()


def _columns(C):
    import torch

    out = []
    for p, t in ((C.s.col_idx, "<i4"), (C.s.val, "<f4")):
        class Raw:
            __cuda_array_interface__ = dict(shape=(C.nnz,), typestr=t,
                                            data=(ctypes.cast(p, ctypes.c_void_p).value, False), version=3)

        out.append(torch.as_tensor(Raw(), device="cuda"))
    return out


@pytest.mark.parametrize("esc", [0, -1])
def test_more_early_rows_than_the_bitmaps_hold(esc):
    """1,000,000 rows of 560 entries: bitmaps of 8,960 bytes a row pass the 8 GB
    set aside for them, and the rows go back to the folds and tables."""
    import torch

    rows, inner, per = 1000000, 50, 560
    rng = np.random.default_rng(1)
    B = gen.coo_to_csr(inner, COLS, np.repeat(np.arange(inner), per),
                       np.concatenate([rng.choice(COLS, per, replace=False) for _ in range(inner)]),
                       rng.uniform(-1, 1, inner * per).astype(np.float32))
    pick = rng.integers(0, inner, rows).astype(np.int32)
    A = gen.Csr(rows, inner, np.arange(rows + 1, dtype=np.int64), pick, np.full(rows, 2.0, np.float32))
    with Engine(0) as eng:
        eng.set_tuning(esc_min_prod=esc)
        C, rep = eng.multiply(DeviceCsr.from_host(A), DeviceCsr.from_host(B), algo="plain", use_tuning=True)
        assert rep["rows_heavy"] == 0 and rep["device_flags"] == 0 and C.nnz == rows * per
        col, val = _columns(C)
        bcol = torch.from_numpy(B.col_idx.reshape(inner, per)).cuda()
        bval = torch.from_numpy(2 * B.val.reshape(inner, per)).cuda()
        at = torch.from_numpy(pick.astype(np.int64)).cuda()
        for r in range(0, rows, 100000):
            part = slice(r * per, (r + 100000) * per)
            assert torch.equal(col[part].view(-1, per), bcol[at[r:r + 100000]])
            assert torch.equal(val[part].view(-1, per), bval[at[r:r + 100000]])
        C.free()


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


def _trim_default_pool():
    cu = ctypes.CDLL("libcuda.so.1")
    dev, pool = ctypes.c_int(), ctypes.c_void_p()
    assert cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), dev) == 0
    assert cu.cuMemPoolTrimTo(pool, ctypes.c_size_t(0)) == 0


def test_bitmaps_are_given_back_when_c_needs_their_memory():
    """A second call finds its bitmaps' 0.9 GB mapped and 0.6 GB of the device
    free: C (0.9 GB) fits only without them."""
    import torch

    A, B = _pair(1000, 20)
    rows = 100000
    A = gen.Csr(rows, A.cols, np.arange(rows + 1, dtype=np.int64) * 20, np.tile(A.col_idx, rows // 1000),
                np.tile(A.val, rows // 1000))
    dA, dB = DeviceCsr.from_host(A), DeviceCsr.from_host(B)
    with Engine(0) as eng:
        C, rep = eng.multiply(dA, dB, algo="plain", skip_validation=True)
        assert rep["rows_heavy"] == rows
        n = C.nnz
        assert 0.8e9 < 8 * n < 1.1e9
        want = [x[:: 1001].clone() for x in _columns(C)]
        C.free()
        torch.cuda.synchronize()
        _trim_default_pool()
        torch.cuda.empty_cache()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - (600 << 20), dtype=torch.uint8, device="cuda")
        try:
            C, rep = eng.multiply(dA, dB, algo="plain", skip_validation=True)
            assert C.nnz == n and rep["rows_heavy"] == rows and rep["device_flags"] == 0
            for x, y in zip(_columns(C), want):
                assert torch.equal(x[:: 1001].view(torch.int32), y.view(torch.int32))
            C.free()
        finally:
            del fill
            torch.cuda.empty_cache()
