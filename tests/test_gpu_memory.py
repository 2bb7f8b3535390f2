"""Work memory: what a call takes, and that what is kept between calls goes back
to the device on request."""
import numpy as np
import pytest

from rtspmspm_b200 import DeviceCsr, Engine, _lib, gen

pytestmark = pytest.mark.gpu


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_trim_memory_gives_work_memory_back():
    A = DeviceCsr.from_host(gen.stencil27(48))
    with Engine(0) as eng:
        eng.trim_memory()
        C, _ = eng.multiply(A, A, algo="learned")
        held = _free()
        eng.trim_memory()
        # the learned product's slab alone: 13 M entries of 8 bytes
        assert _free() - held > 100 << 20
        D, _ = eng.multiply(A, A, algo="learned")
        assert D.nnz == C.nnz
        C.free()
        D.free()
    # what stays when the last context is gone goes back too
    held = _free()
    L = _lib.load()
    assert L.spg_trim_memory(0) == _lib.SPG_OK
    assert _free() - held > 100 << 20
    assert L.spg_trim_memory(0) == _lib.SPG_OK
    assert L.spg_trim_memory(-1) == _lib.SPG_ERR_INVALID_ARG
    assert L.spg_trim_memory(1 << 20) == _lib.SPG_ERR_INVALID_ARG


def test_heavy_rows_take_one_word_a_tile():
    """40,000 heavy rows over 684 column tiles (past the width of the stored
    bitmaps): their tile counts are 109 MB, the rest of the call's work memory
    some 30 MB."""
    rows, per, cols = 40000, 1100, 1400000
    rng = np.random.default_rng(0)
    b = np.sort(rng.integers(0, cols, (64, per)), axis=1)
    B = gen.coo_to_csr(64, cols, np.repeat(np.arange(64), per), b.ravel(), np.ones(64 * per, np.float32))
    A = gen.coo_to_csr(rows, 64, np.repeat(np.arange(rows), 2), np.arange(2 * rows) % 64,
                       np.ones(2 * rows, np.float32))
    with Engine(0) as eng:
        dA, dB = DeviceCsr.from_host(A), DeviceCsr.from_host(B)
        eng.trim_memory()
        C, rep = eng.multiply(dA, dB, algo="plain", skip_validation=True)
        assert rep["rows_heavy"] == rows
        held = _free()
        eng.trim_memory()
        took = _free() - held
        assert (100 << 20) < took < (200 << 20), took
        C.free()
