"""Work memory kept between calls goes back to the device on request."""
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
