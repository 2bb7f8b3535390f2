"""One context per host thread: products of different widths at once, whose
symbolic kernels ask for different amounts of shared memory."""
import threading

import numpy as np
import pytest

from oracle import oracle
from rtspmspm_b200 import DeviceCsr, Engine, gen

from helpers import assert_parity

pytestmark = pytest.mark.gpu


def _banded(cols, width, rows=96, per=40, k=30):
    """Rows of k x per products over `width` neighbouring columns."""
    rng = np.random.default_rng(width + cols)
    A = gen.coo_to_csr(rows, rows, np.repeat(np.arange(rows), k), rng.integers(0, rows, rows * k),
                       rng.uniform(-1, 1, rows * k).astype(np.float32))
    B = gen.coo_to_csr(rows, cols, np.repeat(np.arange(rows), per), rng.integers(0, width, rows * per),
                       rng.uniform(-1, 1, rows * per).astype(np.float32))
    return A, B


# (columns, columns in use) of the threads' products: spans of the three bitmap
# sizes; CTA bitmaps under and over the width that changes their thread count
@pytest.mark.parametrize("widths,per,k", [
    (((70000, 4000), (70000, 30000), (70000, 60000)), 40, 30),
    (((100000, 100000), (390000, 390000)), 120, 40),
    (((400000, 400000), (1300000, 1300000)), 120, 40)])
def test_threads_with_products_of_other_widths(widths, per, k):
    pairs = [_banded(c, w, per=per, k=k) for c, w in widths]
    refs = [oracle.spgemm(a, b) for a, b in pairs]
    errors = []
    gate = threading.Barrier(len(pairs))

    def work(i):
        try:
            with Engine(0) as eng:
                eng.set_tuning(small_rows=-1)
                dA, dB = (DeviceCsr.from_host(m) for m in pairs[i])
                gate.wait(60)
                for n in range(300):
                    C, _ = eng.multiply(dA, dB, algo="plain", skip_validation=True, use_tuning=True)
                    if n % 50 == 0:
                        assert_parity(C.to_host(), refs[i])
                    else:
                        assert C.nnz == refs[i].row_ptr[-1]
                    C.free()
        except BaseException as e:  # noqa: BLE001 - reported by the test
            errors.append((widths[i], repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(pairs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(300)
    assert not errors, errors
