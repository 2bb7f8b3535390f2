"""Batched rows on both sides of the expand-sort-fold bins' product limits (the
learned method folds up to 1,152 products, the plain one up to 2,048), and
batches whose rows' bounds leave bins, or all of them, out."""
import numpy as np
import pytest

from oracle import oracle
from rtspmspm_b200 import DeviceCsr, Engine, gen

from helpers import assert_parity

pytestmark = pytest.mark.gpu


def _rows_of(products, cols=5000, inner=4096, seed=0):
    """Row i of A*B has products[i] products, all of distinct columns."""
    rng = np.random.default_rng(seed)
    B = gen.coo_to_csr(inner, cols, np.arange(inner), rng.choice(cols, inner, replace=False),
                       rng.uniform(-1, 1, inner).astype(np.float32))
    c = [np.sort(rng.choice(inner, n, replace=False)) for n in products]
    r = np.repeat(np.arange(len(products)), products)
    A = gen.coo_to_csr(len(products), inner, r, np.concatenate(c), rng.uniform(-1, 1, r.size).astype(np.float32))
    return A, B


@pytest.mark.parametrize("most", [15, 16, 33, 160, 161, 321, 577, 1153, 2049, 4096])
@pytest.mark.parametrize("algo", ["plain", "learned"])
def test_folds_by_products(algo, most):
    edges = [n + d for n in (16, 32, 320, 640, 1152, 2048, 4010) for d in (-1, 0, 1)] + [1, 4096]
    sizes = [n for n in edges if n <= most] + [most]
    pairs = [_rows_of(sizes * 3, seed=1), _rows_of(sizes[::-1], cols=4500, seed=2)]
    with Engine(0) as eng:
        As, Bs = ([DeviceCsr.from_host(m) for m in ms] for ms in zip(*pairs))
        for _ in range(2):  # captured, replayed
            Cs, rep = eng.multiply_batched(As, Bs, algo=algo, use_graph=True)
            assert rep["device_flags"] == 0 and rep["rows_heavy"] == 0
            for C, (A, B) in zip(Cs, pairs):
                assert_parity(C.to_host(), oracle.spgemm(A, B))


def test_bins_no_row_can_reach_are_not_launched():
    launches = []
    with Engine(0) as eng:
        for most in (15, 16, 161, 2000):
            A, B = _rows_of([most] * 5)
            _, rep = eng.multiply_batched([DeviceCsr.from_host(A)], [DeviceCsr.from_host(B)], algo="plain")
            launches.append(rep["kernel_launches"])
    assert np.diff(launches).tolist() == [1, 1, 2]
