"""cg_quadratic against the oracle over the edges of its matrix-vector product
(GPU): rows per block, vectors per row with and without a scalar tail, rows
shorter and longer than what is brought in ahead, unaligned rows (odd n).
The bars are those of the other parity tests of the solver, 1e-10 of the
largest entry, with the same number of iterations."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 31, 64, 511, 513, 1024, 2050, 2304])
def test_cg_sizes(n, ald_lib, oracle_lib):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n)) / np.sqrt(n)
    A = np.asfortranarray(G @ G.T + np.diag(np.geomspace(1.0, 20.0, n)))
    b, x0 = rng.standard_normal(n), 0.1 * rng.standard_normal(n)
    ref, fref = x0.copy(), C.c_double(0)
    p = lambda a: a.ctypes.data_as(oracle_lib.dp)  # noqa: E731
    it_ref = oracle_lib.lib().orc_cg(n, p(A), p(b), p(ref), C.byref(fref), 200, 4, 2)
    x, fm, it, st = ald_lib.cg_quadratic(A, b, x0, max_iter=200, n_dig_accur=4)
    assert st == 0 and it == it_ref
    assert np.abs(x - ref).max() <= 1e-10 * np.abs(ref).max()
    assert abs(fm - fref.value) <= 1e-10 * abs(fref.value)
