"""The conjugate-gradient kernels of one graph overlap: a kernel's blocks are
resident before the kernel in front of it has ended.  What a kernel of the
chain writes may then only be read with ordinary loads after the wait, never
through the read-only path (__ldg, or a const __restrict__ parameter that lets
the compiler choose it), whose data nobody may write while the kernel lives."""
import os
import re

import numpy as np
import pytest

from conftest import ROOT

CHAIN = {  # what the kernels of an iteration write, by parameter
    "gemv_kernel": ("x", "g", "st"),
    "cg_update_kernel": ("aux", "pden", "pnum", "grad", "conj", "v0", "x", "st"),
    "cg_dir_kernel": ("p4", "grad", "conj", "st"),
}


@pytest.mark.parametrize("kernel", sorted(CHAIN))
def test_written_data_is_not_read_only(kernel):
    src = open(os.path.join(ROOT, "anharmonic-lattice-dynamics_b200", "csrc", "ald_bte.cu")).read()
    m = re.search(r"__global__[^;{]*?\b%s\(([^{]*?)\)\s*\{(.*?)\n}\n" % kernel, src, re.S)
    args, body = " ".join(m.group(1).split()), m.group(2)
    names = set(CHAIN[kernel])
    for name in CHAIN[kernel]:
        assert re.search(r"\*\s*%s(,|$)" % name, args), name
        names.update(re.findall(r"(\w+) = reinterpret_cast<const \w+\*>\(%s\)" % name, body))
    for name in names:  # aliases of them too
        assert not re.search(r"(__ldg|ld\.global\.nc)\(?\s*\(?%s\b" % name, body), name
    before, after = body.split("pdl_wait();")
    assert not any(re.search(r"\b%s(\[|->)" % n, before) for n in names)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [513, 2304, 4800])
def test_repeated_solves(n, ald_lib):
    """The same system between solves of another one: the same bits each time, and A x = b to what the stop rule
    leaves: last step below 1e-8 of x, eigenvalues in 1..24 (rate 0.66 a step), so the error is below 3e-8 |x| <= 3e-8
    |b| and the residual below 24 times that; the bar is 1e-5."""
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n)) / np.sqrt(n)
    A = np.asfortranarray(G @ G.T + np.diag(np.geomspace(1.0, 20.0, n)))
    b, x0 = rng.standard_normal(n), 0.1 * rng.standard_normal(n)
    first = ald_lib.cg_quadratic(A, b, x0, max_iter=200, n_dig_accur=8)
    assert np.linalg.norm(A @ first[0] - b) <= 1e-5 * np.linalg.norm(b)
    for k in range(6):
        ald_lib.cg_quadratic(A, rng.standard_normal(n), x0, max_iter=200, n_dig_accur=8)
        x, fm, it, st = ald_lib.cg_quadratic(A, b, x0, max_iter=200, n_dig_accur=8)
        assert np.array_equal(x, first[0]) and (fm, it, st) == first[1:]
