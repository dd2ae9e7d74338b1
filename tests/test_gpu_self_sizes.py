"""The self-energy's pairs per CTA and the small eigensolver's matrices per
warp at their edges, against the oracle (GPU).

self_energy: meshes whose points do not fill the last CTA, 3, 6 and 12 bands
(32, 4 and fewer pairs to a CTA), at q off every symmetry; the bars of the
self-energy parity tests (1e-8 of a value, 1e-9 of the largest).
Phonons: enough matrices for the wider packing with a remainder in the last
warp; the bars of the phonon parity tests."""
import numpy as np
import pytest

from conftest import make_case
from test_gpu_large import _check_phonons
from test_gpu_self import CL, H, KB, close, grouped

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg,mesh,kw", [
    (0, (3, 3, 3), {}), (0, (5, 5, 5), {}), (1, (3, 3, 3), {}), (1, (5, 5, 5), {}),
    (3, (3, 3, 3), {"p": 1, "rc_sigma": 1.2, "delta": "gauss"})])
@pytest.mark.parametrize("gauss", [False, True])
def test_self_energy_remainders(cfg, mesh, kw, gauss, oracle_lib, ald_lib, workdir):
    d = make_case(workdir, cfg, mesh, **kw)
    O = oracle_lib.Oracle(d)
    O.mesh()
    O.phonons()
    q = np.array([[0.137, 0.291], [0.053, -0.172], [0.211, 0.083]])
    ev, _ = O.frequencies_at(q)
    om0 = np.sqrt(np.abs(ev)) * O.lattice()["cnst"]
    n, temp = O.ndyn, 300.0 * KB / (100 * H * CL)
    qs, las, oms = np.repeat(q, n, axis=1), np.tile(np.arange(1, n + 1), 2), om0.T.ravel()
    ref = O.self_w(qs, las, oms, temp, gauss=gauss)
    with ald_lib.Context(d) as ctx:
        ctx.set_phonons(*O.get_phonons())
        got = ctx.function_self_w(qs, las, oms, temp, gauss=gauss)
    for g, r in zip(got, ref):
        for comp in (np.real, np.imag):
            G = np.concatenate([grouped(comp(g)[p * n:(p + 1) * n], om0[:, p], 0.0) for p in range(2)])
            R = np.concatenate([grouped(comp(r)[p * n:(p + 1) * n], om0[:, p], 0.0) for p in range(2)])
            ok, worst = close(G, R)
            assert ok, worst


@pytest.mark.parametrize("cfg,mesh", [(0, (14, 14, 14)), (1, (13, 13, 13))])
def test_phonons_many(cfg, mesh, oracle_lib, ald_lib, workdir):
    d = make_case(workdir, cfg, mesh)
    O = oracle_lib.Oracle(d)
    O.mesh()
    O.phonons()
    with ald_lib.Context(d) as ctx:
        _check_phonons(O, O.get_phonons(), ctx.get_frequencies())
