"""|V3|^2 of cells of 9 to 36 bands formed in shared memory (ald_v3_tile.cu) and
the Gaussian delta that walks l3 (GPU), against the factorised oracle and the
per-stage kernels.

Random unit eigenvectors and eigenvalues are injected, so no entry is 0/0.  The
cells are rows of n atoms (3 n bands): n = 3, 5, 7, 9 leave remainders in the
3 x 3 and 4 x 4 register tiles and in the steps over l1, n = 4, 8, 12 do not;
27 mesh points leave a remainder in the tiles of 4 and 2 points.  FP64: the
bars of test_gpu_parity.py; mixed: FP32 products of unit vectors, 1e-5 normwise.
The pipeline's linewidths against V3 -> FGR -> tau of the per-stage entry points:
the same terms with the products regrouped, 1e-12 of each sum of positive terms.
"""
import os

import numpy as np
import pytest

import oracle_dense
from test_gpu_parity import close

pytestmark = pytest.mark.gpu


def chain(workdir, n, mesh):
    """n atoms along x of a simple-cubic Lennard-Jones lattice, random masses."""
    from ald import inputs as I
    a = 3.9
    rng = np.random.default_rng(n)
    st = I.Structure(
        name="chain-%d" % n, conv_abc=(float(n), 1.0, 1.0), prim_in_conv=np.eye(3), lattice_parameter=a,
        atom_types=[1] * n, atom_red_conv=[(k / n, 0.0, 0.0) for k in range(n)], type_masses=[40.0],
        type_names=["Ar"], pairs=[(1, 1, 0.1, 1.05 * a, I.lennard_jones(0.0104, 3.4))],
        atom_masses=[float(m) for m in rng.uniform(20.0, 80.0, n)])
    d = os.path.join(str(workdir), "chain%d_%s" % (n, "x".join(map(str, mesh))))
    if not os.path.exists(d):
        I.write_inputs(st, I.RunParams(mesh=mesh, delta="gauss", width_cm=40.0), d)
    return d


def random_phonons(nk, b, seed):
    rng = np.random.default_rng(seed)
    z = rng.normal(size=(nk, b, b)) + 1j * rng.normal(size=(nk, b, b))
    vec = np.linalg.qr(z)[0].transpose(1, 2, 0)
    return (np.asfortranarray(np.sort(rng.uniform(0.01, 0.2, (b, nk)), axis=0)), np.asfortranarray(vec),
            np.asfortranarray(rng.normal(size=(3, b, nk)) * 1e-5))


class Injected:
    """The oracle with other eigenpairs."""

    def __init__(self, O, ph):
        self.O, self.ph = O, ph

    def __getattr__(self, k):
        return getattr(self.O, k)

    def get_phonons(self):
        return self.ph


@pytest.mark.parametrize("n", [3, 4, 5, 7, 8, 9, 12])
def test_tile_v3(oracle_lib, ald_lib, workdir, n):
    d = chain(workdir, n, (3, 3, 3))
    O = oracle_lib.Oracle(d)
    O.mesh()
    O.phonons()
    O.tet()
    ph = random_phonons(O.nkc, O.ndyn, n)
    row = (2, 2)
    q2s = np.array([0, 5, 22, 23, 24, 26])  # the first tile, the last ones
    ref = oracle_dense.v3_factorised(Injected(O, ph), *row, q2s=q2s)[:, q2s]
    for prec in (ald_lib.FP64, ald_lib.MIXED):
        with ald_lib.Context(d, ald_lib.default_options(precision=prec, delta=ald_lib.DELTA_GAUSS)) as ctx:
            ctx.set_phonons(*ph)
            v = ctx.calculate_w3_ibz_split_sq(list(row))[:, q2s]
        if prec == ald_lib.FP64:
            ok, worst = close(v, ref)
            assert ok, worst
        else:
            assert np.linalg.norm(v - ref) <= 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 6])
def test_gauss_walking_l3(ald_lib, workdir, n, prec):
    d = chain(workdir, n, (3, 3, 3))
    P = ald_lib.FP64 if prec == "fp64" else ald_lib.MIXED
    with ald_lib.Context(d, ald_lib.default_options(precision=P, delta=ald_lib.DELTA_GAUSS)) as ctx:
        ctx.set_phonons(*random_phonons(ctx.nkc, ctx.ndyn, n))
        out = ctx.kappa_pipeline(300.0)
        rows = [1, ctx.nibz]
        v = ctx.calculate_w3_ibz_split_sq(rows)
        P1, P2 = ctx.calculate_fgr(rows, v)
        ctx.distribution(300.0)
        Q, QN, QU, _, _ = ctx.calculate_tau_rta(rows, 300.0, P1, P2, want_p=False)
    tol = 1e-12 if prec == "fp64" else 1e-6  # mixed: FP32 |V3|^2 and weights in the pipeline
    for a, r in ((out["Q"], Q), (out["QN"], QN), (out["QU"], QU)):
        assert np.all(np.abs(a - r) <= tol * np.abs(r).max(axis=0)), np.abs(a - r).max()
