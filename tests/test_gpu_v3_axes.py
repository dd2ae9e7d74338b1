"""The three mesh axes of the V3 kernels that treat them differently, on
crystals whose mesh has another number of points along each (GPU).

|V3|^2 of 3 and 6 bands, class sums taken axis by axis, against the factorised
oracle: FP64 with the bars of test_gpu_parity.py, mixed 1e-5 normwise, as in
test_gpu_v3_line.py.  The one-pass kernel of 3 bands with several rows to a
launch and a remainder, against the two kernels: 1e-13 of each value, as there.
"""
import numpy as np
import pytest

import oracle_dense
from ortho import make_ortho
from test_gpu_parity import close, gamma_acoustic_mask
from test_gpu_v3_tile import Injected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms", [1, 2])
@pytest.mark.parametrize("mesh", [(4, 6, 8), (10, 4, 2), (2, 8, 4), (3, 4, 5), (5, 7, 3)])
def test_axes(oracle_lib, ald_lib, workdir, atoms, mesh):
    d = make_ortho(workdir, atoms, mesh, delta="gauss")
    O = oracle_lib.Oracle(d)
    O.mesh()
    O.phonons()
    O.tet()
    ev, vec, vel = O.get_phonons()
    ph = np.maximum(ev, 1e-10 * ev.max()), vec, vel  # an exact zero at the zone centre is refused
    rows = (O.nibz // 2, O.nibz // 2 + 1)
    ref = oracle_dense.v3_factorised(Injected(O, ph), *rows)
    keep = ~gamma_acoustic_mask(O, ev, *rows)
    for prec in (ald_lib.FP64, ald_lib.MIXED):
        with ald_lib.Context(d, ald_lib.default_options(precision=prec, delta=ald_lib.DELTA_GAUSS)) as ctx:
            ctx.set_phonons(*ph)
            v = ctx.calculate_w3_ibz_split_sq(list(rows))
        if prec == ald_lib.FP64:
            ok, worst = close(v[keep], ref[keep])
            assert ok, worst
        else:
            assert np.linalg.norm(v[keep] - ref[keep]) <= 1e-5 * np.linalg.norm(ref[keep])


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("mesh", [(4, 6, 8), (6, 4, 10), (3, 5, 7)])
def test_one_pass_rows(ald_lib, workdir, mesh, prec):
    d = make_ortho(workdir, 1, mesh, delta="gauss")
    P = ald_lib.FP64 if prec == "fp64" else ald_lib.MIXED
    nkc, out, launches = int(np.prod(mesh)), [], []
    for chunk in (0, 20 * nkc * 27 * 8, 1):  # two kernels; one pass, several rows to a launch; one row
        with ald_lib.Context(d, ald_lib.default_options(precision=P, delta=ald_lib.DELTA_GAUSS,
                                                        chunk_bytes=chunk)) as ctx:
            if not out:
                ev, vec, vel = ctx.get_frequencies()
                ph = np.maximum(ev, 1e-10 * ev.max()), vec, vel
            ctx.set_phonons(*ph)
            out.append(ctx.kappa_pipeline(300.0))
            launches.append(out[-1]["launches"]["delta"] // 4)
    assert out[0]["launches"]["v3"] > 0 and out[1]["launches"]["v3"] == out[2]["launches"]["v3"] == 0
    assert 1 < launches[1] < launches[2] == ctx.nibz
    for k in ("Q", "QN", "QU"):
        assert np.all(np.abs(out[1][k] - out[0][k]) <= 1e-13 * np.abs(out[0][k])), k
        assert np.array_equal(out[1][k], out[2][k]), k
