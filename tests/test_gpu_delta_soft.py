"""The one-pass deterministic tetrahedron delta beside a mode of nearly
vanishing frequency (GPU).

The lowest mode of one mesh point and of its negative, away from the point of
the zone-centre test, gets `soft` of the largest eigenvalue: |V3|^2 and the
occupation of every triplet with it grow as 1/sqrt(soft) each, whether or not
the triplet has weight.  A sum's other terms must keep their digits.  At 1e-18
the one-pass form (5 delta launches) still does; at 1e-24 the pipeline must
take the two-pass form (4).  Either way Q, Q_N and Q_U come within 1e-12 of
those of the FP64-atomic form, each value (sums of positive terms, a few
thousand of them: 1e-13 of rounding), with the same bits twice.
"""
import numpy as np
import pytest

from conftest import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("soft", [1e-10, 1e-18, 1e-24])
@pytest.mark.parametrize("cfg,mesh,point", [(1, (5, 5, 5), (0, 1, 2)), (1, (6, 6, 6), (1, 2, 4)), (0, (7, 7, 7), (2, 0, 1))],
                         ids=["nacl_odd", "nacl_even", "lj_odd"])
def test_soft_mode(ald_lib, workdir, cfg, mesh, point, soft):
    d = make_case(workdir, cfg, mesh, delta="tetra")
    neg = tuple(-p % n for p, n in zip(point, mesh))
    out = []
    for det in (1, 1, 0):
        with ald_lib.Context(d, ald_lib.default_options(precision=ald_lib.FP64, deterministic=det)) as ctx:
            ev, vec, vel = ctx.get_frequencies()
            ev = np.maximum(ev, 1e-8 * ev.max())  # the acoustic modes of the zone centre
            for q in (point, neg):
                ev[0, np.ravel_multi_index(q, mesh)] = soft * ev.max()
            ctx.set_phonons(ev, vec, vel)
            out.append(ctx.kappa_pipeline(300.0))
    assert out[0]["launches"]["delta"] == (4 if soft < 1e-20 else 5) and out[2]["launches"]["delta"] == 1
    for k in ("Q", "QN", "QU", "kappa_rta_modes"):
        a, b = np.asarray(out[0][k]), np.asarray(out[2][k])
        assert np.array_equal(a, np.asarray(out[1][k]), equal_nan=True), k
        if k[0] == "Q":
            assert np.isfinite(b).all() and b.max() > 0
            assert np.all(np.abs(a - b) <= 1e-12 * np.abs(b)), (k, np.max(np.abs(a - b) / np.maximum(b, 1e-300)))
