"""The one-pass deterministic tetrahedron delta where its fixed-point scale does
not reach (GPU).

The scale leaves room for corner weights up to 2^22 cm.  Flat bands at 0.5 and
1.0 cm^-1 that differ from point to point by 1e-7 put omega1 into tetrahedra a
few single-precision steps wide, whose weights are larger; the pipeline must then
take the two-pass form (4 delta launches against 5) and give its results: the
same bits twice, and the sums of the FP64-atomic form to 1e-12 of each value.
"""
import numpy as np
import pytest

from conftest import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flat", [False, True])
def test_weights_beyond_the_scale(ald_lib, workdir, flat):
    d = make_case(workdir, 1, (4, 4, 4))
    out = []
    for det in (1, 1, 0):
        with ald_lib.Context(d, ald_lib.default_options(precision=ald_lib.FP64, deterministic=det)) as ctx:
            ev, vec, vel = ctx.get_frequencies()
            if flat:
                rng = np.random.default_rng(0)
                f = np.where(np.arange(6) < 3, 0.5, 1.0)[:, None] * (1 + 1e-7 * rng.uniform(-1, 1, ev.shape))
                ctx.set_phonons((f / 521.1098918) ** 2, vec, vel)
            out.append(ctx.kappa_pipeline(300.0))
    assert out[0]["launches"]["delta"] == (4 if flat else 5)
    assert np.isfinite(out[0]["Q"]).all() and out[0]["Q"].max() > 0
    for k in ("Q", "QN", "QU", "kappa_rta"):
        assert np.array_equal(out[0][k], out[1][k], equal_nan=True), k  # flat: modes without decay, kappa 0/0
    for k in ("Q", "QN", "QU"):
        assert np.all(np.abs(out[0][k] - out[2][k]) <= 1e-12 * np.abs(out[2][k])), k
