"""|V3|^2 of 3-band cells with the class sums taken axis by axis, and V3 with
the Gaussian delta in one pass (GPU).

The line kernel works on 128 consecutive mesh points and the mesh lines they
touch, so the edges that matter are those of N (points per line: 3 and 4 put
many lines into a block, 12 and 13 a remainder at both ends) and of nkc mod
128 (at 2 every point is its own negative and all of V3 vanishes by inversion).  |V3|^2 is compared with the factorised oracle in FP64 (the bars of
test_gpu_parity.py) and the FP32 form with it normwise; a chunk of one row
makes the pipeline take the one-pass kernel, whose linewidths must equal the
two-kernel path's (same terms, products regrouped: 1e-13 of each value leaves
a factor 100 over the rounding of their six factors; sums of positive terms).
"""
import numpy as np
import pytest

import oracle_dense
from conftest import make_case
from test_gpu_parity import close, gamma_acoustic_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 4, 5, 8, 12, 13])
def test_line_v3(oracle_lib, ald_lib, workdir, n):
    d = make_case(workdir, 0, (n, n, n), rc_sigma=1.2 if n > 8 else 2.5, delta="gauss")
    O = oracle_lib.Oracle(d)
    O.mesh()
    O.phonons()
    O.tet()  # the double-precision mesh that V3's phases go by
    ph = O.get_phonons()
    row = (1, 1) if n % 2 == 0 else (O.nibz, O.nibz)  # not the zone centre, whose entries are all 0/0
    q2s = np.unique(np.r_[0:min(O.nkc, 40), max(0, O.nkc - 40):O.nkc])
    ref = oracle_dense.v3_factorised(O, *row, q2s=q2s)[:, q2s]
    keep = ~gamma_acoustic_mask(O, ph[0], *row)[:, q2s]
    for prec in (ald_lib.FP64, ald_lib.MIXED):
        with ald_lib.Context(d, ald_lib.default_options(precision=prec, delta=ald_lib.DELTA_GAUSS)) as ctx:
            ctx.set_phonons(*ph)
            v = ctx.calculate_w3_ibz_split_sq(list(row))[:, q2s]
        if prec == ald_lib.FP64:
            ok, worst = close(v[keep], ref[keep])
            assert ok, worst
        else:
            assert np.linalg.norm(v[keep] - ref[keep]) <= 1e-5 * np.linalg.norm(ref[keep])


@pytest.mark.parametrize("n", [3, 4, 6, 10])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_v3_gauss_one_pass(ald_lib, workdir, n, prec):
    d = make_case(workdir, 0, (n, n, n), delta="gauss")
    P = ald_lib.FP64 if prec == "fp64" else ald_lib.MIXED
    out = []
    for chunk in (0, 1):
        with ald_lib.Context(d, ald_lib.default_options(precision=P, delta=ald_lib.DELTA_GAUSS,
                                                        chunk_bytes=chunk)) as ctx:
            if not out:
                ph = ctx.get_frequencies()
            ctx.set_phonons(*ph)
            out.append(ctx.kappa_pipeline(300.0))
            rows = ctx.nibz
    assert out[0]["launches"]["v3"] > 0 and (out[1]["launches"]["v3"] == 0 or rows == 1)
    for k in ("Q", "QN", "QU"):
        assert np.all(np.abs(out[1][k] - out[0][k]) <= 1e-13 * np.abs(out[0][k])), k
