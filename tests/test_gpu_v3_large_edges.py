"""|V3|^2 of cells beyond the shared-memory kernel (GPU): the batched FP64 GEMMs
and, mixed, the T1 kernel and the tcgen05 GEMMs, at band counts that leave
remainders in their tiles (b not a multiple of 16 pads K; b^2 rows in tiles of
128; 8 atoms per thread of the T1 kernel).  Chains of n atoms with injected
eigenpairs as in test_gpu_v3_tile.py, against the factorised oracle: FP64 with
the bars of test_gpu_parity.py, mixed 1e-5 normwise.

With `soft`, the lowest mode of a row's q1 has 1e-12 of the largest eigenvalue:
the mixed path forms that row's entries of it, and the pairs whose q2 or q3 is
that point, again with the FP64 GEMMs on a pair list (the FP64 bars hold there).
"""
import numpy as np
import pytest

import oracle_dense
from test_gpu_parity import close
from test_gpu_v3_tile import Injected, chain, random_phonons

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("soft", [False, True], ids=["plain", "soft"])
@pytest.mark.parametrize("n,mesh", [(17, (3, 2, 2)), (20, (2, 2, 2)), (28, (2, 2, 2))])
def test_large_v3(oracle_lib, ald_lib, workdir, n, mesh, soft):
    d = chain(workdir, n, mesh)
    O = oracle_lib.Oracle(d)
    O.mesh()
    O.phonons()
    O.tet()
    ev, vec, vel = random_phonons(O.nkc, O.ndyn, n)
    row = (2, 2)
    q1 = O.ibz()["mapinv"][1] - 1
    if soft:
        ev[0, q1] = 1e-12 * ev.max()
    ph = ev, vec, vel
    kpc = O.kpc()
    at_q1 = [q2 for q2 in range(O.nkc) if q1 in (q2, O.get_k_info(-kpc[:, q1] - kpc[:, q2])[0] - 1)]
    q2s = np.unique([0, 1, O.nkc - 2, O.nkc - 1] + at_q1)
    ref = oracle_dense.v3_factorised(Injected(O, ph), *row, q2s=q2s)[:, q2s]
    for prec in (ald_lib.FP64, ald_lib.MIXED):
        with ald_lib.Context(d, ald_lib.default_options(precision=prec, delta=ald_lib.DELTA_GAUSS)) as ctx:
            ctx.set_phonons(*ph)
            v = ctx.calculate_w3_ibz_split_sq(list(row))[:, q2s]
            if not soft:  # the shared-memory kernel's V3 is three launches
                assert ctx.kappa_pipeline(300.0)["launches"]["v3"] > 3
        if prec == ald_lib.FP64:
            ok, worst = close(v, ref)
            assert ok, worst
        elif not soft:
            assert np.linalg.norm(v - ref) <= 1e-5 * np.linalg.norm(ref)
        else:
            redone = np.isin(q2s, at_q1)
            rest = v[:, ~redone][:, :, 1:], ref[:, ~redone][:, :, 1:]
            assert np.linalg.norm(rest[0] - rest[1]) <= 1e-5 * np.linalg.norm(rest[1])
            for a, b in ((v[:, redone], ref[:, redone]), (v[:, :, 0], ref[:, :, 0])):
                ok, worst = close(a, b)
                assert ok, worst


@pytest.mark.parametrize("n,mesh", [(2, (5, 5, 5)), (3, (3, 6, 6)), (4, (7, 4, 4))])
def test_gauss_walking_l3_over_several_blocks(ald_lib, workdir, n, mesh):
    """More mesh points than the 32 of a block, not a multiple of them: R2 goes to -q in another block.  FP64, 1e-12 of
    each sum of positive terms."""
    d = chain(workdir, n, mesh)
    with ald_lib.Context(d, ald_lib.default_options(precision=ald_lib.FP64, delta=ald_lib.DELTA_GAUSS)) as ctx:
        ctx.set_phonons(*random_phonons(ctx.nkc, ctx.ndyn, n))
        out = ctx.kappa_pipeline(300.0)
        for r in (1, ctx.nibz // 2, ctx.nibz):
            v = ctx.calculate_w3_ibz_split_sq([r, r])
            P1, P2 = ctx.calculate_fgr([r, r], v)
            ctx.distribution(300.0)
            Q, QN, QU, _, _ = ctx.calculate_tau_rta([r, r], 300.0, P1, P2, want_p=False)
            for a, b in ((out["Q"], Q), (out["QN"], QN), (out["QU"], QU)):
                assert np.all(np.abs(a[r - 1] - b[0]) <= 1e-12 * np.abs(b[0])), r
