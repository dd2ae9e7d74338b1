"""The deterministic delta of the row-sharded pipeline (GPU): a rank's rows are
formed as the single context forms them, so Q, Q_N and Q_U are the same bits
(FP64, tetrahedra).  Where the one-pass form's scale does not reach (flat
bands, as in test_gpu_delta_wide.py), a rank takes its own rows again in two
passes, without the other rank and before the exchange: 1e-12 of each value
of the single context's, which takes every row again.  The ranks are host
threads on the one GPU; only the host waits."""
import threading

import numpy as np
import pytest

from conftest import make_case
from test_gpu_shard import InProcessGather

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flat", [False, True])
def test_sharded_rows_have_the_single_contexts_bits(ald_lib, workdir, flat):
    d = make_case(workdir, 1, (6, 6, 6))
    n = 2
    ctxs = [ald_lib.Context(d, ald_lib.default_options(precision=ald_lib.FP64)) for _ in range(n + 1)]
    ev, vec, vel = ctxs[0].get_frequencies()
    if flat:
        rng = np.random.default_rng(0)
        f = np.where(np.arange(6) < 3, 0.5, 1.0)[:, None] * (1 + 1e-7 * rng.uniform(-1, 1, ev.shape))
        ev = (f / 521.1098918) ** 2
    for c in ctxs:
        c.set_phonons(ev, vec, vel)
    g, outs, errs = InProcessGather(n), [None] * n, []

    def work(r):
        try:
            outs[r] = ctxs[r].kappa_pipeline_sharded(r, n, g.for_rank(r), 300.0)
        except Exception as ex:
            errs.append(ex)
            g.barrier.abort()

    th = [threading.Thread(target=work, args=(r,)) for r in range(n)]
    for t in th:
        t.start()
    for t in th:
        t.join(timeout=600)
    assert not errs, errs
    ref = ctxs[n].kappa_pipeline(300.0)
    for c in ctxs:
        c.close()
    assert ref["Q"].max() > 0
    for o in outs:
        for k in ("Q", "QN", "QU"):
            if flat:
                assert np.all(np.abs(o[k] - ref[k]) <= 1e-12 * np.abs(ref[k])), k
            else:
                assert np.array_equal(o[k], ref[k]), k
