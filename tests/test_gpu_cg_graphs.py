"""The solver's captured graphs after a row-sharded call on the same context
(GPU).  The sharded solver resizes two of the workspaces that the graphs were
captured with; once the freed blocks have gone back to the driver, the next
single-context call must not run those graphs again.  The Gaussian delta's
sums are in a fixed order, so the results are the same bits."""
import numpy as np
import pytest

from conftest import make_case

pytestmark = pytest.mark.gpu


def test_graphs_after_a_sharded_call(ald_lib, workdir):
    d = make_case(workdir, 0, (6, 6, 6), delta="gauss")
    with ald_lib.Context(d, ald_lib.default_options(precision=ald_lib.FP64, delta=ald_lib.DELTA_GAUSS)) as ctx:
        first = ctx.kappa_pipeline(300.0)
        one = ctx.kappa_pipeline_sharded(0, 1, lambda mine, counts: np.array(mine), 300.0)
        ald_lib.release_cached_memory()
        again = ctx.kappa_pipeline(300.0)
    for k in ("Q", "x", "kappa_cg_modes"):
        assert np.array_equal(again[k], first[k]), k
    assert one["cg_iters"] == first["cg_iters"]
