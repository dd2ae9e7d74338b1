"""What the autotuner may and may not change (GPU): it times the pair-batch
workspace only where the tensor-core GEMMs form V3, and its chunk changes how
rows are grouped, not which kernels form them: 3 bands with the Gaussian delta
have one for V3 and delta together, taken by the chunk that the context was
created with (the sums are in a fixed order, so the same kernels give the same
bits)."""
import numpy as np
import pytest

from conftest import make_case

pytestmark = pytest.mark.gpu


def test_no_gemm_candidates_for_cells_in_shared_memory(ald_lib, workdir):
    d = make_case(workdir, 3, (4, 4, 4), rc_sigma=1.2, delta="gauss")  # 12 bands
    with ald_lib.Context(d, ald_lib.default_options(precision=ald_lib.MIXED, delta=ald_lib.DELTA_GAUSS)) as ctx:
        t = ctx.autotune(None, budget_s=30)
    # the context's own choice and three chunk sizes
    assert t["v3_gemm_bytes"] == 0 and t["candidates"] == 4


@pytest.mark.parametrize("asked,tuned", [(0, 1), (1, 0), (1, 1 << 30), (0, 20000)])
def test_tuned_chunk_leaves_the_bits(ald_lib, workdir, asked, tuned):
    d = make_case(workdir, 0, (6, 6, 6), delta="gauss")
    opts = ald_lib.default_options(precision=ald_lib.FP64, delta=ald_lib.DELTA_GAUSS, chunk_bytes=asked)
    with ald_lib.Context(d, opts) as ctx:
        ref = ctx.kappa_pipeline(300.0)
        ctx.set_tuning(chunk_bytes=tuned)
        got = ctx.kappa_pipeline(300.0)
    for k in ("Q", "QN", "QU", "x"):
        assert np.array_equal(got[k], ref[k]), k
