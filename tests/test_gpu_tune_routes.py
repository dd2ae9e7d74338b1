"""What the autotuner may and may not change (GPU): it times the pair-batch
workspace only where the tensor-core GEMMs form V3."""
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
