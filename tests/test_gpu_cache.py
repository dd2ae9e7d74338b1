"""The library's device-memory cache in a process that has run large cells
(GPU): the sizes in use now stay cached although the cache is full of others.

Rock-salt contexts from 20^3 down, whose chunks hold every row, leave more than
the cache's 32 GiB behind, in blocks small enough to fill it.  A 12^3 context that ran once and was closed then serves
the next one of its shape: that one's whole run, about 1 GB of workspaces, may
take no more than 64 MiB from the driver."""
import gc

import pytest

from conftest import make_case

pytestmark = pytest.mark.gpu


def test_sizes_in_use_stay_cached(ald_lib, workdir):
    torch = pytest.importorskip("torch")
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    gc.collect()
    ald_lib.release_cached_memory()
    start = free()
    opts = ald_lib.default_options(precision=ald_lib.FP64, chunk_bytes=16 << 30)
    ctxs = [ald_lib.Context(make_case(workdir, 1, (n, n, n)), opts) for n in (20, 20, 20, 18, 18, 16, 16, 14, 14, 10, 10, 10)]
    for c in ctxs:
        c.kappa_pipeline(300.0)
    assert start - free() > 40 << 30
    for c in ctxs:
        c.close()
    assert start - free() < 33 << 30  # the cache's limit, and the driver's own
    small = make_case(workdir, 1, (12, 12, 12))
    for _ in range(3):  # the first ones may push the older blocks out
        with ald_lib.Context(small) as c:
            c.kappa_pipeline(300.0)
    before = free()
    with ald_lib.Context(small) as c:
        c.kappa_pipeline(300.0)
        taken = before - free()
    assert start - free() < 33 << 30
    ald_lib.release_cached_memory()
    assert taken <= 64 << 20, taken
