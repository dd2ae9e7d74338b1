"""Device memory of the class sums taken axis by axis (GPU): per |V3|^2 byte
they go as one over the points of the last axis, so a mesh that is thin there
must not take several times the chunk's bytes for them; taking a chunk's rows
in several batches leaves the bits as they are."""
import gc

import numpy as np
import pytest

from ortho import make_ortho

pytestmark = pytest.mark.gpu


def test_thin_mesh_stays_within_the_chunk(ald_lib, workdir):
    torch = pytest.importorskip("torch")
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    d = make_ortho(workdir, 2, (32, 32, 2), delta="tetra")
    chunk = 512 << 20
    gc.collect()
    with ald_lib.Context(d, ald_lib.default_options(precision=ald_lib.FP64, chunk_bytes=chunk)) as ctx:
        b, nkc, nibz = 6, 2048, ctx.nibz
        ald_lib.release_cached_memory()
        before = free()
        ctx.kappa_pipeline(300.0)
        used = before - free()
    rsz = 8 * nkc * b * b
    rows = chunk // (rsz * b)
    sums = 2 * nibz * rsz + 4 * rows * rsz + 2 * 2 * rows * nkc * b * b  # R1, R2, the chunk's lower parts and scales
    matrix = 8 * (3 * b * nibz) ** 2
    # |V3|^2 and the line sums of a chunk, and 256 MiB for all that is small
    assert used <= sums + matrix + 2 * chunk + (256 << 20), (used, sums, matrix)


@pytest.mark.parametrize("atoms,mesh", [(1, (6, 10, 2)), (2, (6, 8, 2))])
def test_rows_in_batches(ald_lib, workdir, atoms, mesh):
    d = make_ortho(workdir, atoms, mesh, delta="tetra")
    out = []
    for chunk in (0, 1 << 20, 1):
        with ald_lib.Context(d, ald_lib.default_options(precision=ald_lib.FP64, chunk_bytes=chunk)) as ctx:
            if not out:
                ev, vec, vel = ctx.get_frequencies()
                # an eigenvalue of the zone centre that is exactly zero is refused
                ph = np.maximum(ev, 1e-10 * ev.max()), vec, vel
            ctx.set_phonons(*ph)
            out.append(ctx.kappa_pipeline(300.0))
    assert out[1]["launches"]["v3"] > out[0]["launches"]["v3"]
    for o in out[1:]:
        for k in ("Q", "QN", "QU"):
            assert np.array_equal(o[k], out[0][k]), k


def test_batch_on_a_nearly_full_device(ald_lib, workdir):
    """Six structures of about 3.1 GB each with 9 GB free: the batched entry point starts as many at once as fit."""
    torch = pytest.importorskip("torch")
    d = make_ortho(workdir, 2, (32, 32, 2), delta="tetra")
    opts = ald_lib.default_options(precision=ald_lib.FP64)
    ctxs = [ald_lib.Context(d, opts) for _ in range(6)]
    gc.collect()
    ald_lib.release_cached_memory()
    torch.cuda.empty_cache()
    ballast = torch.empty(torch.cuda.mem_get_info()[0] - (9 << 30), dtype=torch.uint8, device="cuda")
    try:
        out, status = ald_lib.kappa_batched(ctxs, [300.0] * 6)
    finally:
        del ballast
        torch.cuda.empty_cache()
        for c in ctxs:
            c.close()
        ald_lib.release_cached_memory()
    assert status == [0] * 6
    for o in out[1:]:
        assert np.array_equal(o["kappa_rta"], out[0]["kappa_rta"], equal_nan=True)
