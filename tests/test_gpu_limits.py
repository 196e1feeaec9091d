"""Blocks at the end of what shared memory holds, and every CTA size that the options
document: each call runs, and gives the bits, iterations and visit counts of the routes
that such a limit does not touch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def kuhn_box(mg, nx, ny, nz):
    """A box of nx x ny x nz vertices: a corner of the flat Kuhn cube."""
    n = max(nx, ny, nz)
    xyz, tets = mg.kuhn_cube(n, 0.0)
    k, j, i = np.unravel_index(np.arange(n ** 3), (n, n, n))
    keep = (i < nx) & (j < ny) & (k < nz)
    new = np.cumsum(keep) - 1
    return xyz[keep], new[tets[keep[tets].all(1)]].astype(np.int32)


def outcome(e):
    e.solveEikonal()
    s = e.stats()
    return [e.getFinalResult().view(np.uint32).copy(),
            np.array([s[k] for k in ("iterations", "vertex_updates", "fim_visits", "check_visits")])]


@pytest.mark.parametrize("box,vpb,slots", [
    ((14, 19, 19), 440, 3074),
    ((14, 19, 19), 460, 3364),  # the visit's state fits, beside what the loop kernel keeps itself it does not
    ((14, 19, 21), 468, 3362),
])
def test_blocks_at_the_shared_memory_limit(need_gpu, eik, mg, box, vpb, slots):
    xyz, tets = kuhn_box(mg, *box)
    metric = (1.0 / mg.log_uniform_speeds(tets.shape[0], seed=3).astype(np.float64) ** 2).astype(np.float32)
    got = []
    for opts in ({}, {"directLaunch_": 1}, {"precisionMode_": 1, "precisionKappa_": 1e30}):
        e = eik.Eikonal(False)
        e.set_mesh(xyz, tets)
        e.initSpeedMtxMultipliers(metric)
        e.setSeeds([0, xyz.shape[0] // 2])
        e.maxVertsPerBlock_ = vpb
        e.maxIterations_ = 1000
        e.keepHistory_ = 0
        for k, v in opts.items():
            setattr(e, k, v)
        got.append(outcome(e))
        assert e.stats()["max_slots_per_block"] == slots
    for other in got[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(got[0], other))


def test_precision_mode_at_every_cta_size(need_gpu, eik, mg):
    """A mesh with flagged tets; 1024 threads leave each 64 registers."""
    xyz, tets = mg.kuhn_cube(13, 0.2, seed=4)
    xyz[:, 2] = np.where(xyz[:, 2] > 0.5, xyz[:, 2] - 0.97 / 12 * np.minimum(1.0, (xyz[:, 2] - 0.5) * 12), xyz[:, 2])
    metric = mg.anisotropic_metrics(tets.shape[0], seed=4)
    got = []
    for threads in (0, 128, 256, 384, 512, 768, 1024):
        e = eik.Eikonal(False)
        e.set_mesh(xyz, tets)
        e.initSpeedMtxMultipliers(metric)
        e.setSeeds([5, 1000])
        e.maxIterations_ = 1000
        e.keepHistory_ = 0
        e.precisionMode_ = 1
        e.threadsPerBlock_ = threads
        got.append(outcome(e))
        assert e.stats()["flagged_tets"] > 0
    for other in got[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(got[0], other))
