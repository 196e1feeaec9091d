"""The 2D loop kernels (one resident CTA per block, or active lists) against the same
solve with the loop's kernels launched one by one: results, history, iteration and visit
counts are equal, bit for bit, at the sizes where the launch rule changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _handle(eik, mg, mesh, n, vpb, seeds, cap=1000, history=0, init=None, speeds=True):
    if mesh == "ico":
        xyz, faces = mg.icosphere(n)
    else:
        xyz, faces = mg.grid2d(n)
        if mesh == "obtuse":
            rng = np.random.default_rng(n)
            d = rng.uniform(-0.3, 0.3, size=(n, n, 2)) / (n - 1)
            d[0] = d[-1] = 0
            d[:, 0] = d[:, -1] = 0
            xyz = xyz.copy()
            xyz[:, :2] += d.reshape(-1, 2).astype(np.float32)
    e = eik.Eikonal(True)
    e.set_mesh(xyz, faces)
    e.maxVertsPerBlock_ = vpb
    e.maxIterations_ = cap
    e.keepHistory_ = history
    if isinstance(speeds, tuple):
        e.initSpeedMtxMultipliers((10.0 ** np.random.default_rng(n).uniform(*speeds, len(faces))).astype(np.float32))
    elif speeds:
        e.initSpeedMtxMultipliers(mg.batch_speed(xyz, faces))
    if init is not None:
        v = np.full(xyz.shape[0], 1e7, np.float32)
        v[seeds] = 0
        v[init] = 3.0  # initial values that are neither 0 nor unreached
        e.initializeVertices(v)
    else:
        e.setSeeds(seeds)
    return e


def _snapshot(e):
    e.solveEikonal()
    s = e.stats()
    out = [e.getFinalResult().view(np.uint32), np.array([s[k] for k in (
        "iterations", "vertex_updates", "fim_visits", "check_visits", "slot_visits", "halo_visits", "owned_visits",
        "fim_slots", "fim_halo", "fim_owned")])]
    if e.keepHistory_:
        out += [e.getResultAtIteration(i).view(np.uint32) for i in range(e.numIterations())]
    return out


# blocks: 10 (one warp-sized group), 68, 96/97 (polling rule), 160, 320, 760/761 (residency
# rule at 152 SMs), 1300 (lists); 320/321 slots and more per block (lanes rule)
@pytest.mark.parametrize("mesh,n,vpb,seeds,kw", [
    ("grid", 33, 16, [0, 700], dict(speeds=False, history=1)),
    ("grid", 5, 64, [0], {}),
    ("ico", 2, 32, [0, 90], dict(history=1)),
    ("ico", 4, 26, [0, 7], {}),
    ("ico", 4, 27, [0, 7], {}),
    ("ico", 5, 64, [0], dict(history=1)),
    ("ico", 5, 32, [0, 9000], {}),
    ("obtuse", 156, 32, [0, 1, 20000, 24000], {}),
    ("obtuse", 157, 32, [0, 1, 20000, 24000], dict(history=1, cap=100)),
    ("ico", 6, 32, [0, 5, 30000], {}),
    ("ico", 5, 140, [0, 9000], {}),
    ("ico", 6, 170, [0, 9000], {}),
    ("ico", 5, 400, [0], {}),
    ("ico", 5, 64, [0, 50], dict(cap=3, history=1)),
    ("ico", 6, 32, [0, 50], dict(cap=2)),
    ("ico", 5, 64, [0, 50], dict(init=[7, 8, 9])),
    ("ico", 6, 32, [0, 50], dict(init=[7, 8, 9])),
])
def test_loop_kernels_equal_single_launches(eik, mg, mesh, n, vpb, seeds, kw):
    e = _handle(eik, mg, mesh, n, vpb, seeds, **kw)
    got = _snapshot(e)
    again = _snapshot(e)
    e.directLaunch_ = 1
    want = _snapshot(e)
    e.directLaunch_ = 0
    after = _snapshot(e)
    for other in (again, want, after):
        assert len(got) == len(other)
        assert all(np.array_equal(a, b) for a, b in zip(got, other))


@pytest.mark.parametrize("levels,vpb", [([2, 3, 2, 4], 32), ([2, 3, 4, 5, 3], 16), ([5, 6, 2, 6], 32), ([5, 4], 160)])
def test_batches_equal_single_solves(eik, mg, levels, vpb):
    hs = [_handle(eik, mg, "ico", lv, vpb, [0, 3 * i + 1], cap=1000 if i else 2) for i, lv in enumerate(levels)]
    hs.append(_handle(eik, mg, "grid", 3, vpb, [0], cap=0))  # runs nothing
    b = eik.EikonalBatch(hs)
    for _ in range(2):
        b.solveEikonal()
        res = [r.copy() for r in b.getFinalResults()]
        for i, h in enumerate(hs):
            h.directLaunch_ = 1
            h.solveEikonal()
            h.directLaunch_ = 0
            assert np.array_equal(res[i].view(np.uint32), h.getFinalResult().view(np.uint32)), i
            assert b.numIterations(i) == h.numIterations()


# resident blocks, lists with three lanes, lists with one lane per slot
@pytest.mark.parametrize("grow,blocks", [(1, (1, 760)), (2.5, (761, 2736)), (4.5, (2737, 20000))])
def test_batches_of_obtuse_meshes_and_extreme_speeds(eik, mg, grow, blocks):
    """With one lane per slot a batch leaves out the update of a slot's earliest corner
    where it cannot fall: equal times, virtual faces, times from 1e-4 to unreachable and the
    caller's own initial values take every side of that rule."""
    hs = []
    for i, (mesh, n, lo, hi) in enumerate([("obtuse", 40, 0, 0), ("grid", 33, 0, 0), ("obtuse", 25, -6, 6),
                                           ("ico", 3, -30, 30), ("obtuse", 50, -2, 1), ("grid", 9, -37, -36)]):
        e = _handle(eik, mg, mesh, int(n * grow) if mesh != "ico" else n, 32, [0, 3 * i + 1], cap=200,
                    init=[5, 6, 11] if i % 2 else None, speeds=(lo, hi))
        hs.append(e)
    b = eik.EikonalBatch(hs)
    b.solveEikonal()
    assert blocks[0] <= b.stats()["num_blocks"] <= blocks[1]
    res = [r.copy() for r in b.getFinalResults()]
    for i, h in enumerate(hs):
        h.directLaunch_ = 1
        h.solveEikonal()
        h.directLaunch_ = 0
        assert np.array_equal(res[i].view(np.uint32), h.getFinalResult().view(np.uint32)), i
        assert b.numIterations(i) == h.numIterations()


def test_concurrent_solves_of_several_threads(eik, mg):
    """Loop kernels that each fill the GPU, launched from four threads at once."""
    import threading

    hs = [_handle(eik, mg, "ico", 6 if i % 2 else 5, 32, [0, 11 * i + 1]) for i in range(4)]
    want = []
    for h in hs:
        h.solveEikonal()
        want.append(h.getFinalResult().view(np.uint32).copy())
    failures = []

    def work(h, w):
        try:
            for _ in range(5):
                h.solveEikonal()
                if not np.array_equal(h.getFinalResult().view(np.uint32), w):
                    failures.append("bits")
        except Exception as ex:  # reported below
            failures.append(repr(ex))

    ts = [threading.Thread(target=work, args=x) for x in zip(hs, want)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failures
