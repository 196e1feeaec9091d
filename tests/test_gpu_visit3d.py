"""The 3D item visit (copies put off, one update body for all apexes): the resident loop,
precision mode with no tet flagged and the kernel-by-kernel loop agree on results,
iteration and visit counts, bit for bit, over block shapes around a CTA's and a warp's
size, scalar and anisotropic metrics, slivers, caps and several seeds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(mg, mesh, n):
    xyz, tets = mg.kuhn_cube(n, 0.0 if mesh == "flat" else 0.2, seed=n)
    if mesh == "layers":  # a thin layer: slivers
        xyz = xyz.copy()
        z = xyz[:, 2]
        xyz[:, 2] = np.where(z > 0.5, z - 0.97 / (n - 1) * np.minimum(1.0, (z - 0.5) * (n - 1)), z)
    return xyz, tets


def _solve(eik, xyz, tets, metric, seeds, vpb, cap, slots, **opts):
    e = eik.Eikonal(False)
    e.set_mesh(xyz, tets)
    e.maxVertsPerBlock_ = vpb
    e.maxIterations_ = cap
    for k, v in opts.items():
        setattr(e, k, v)
    if slots:
        e.precisionMode_ = 1
        e.precisionKappa_ = 1e30
    if metric is not None:
        e.initSpeedMtxMultipliers(metric)
    e.setSeeds(seeds)
    e.solveEikonal()
    first = e.getFinalResult().view(np.uint32).copy()
    e.solveEikonal()
    assert np.array_equal(first, e.getFinalResult().view(np.uint32))
    s = e.stats()
    assert s["flagged_tets"] == 0
    return [first, np.array([s[k] for k in ("iterations", "vertex_updates", "fim_visits", "check_visits")])] + [
        e.getResultAtIteration(i).view(np.uint32) for i in range(e.numIterations())]


@pytest.mark.parametrize("mesh,n,vpb,metric,seeds,cap", [
    ("cube", 3, 64, 1, [0], 100),
    ("cube", 5, 2, 1, [0, 100], 200),
    ("cube", 9, 8, 1, [0], 200),
    ("cube", 13, 33, 6, [5, 1000], 200),
    ("cube", 17, 64, 1, [0, 2000, 4912], 100),
    ("cube", 17, 64, 0, [2456], 100),
    ("flat", 17, 64, 0, [2456], 100),
    ("cube", 21, 100, 1, [7], 200),
    ("cube", 21, 280, 1, [7], 200),  # blocks of 2700 and 3000 slots, at the end of what
    ("cube", 21, 310, 6, [7, 9000], 200),  # shared memory holds
    ("layers", 17, 64, 6, [0, 4000], 300),
    ("layers", 15, 48, 1, [1687], 300),
    ("cube", 25, 64, 6, [0, 7812, 15000], 1),
    ("cube", 25, 64, 1, [0, 7812, 15000], 2),
    ("cube", 25, 64, 1, [0, 7812, 15000], 7),
])
def test_item_visits_agree(eik, mg, mesh, n, vpb, metric, seeds, cap):
    xyz, tets = _mesh(mg, mesh, n)
    m = None
    if metric == 1:
        m = (1.0 / mg.log_uniform_speeds(tets.shape[0], seed=n).astype(np.float64) ** 2).astype(np.float32)
    elif metric == 6:
        m = mg.anisotropic_metrics(tets.shape[0], seed=n)
    got = _solve(eik, xyz, tets, m, seeds, vpb, cap, False)
    want = _solve(eik, xyz, tets, m, seeds, vpb, cap, True)
    one_by_one = _solve(eik, xyz, tets, m, seeds, vpb, cap, False, directLaunch_=1)
    for other in (want, one_by_one):
        assert len(got) == len(other)
        assert all(np.array_equal(a, b) for a, b in zip(got, other))


def test_batch_with_caps_equals_single_solves(eik, mg):
    """Instances that stop at their caps keep their times while the others run on."""
    hs = []
    for i, (n, cap) in enumerate([(9, 1), (13, 4), (17, 1000), (21, 6), (7, 0), (15, 1000), (17, 11)]):
        xyz, tets = mg.kuhn_cube(n, 0.2, seed=n)
        e = eik.Eikonal(False)
        e.set_mesh(xyz, tets)
        e.maxIterations_ = cap
        e.keepHistory_ = 0
        e.initSpeedMtxMultipliers(mg.log_uniform_speeds(tets.shape[0], seed=i))
        e.setSeeds([i, xyz.shape[0] // 2])
        hs.append(e)
    b = eik.EikonalBatch(hs)
    for _ in range(2):
        b.solveEikonal()
        res = [r.copy() for r in b.getFinalResults()]
        total = b.stats()
        visits = np.zeros(4, np.int64)
        for i, h in enumerate(hs):
            h.directLaunch_ = 1
            h.solveEikonal()
            h.directLaunch_ = 0
            s = h.stats()
            visits += [s["vertex_updates"], s["fim_visits"], s["check_visits"], s["slot_visits"]]
            assert np.array_equal(res[i].view(np.uint32), h.getFinalResult().view(np.uint32)), i
            assert b.numIterations(i) == h.numIterations()
        assert visits.tolist() == [total[k] for k in ("vertex_updates", "fim_visits", "check_visits", "slot_visits")]


def test_concurrent_solves_of_several_threads(eik, mg):
    """Loop kernels that each fill the GPU, launched from four threads at once."""
    import threading

    hs, want, failures = [], [], []
    for i in range(4):
        xyz, tets = mg.kuhn_cube(27 + i, 0.2, seed=i)
        e = eik.Eikonal(False)
        e.set_mesh(xyz, tets)
        e.keepHistory_ = 0
        e.setSeeds([i])
        e.solveEikonal()
        hs.append(e)
        want.append(e.getFinalResult().view(np.uint32).copy())

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
