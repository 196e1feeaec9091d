"""Several threads with a handle each: their solves share the GPU, and none of them gives
other bits than alone."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cube(eik, mg, n, seed, **opts):
    xyz, tets = mg.kuhn_cube(n, 0.2, seed=seed)
    e = eik.Eikonal(False)
    e.set_mesh(xyz, tets)
    e.initSpeedMtxMultipliers((1.0 / mg.log_uniform_speeds(tets.shape[0], seed=seed) ** 2).astype(np.float32))
    e.setSeeds([seed, xyz.shape[0] // 2])
    e.maxIterations_ = 1000
    e.keepHistory_ = 0
    for k, v in opts.items():
        setattr(e, k, v)
    for _ in range(2):
        e.solveEikonal()
    return e


def _rate(handles, seconds=0.3):
    """Solves a second, a thread per handle."""
    count, end = [0] * len(handles), time.perf_counter() + seconds

    def work(i):
        while time.perf_counter() < end:
            handles[i].solveEikonal()
            count[i] += 1

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(handles))]
    t0 = time.perf_counter()
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    return sum(count) / (time.perf_counter() - t0)


def _surface(eik, mg, n, vpb, seed):
    xyz, faces = mg.icosphere(n) if n < 10 else mg.grid2d(n)
    e = eik.Eikonal(True)
    e.set_mesh(xyz, faces)
    e.maxVertsPerBlock_ = vpb
    e.initSpeedMtxMultipliers(mg.batch_speed(xyz, faces))
    e.setSeeds([0, seed])
    e.maxIterations_ = 1000
    e.keepHistory_ = 0
    for _ in range(2):
        e.solveEikonal()
    return e


def test_a_solve_does_not_hold_up_other_threads_in_the_driver(need_gpu, eik, mg):
    """Two threads whose solves a graph runs (other sweep counts than the reference's), short
    ones beside long ones: several short solves end during a long one, where a wait inside
    the driver lets about one through."""
    long, short, stop, n = _cube(eik, mg, 57, 1, fimSweeps_=3), _surface(eik, mg, 33, 16, 5), threading.Event(), [0]
    short.fimSweeps_ = 5
    for _ in range(2):
        short.solveEikonal()

    def work():
        while not stop.is_set():
            long.solveEikonal()
            n[0] += 1

    t = threading.Thread(target=work)
    t.start()
    while n[0] < 2:
        time.sleep(0.001)
    first, count = n[0], 0
    while n[0] < first + 30:
        short.solveEikonal()
        count += 1
    stop.set()
    t.join()
    assert count > 2.5 * 30, count


def test_threads_share_the_gpu(need_gpu, eik, mg):
    """Loops of 160 blocks fill the GPU one at a time: beside one another the solves run
    by the graph.  Eight threads get three times the solves of one or more."""
    hs = [_surface(eik, mg, 5, 64, i + 1) for i in range(8)]
    ratio = max(_rate(hs) / _rate(hs[:1]) for _ in range(3))
    assert ratio > 2.2, ratio


def test_requests_are_served_beside_solves(need_gpu, eik, mg):
    """A burst of requests beside a thread whose solves follow one another."""
    srv = eik.EikonalServer(hbm_budget_bytes=1 << 30)
    mid = srv.add_mesh(_cube(eik, mg, 21, 1), slots=4)
    srv.start()

    def burst():
        t0 = time.perf_counter()
        for i in range(8):
            srv.submit(mid, [100 * i], 1.0 + i / 8)
        srv.drain(timeout_ms=60000)
        assert all(c["status"] == 0 for c in srv.poll())
        return time.perf_counter() - t0

    burst()
    alone = min(burst() for _ in range(3))
    big, stop = _cube(eik, mg, 65, 2), threading.Event()

    def work():
        while not stop.is_set():
            big.solveEikonal()

    t = threading.Thread(target=work)
    t.start()
    try:
        beside = min(burst() for _ in range(3))
    finally:
        stop.set()
        t.join()
        srv.close()
    # kernels that take turns with the solves' (three times the time alone), not a wait for a
    # whole solve at every kernel boundary (twenty times)
    assert beside < 6 * alone, (beside, alone)


def test_bits_do_not_depend_on_other_calls(need_gpu, eik, mg):
    """Small loops, loops that give way to the graph, a batch, precision mode and served
    requests, all at once."""
    def batch(k):
        b = eik.EikonalBatch([_surface(eik, mg, 2 + i % 3, 32, i + 1) for i in range(k)])
        b.solveEikonal()
        return b

    calls = [_surface(eik, mg, 33, 16, 5), _surface(eik, mg, 5, 64, 6), _surface(eik, mg, 6, 64, 7),
             _cube(eik, mg, 9, 1), _cube(eik, mg, 25, 2), _cube(eik, mg, 17, 3, precisionMode_=1), batch(6), batch(40)]
    srv = eik.EikonalServer(hbm_budget_bytes=1 << 30, keep_results=True)
    ids = [srv.add_mesh(_surface(eik, mg, 4, 64, 1), slots=2), srv.add_mesh(_cube(eik, mg, 17, 4), slots=2)]
    srv.start()

    def outcome(c):
        if isinstance(c, eik.EikonalBatch):
            return np.concatenate(c.getFinalResults()).view(np.uint32).copy(), [c.numIterations(i) for i in range(len(c))]
        return c.getFinalResult().view(np.uint32).copy(), c.numIterations()

    def ask():
        rs = [(srv.submit(ids[k], [i], 1.0 + k), ids[k]) for i in range(3) for k in (0, 1)]
        srv.drain(timeout_ms=60000)
        assert all(c["status"] == 0 for c in srv.poll())
        return [srv.result(r, m).view(np.uint32).copy() for r, m in rs]

    want, served = [outcome(c) for c in calls], ask()
    wrong = []

    def work(c, w):
        try:
            for _ in range(12):
                c.solveEikonal()
                bits, iters = outcome(c)
                if not np.array_equal(bits, w[0]) or iters != w[1]:
                    wrong.append(type(c).__name__)
        except Exception as ex:  # reported below
            wrong.append(repr(ex))

    ts = [threading.Thread(target=work, args=x) for x in zip(calls, want)]
    for t in ts:
        t.start()
    while any(t.is_alive() for t in ts):
        if not all(np.array_equal(a, b) for a, b in zip(ask(), served)):
            wrong.append("served")
    for t in ts:
        t.join()
    srv.close()
    assert not wrong
