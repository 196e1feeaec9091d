"""The work that users of this solver have it do, as cases that can be timed.

Every case is a whole call through the Python classes (Eikonal, EikonalBatch,
EikonalServer): the solve, and the travel times read back to the host, which is where
the reference's callers take them.  Sizes follow the repository's own workloads (the
33 x 33 grid, the 17^3 to 97^3 jittered cubes, icospheres of levels 2 to 7, the
256-icosphere batch, the request pool, the sliver mesh).

Keys of a case:
  kind       tri / tet: one handle solved again and again (prepare holds the handle)
             fresh3d: a new handle for every solve, as a command-line program has it
             batch: many meshes in one EikonalBatch
             serve: requests to an EikonalServer's resident pool
             prec: the mixed FP32/FP64 precision mode on a mesh with slivers
  mesh, n    grid / jgrid (jittered grid, obtuse corners): n x n vertices;
             ico: icosphere of level n; cube: n^3 vertices,
             layers: the same with a tenth of its layers squeezed into slivers
  vpb        vertices per block;  seeds: seed vertices (surfaces: vertex 0 and these;
             0: a cube's middle vertex);  cap: iteration cap
  metric     1: a scalar per tet, 6: an anisotropic metric per tet, 0: speed 1
  history    per-iteration snapshots kept (the reference's, and this class's, default)
  renew      speeds handed over anew before every solve (an inversion's loop)
  pinned     times read back into a pinned buffer of the caller's
"""
import importlib
import math

import numpy as np
import torch

E = importlib.import_module("sci-solver_eikonal_gb300")
mg = importlib.import_module("sci-solver_eikonal_gb300.meshgen")


def listed():
    return [
        # the smallest 2D solve: a 33 x 33 grid, one seed, launches and latency only
        dict(name="tri grid 33x33", kind="tri", mesh="grid", n=33, vpb=16, seeds=1, metric=0, history=False, cap=100),
        # an ordinary surface with every option at its default (history kept, cap 100)
        dict(name="tri icosphere 5 defaults", kind="tri", mesh="ico", n=5, vpb=64, seeds=1, metric=1, history=True,
             cap=100),
        # a surface with obtuse corners (virtual faces), odd size, several seeds
        dict(name="tri obtuse 151x151", kind="tri", mesh="jgrid", n=151, vpb=32, seeds=4, metric=1, history=False,
             cap=1000),
        # the largest 2D mesh of the request pool
        dict(name="tri icosphere 7", kind="tri", mesh="ico", n=7, vpb=64, seeds=8, metric=1, history=False, cap=1000),
        # a small volume with every option at its default
        dict(name="tet cube 17 defaults", kind="tet", mesh="cube", n=17, vpb=64, seeds=3, metric=1, history=True,
             cap=100),
        # a program that loads one mesh, solves it once and ends: set-up and solve
        dict(name="tet cube 33 one solve", kind="fresh3d", mesh="cube", n=33, vpb=64, seeds=1, metric=1, history=True,
             cap=100),
        # anisotropic metrics handed over anew before every solve, as an inversion does
        dict(name="tet cube 41 new metrics", kind="tet", mesh="cube", n=41, vpb=64, seeds=4, metric=6, history=False,
             cap=1000, renew=True),
        # the headline solve: 1.57 M tets, the seed in the middle
        dict(name="tet cube 65", kind="tet", mesh="cube", n=65, vpb=64, seeds=0, metric=1, history=False, cap=100,
             pinned=True),
        # the largest volume of the request pool, with a request's 16 seeds
        dict(name="tet cube 97", kind="tet", mesh="cube", n=97, vpb=64, seeds=16, metric=1, history=False, cap=1000,
             pinned=True),
        # mixed precision on a mesh with slivers and anisotropic metrics
        dict(name="precision sliver 25", kind="prec", mesh="layers", n=25, vpb=64, seeds=4, metric=6, history=False,
             cap=1000),
        # many uneven surfaces in one call
        dict(name="batch 256 icospheres", kind="batch", mesh="ico", n=2, n_hi=6, count=256, mesh_seed=3, vpb=32,
             seeds=8, metric=1, history=False, cap=1000, pinned=True),
        # a burst of requests to a mixed resident pool
        dict(name="serve 32 requests", kind="serve", mesh="pool", count=32, mesh_seed=7, vpb=64, seeds=16, metric=1,
             history=False, cap=1000, ico="5,6", cube="33,49", slots=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tri"] * 5 + ["tet"] * 8 + ["fresh3d", "batch", "batch", "batch3d", "serve", "prec"])
    c = dict(kind=kind, vpb=rng.choice([32, 64, 64, 128]), seeds=_log_int(rng, 1, 16), metric=1, history=False,
             cap=1000)
    if kind == "tri":
        c["mesh"] = rng.choice(["grid", "ico", "jgrid"])
        c["n"] = rng.randint(2, 7) if c["mesh"] == "ico" else _log_int(rng, 9, 400)
        if c["mesh"] != "ico":
            c["vpb"] = 32 if c["seeds"] >= 4 and rng.random() < 0.6 else 16
        elif c["n"] == 2:
            c["vpb"] = 32
        c["metric"] = rng.choice([0, 1, 1])
        c["history"] = rng.random() < 0.3 and (c["n"] <= 5 if c["mesh"] == "ico" else c["n"] <= 128)
    elif kind in ("tet", "fresh3d"):
        c["mesh"] = "cube"
        c["n"] = _log_int(rng, 7, 90 if kind == "tet" else 45)
        c["metric"] = rng.choice([0, 1, 1, 6]) if c["n"] <= 49 else 1
        c["history"] = rng.random() < 0.3 and c["n"] <= 41
        c["renew"] = kind == "tet" and rng.random() < 0.25
        c["pinned"] = rng.random() < 0.5
    elif kind == "batch":
        c.update(mesh="ico", n=2, n_hi=rng.randint(3, 6), count=_log_int(rng, 4, 200), mesh_seed=rng.randint(0, 9999),
                 vpb=32, pinned=True)
    elif kind == "batch3d":
        c.update(kind="batch", mesh="cube", n=7, n_hi=rng.randint(11, 25), count=_log_int(rng, 4, 32),
                 mesh_seed=rng.randint(0, 9999), vpb=64, pinned=True)
    elif kind == "serve":
        c.update(mesh="pool", count=rng.randint(4, 30), mesh_seed=rng.randint(0, 9999), vpb=64,
                 ico="%d" % rng.randint(3, 6), cube="%d,%d" % (rng.randint(9, 25), rng.randint(26, 45)),
                 slots=rng.randint(1, 4))
    else:
        c.update(mesh="layers", n=rng.randint(9, 24), vpb=64, seeds=rng.randint(1, 8), metric=6)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rng(*key):
    return np.random.Generator(np.random.PCG64(list(key)))


def _jittered_grid(n, seed):
    xyz, faces = mg.grid2d(n)
    d = _rng(seed, 11).uniform(-0.3, 0.3, size=(n, n, 2)) / (n - 1)
    d[0] = d[-1] = 0
    d[:, 0] = d[:, -1] = 0
    xyz = xyz.astype(np.float64)
    xyz[:, :2] += d.reshape(-1, 2)
    return xyz.astype(np.float32), faces


def _layered_cube(n, seed):
    """A jittered cube whose tets are slivers in a tenth of its layers along z (at
    least one), flattened to 2-5% of the others' height, as boundary layers are."""
    h = 1.0 / (n - 1)
    xyz, tets = mg.kuhn_cube(n, 0.0)
    g = _rng(seed, 17)
    height = np.ones(n - 1)
    thin = g.choice(n - 1, size=max(1, (n - 1) // 10), replace=False)
    height[thin] = g.uniform(0.02, 0.05, size=thin.size)
    z = np.concatenate([[0.0], np.cumsum(height)]) * h
    k = np.arange(n ** 3) // (n * n)
    room = np.minimum(height[np.maximum(k - 1, 0)], height[np.minimum(k, n - 2)]) * h
    d = g.uniform(-0.2, 0.2, size=(n ** 3, 3)) * np.stack([np.full(n ** 3, h), np.full(n ** 3, h), room], 1)
    p = xyz.astype(np.float64)
    d[(p <= 0.0) | (p >= 1.0)] = 0.0
    p[:, 2] = z[k]
    return (p + d).astype(np.float32), tets


def _geometry(mesh, n, seed):
    if mesh == "grid":
        return mg.grid2d(n)
    if mesh == "jgrid":
        return _jittered_grid(n, seed)
    if mesh == "ico":
        return mg.icosphere(n)
    if mesh == "cube":
        return mg.kuhn_cube(n, 0.2, seed=seed)
    if mesh == "layers":
        return _layered_cube(n, seed)
    raise ValueError(mesh)


def _speeds(metric, xyz, elems, seed):
    """What initSpeedMtxMultipliers takes: smooth face speeds with a phase of the
    seed's (2D), 1/v^2 of log-uniform speeds or anisotropic metrics (3D)."""
    if metric == 0:
        return None
    if elems.shape[1] == 3:
        c = xyz[elems].mean(axis=1).astype(np.float64)
        p = _rng(seed, 12).uniform(0, 2 * np.pi, 3)
        return (1 + 0.5 * np.sin(3 * c[:, 0] + p[0]) * np.cos(2 * c[:, 1] + p[1]) * np.sin(c[:, 2] + p[2])).astype(
            np.float32)
    if metric == 6:
        return mg.anisotropic_metrics(elems.shape[0], seed=seed)
    v = mg.log_uniform_speeds(elems.shape[0], 0.5, 2.0, seed=seed)
    return (1.0 / v.astype(np.float64) ** 2).astype(np.float32)


def _seeds(nv, per, k, seed):
    """k seed vertices; on surfaces vertex 0, the reference's default seed, and k
    others.  (The 2D scheme can end early from a seed deep inside a block; with
    vertex 0 and the block sizes above it covers the mesh, as a user wants it to.)"""
    s = _rng(seed, 13).choice(nv, size=min(k, nv), replace=False)
    return np.unique(np.append(s, 0) if per == 3 else s).astype(np.int32)


def _problem(case, seed):
    xyz, elems = _geometry(case["mesh"], case["n"], seed)
    seeds = (_seeds(xyz.shape[0], elems.shape[1], case["seeds"], seed) if case["seeds"] else
             np.array([mg.center_vertex(case["n"])], dtype=np.int32))
    return xyz, elems, _speeds(case["metric"], xyz, elems, seed), seeds


def _batch_problems(case, seed):
    g = _rng(case["mesh_seed"], 14)
    out = []
    for i in range(case["count"]):
        n = int(g.integers(case["n"], case["n_hi"] + 1))
        k = int(g.integers(1, case["seeds"] + 1))
        xyz, elems = _geometry(case["mesh"], n, seed * 1000 + i)
        out.append((xyz, elems, _speeds(case["metric"], xyz, elems, seed * 1000 + i),
                    _seeds(xyz.shape[0], elems.shape[1], k, seed * 1000 + i)))
    return out


def _pool(case, seed):
    meshes = [("ico", int(n)) for n in case["ico"].split(",")] + [("cube", int(n)) for n in case["cube"].split(",")]
    pool = []
    for i, (mesh, n) in enumerate(meshes):
        xyz, elems = _geometry(mesh, n, seed + i)
        pool.append((xyz, elems, _speeds(1, xyz, elems, seed + i)))
    g = _rng(case["mesh_seed"], 15)
    which = [int(g.integers(0, len(pool))) for _ in range(case["count"])]
    h = _rng(seed, 16)
    requests = []
    for i, m in enumerate(which):
        k = int(h.integers(1, case["seeds"] + 1))
        scale = float(np.float32(math.exp(h.uniform(math.log(0.5), math.log(2.0)))))
        requests.append((m, _seeds(pool[m][0].shape[0], pool[m][1].shape[1], k, seed * 1000 + i), scale))
    return pool, requests


def _handle(case, xyz, elems, speeds, seeds):
    e = E.Eikonal(elems.shape[1] == 3)
    e.set_mesh(xyz, elems)
    e.maxVertsPerBlock_ = case["vpb"]
    e.maxIterations_ = case["cap"]
    if not case["history"]:
        e.keepHistory_ = 0
    if case["kind"] == "prec":
        e.precisionMode_ = 1
    if speeds is not None:
        e.initSpeedMtxMultipliers(speeds)
    if seeds is not None:
        e.setSeeds(seeds)
    return e


def _pinned(n):
    return torch.empty(n, dtype=torch.float32, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "batch":
        s["handles"] = [_handle(case, *p) for p in _batch_problems(case, seed)]
        s["batch"] = E.EikonalBatch(s["handles"])
        s["out"] = _pinned(sum(e.numVertices() for e in s["handles"]))
    elif case["kind"] == "serve":
        pool, s["requests"] = _pool(case, seed)
        s["server"] = E.EikonalServer(hbm_budget_bytes=8 << 30, keep_results=True)
        s["ids"] = [s["server"].add_mesh(_handle(case, *p, None), case["slots"]) for p in pool]
        s["server"].start()
    else:
        s["input"] = _problem(case, seed)
        if case["kind"] != "fresh3d":
            s["handle"] = _handle(case, *s["input"])
        s["out"] = _pinned(s["input"][0].shape[0]) if case.get("pinned") else None
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "batch":
        s["batch"].solveEikonal()
        s["batch"].getFinalResults(out=s["out"])
        return {"t": s["out"], "iterations": np.array([s["batch"].numIterations(i) for i in range(len(s["batch"]))])}
    if case["kind"] == "serve":
        srv, ids = s["server"], s["ids"]
        asked = [srv.submit(ids[m], seeds, scale) for m, seeds, scale in s["requests"]]
        done = {}
        while len(done) < len(asked):
            for c in srv.poll(wait_ms=1000):
                if c["status"]:
                    raise RuntimeError("request failed: %r" % (c,))
                done[c["id"]] = c["iterations"]
        return {"t": [srv.result(r, ids[q[0]]) for r, q in zip(asked, s["requests"])],
                "iterations": np.array([done[r] for r in asked])}
    e = _handle(case, *s["input"]) if case["kind"] == "fresh3d" else s["handle"]
    if case.get("renew") and s["input"][2] is not None:
        e.initSpeedMtxMultipliers(s["input"][2])
    e.solveEikonal()
    out = {"t": e.getFinalResult(out=s["out"]), "iterations": e.numIterations()}
    if case["history"]:
        out["half"] = e.getResultAtIteration(e.numIterations() // 2)
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _counts(mesh, n):
    """Vertices, elements, corners per element."""
    if mesh in ("grid", "jgrid"):
        return n * n, 2 * (n - 1) ** 2, 3
    if mesh == "ico":
        return 10 * 4 ** n + 2, 20 * 4 ** n, 3
    return n ** 3, 6 * (n - 1) ** 3, 4


def work(case):
    """Each vertex's coordinates and each element's corners and speed read once, each
    travel time written once; each corner's update from its element run once (about
    50 operations a triangle corner, 300 a tet corner)."""
    if case["kind"] == "batch":
        g = _rng(case["mesh_seed"], 14)
        sizes = []
        for _ in range(case["count"]):
            sizes.append(_counts(case["mesh"], int(g.integers(case["n"], case["n_hi"] + 1))))
            g.integers(1, case["seeds"] + 1)
    elif case["kind"] == "serve":
        pool = [("ico", int(n)) for n in case["ico"].split(",")] + [("cube", int(n)) for n in case["cube"].split(",")]
        g = _rng(case["mesh_seed"], 15)
        sizes = [_counts(*pool[int(g.integers(0, len(pool)))]) for _ in range(case["count"])]
    else:
        sizes = [_counts(case["mesh"], case["n"])]
    nbytes = sum(4 * (4 * nv + ne * (c + max(case["metric"], 0))) for nv, ne, c in sizes)
    return {"bytes": nbytes, "flops": sum(ne * c * (50 if c == 3 else 300) for _, ne, c in sizes)}


# ---------------------------------------------------------------------------
# the travel times in 64 bits: the smallest times that no element's update lowers
# ---------------------------------------------------------------------------
_FAR = 1e9


def _edge(TP, TQ, PP, PQ, QQ):
    """Least time at the apex from the segment P-Q: points of it are Q + a (P - Q);
    PP, PQ, QQ: the metric products of P - apex and Q - apex."""
    G = PP - 2 * PQ + QQ          # |P - Q|^2
    w = (QQ - PQ) / G             # foot of the apex on the line
    h2 = (QQ - w * w * G).clamp_min(0)
    t = TP - TQ
    s = t * t / G
    a = w - torch.sqrt(h2 / (1 - s).clamp_min(1e-300)) * t / G
    ok = (s < 1) & (a >= 0) & (a <= 1)
    a = torch.where(ok, a, torch.zeros_like(a))
    f = TQ + a * t + torch.sqrt((a * a * PP + 2 * a * (1 - a) * PQ + (1 - a) ** 2 * QQ).clamp_min(0))
    ends = torch.minimum(TP + torch.sqrt(PP), TQ + torch.sqrt(QQ))
    return torch.minimum(torch.where(ok, f, ends), ends)


def _face(TA, TB, TC, AA, AB, AC, BB, BC, CC):
    """Least time at the apex from the triangle A B C (products of A - apex, ...)."""
    best = torch.minimum(torch.minimum(_edge(TA, TB, AA, AB, BB), _edge(TA, TC, AA, AC, CC)),
                         _edge(TB, TC, BB, BC, CC))
    g11, g12, g22 = AA - 2 * AC + CC, AB - AC - BC + CC, BB - 2 * BC + CC
    r1, r2 = CC - AC, CC - BC
    det = g11 * g22 - g12 * g12
    w1, w2 = (g22 * r1 - g12 * r2) / det, (g11 * r2 - g12 * r1) / det
    h2 = (CC - w1 * r1 - w2 * r2).clamp_min(0)
    t1, t2 = TA - TC, TB - TC
    u1, u2 = (g22 * t1 - g12 * t2) / det, (g11 * t2 - g12 * t1) / det
    s = t1 * u1 + t2 * u2
    k = torch.sqrt(h2 / (1 - s).clamp_min(1e-300))
    a, b = w1 - k * u1, w2 - k * u2
    c = 1 - a - b
    ok = (s < 1) & (det > 0) & (a >= 0) & (b >= 0) & (c >= 0)
    q = a * a * AA + b * b * BB + c * c * CC + 2 * (a * b * AB + a * c * AC + b * c * BC)
    f = a * TA + b * TB + c * TC + torch.sqrt(q.clamp_min(0))
    return torch.where(ok, torch.minimum(f, best), best)


def _fixed_point(xyz, elems, speeds, seeds, scale=1.0):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.as_tensor(xyz, device=dev).double()
    el = torch.as_tensor(elems, device=dev).long()
    nv, per = x.shape[0], el.shape[1]
    if per == 3:
        F2 = torch.ones(el.shape[0], device=dev, dtype=torch.float64)
        if speeds is not None:
            F2 = (torch.as_tensor(speeds, device=dev).double() * scale) ** -2
        M = None
    else:
        M = torch.ones(el.shape[0], 1, device=dev, dtype=torch.float64)
        if speeds is not None:
            M = torch.as_tensor(speeds, device=dev).double().reshape(el.shape[0], -1)
        M = M * float(np.float32(1.0 / (scale * scale)))
    T = torch.full((nv,), _FAR, device=dev, dtype=torch.float64)
    T[torch.as_tensor(seeds, device=dev).long()] = 0
    changed = T < _FAR
    for _ in range(20000):
        if not bool(changed.any()):
            break
        on = torch.nonzero(changed[el].any(1))[:, 0]
        new = T.clone()
        for part in torch.split(on, 1 << 20):
            e = el[part]
            P, t = x[e], T[e]
            for k in range(per):
                o = [j for j in range(per) if j != k]
                d = [P[:, j] - P[:, k] for j in o]
                if per == 3:
                    f2 = F2[part]

                    def dot(u, v):
                        return (u * v).sum(1) * f2
                else:
                    m = M[part]

                    def dot(u, v):
                        if m.shape[1] == 1:
                            return (u * v).sum(1) * m[:, 0]
                        return (u[:, 0] * (m[:, 0] * v[:, 0] + m[:, 1] * v[:, 1] + m[:, 2] * v[:, 2]) +
                                u[:, 1] * (m[:, 1] * v[:, 0] + m[:, 3] * v[:, 1] + m[:, 4] * v[:, 2]) +
                                u[:, 2] * (m[:, 2] * v[:, 0] + m[:, 4] * v[:, 1] + m[:, 5] * v[:, 2]))
                if per == 3:
                    c = _edge(t[:, o[0]], t[:, o[1]], dot(d[0], d[0]), dot(d[0], d[1]), dot(d[1], d[1]))
                else:
                    c = _face(t[:, o[0]], t[:, o[1]], t[:, o[2]], dot(d[0], d[0]), dot(d[0], d[1]), dot(d[0], d[2]),
                              dot(d[1], d[1]), dot(d[1], d[2]), dot(d[2], d[2]))
                new.scatter_reduce_(0, e[:, k], c, "amin")
        changed = new < T - 1e-12
        T = new
    return T


def _union(problems):
    xs, es, ss, sd, off = [], [], [], [], 0
    for xyz, elems, speeds, seeds in problems:
        xs.append(xyz)
        es.append(elems + off)
        ss.append(speeds)
        sd.append(seeds + off)
        off += xyz.shape[0]
    return np.concatenate(xs), np.concatenate(es), np.concatenate(ss), np.concatenate(sd)


def exact(case, seed):
    if case["kind"] == "batch":
        return {"t": _fixed_point(*_union(_batch_problems(case, seed))), "iterations": None}
    if case["kind"] == "serve":
        pool, requests = _pool(case, seed)
        return {"t": [_fixed_point(*pool[m], seeds, scale) for m, seeds, scale in requests], "iterations": None}
    if case["mesh"] == "jgrid":
        return None  # obtuse corners: the scheme's virtual faces are not the mesh's
    out = {"t": _fixed_point(*_problem(case, seed)), "iterations": None}
    if case["history"]:
        out["half"] = None
    return out
