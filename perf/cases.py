"""Timed cases: the work a user of galpha_b200 has it do, through its public entry points.

A case is a dict of plain values with a "kind":

  call      galphaComputeAll on host points: triangulation + alpha arrays back on the host in one call
            ("lines" > 0: with constrained edges, GPUDTPARAMS.nConstraints)
  mesh      galphaCompute + galphaMasterList of a given host triangulation (the reference's main)
  device    Engine.run_device on points in device memory, then alpha queries at the spectrum quantiles
            0.1 / 0.5 / 0.9 on the resident mesh and the points' classes at the last of them ("fetch": the alpha
            arrays are downloaded instead, galphaComputeResident)
  batch     Engine.run_batch_device: many independent sets at once, then Engine.batch_query and the classes
  host      galphaRunBatchHost on host sets, and galphaBatchCopy of every result
  serve     one micro-batch of the request loop: Engine.run_batch on host sets, three Engine.batch_query

Results that go to the host go to pinned buffers of the caller, sized for the largest result of that many points
and kept with the inputs (what lies past a result stays zero).  The order of a triangulation's triangles, and
with it the numbering of its edges, is not reproducible from run to run, so the cases that triangulate return
what does not depend on it: the spectrum and the point intervals, or the query results, classes and counts.  The
mesh case is given its triangles in a fixed order and returns everything.

Points follow the recipes of galpha_b200.datasets (uniform square, disk, annulus, Gaussian blobs, the degenerate
mix of blobs, uniform and lattice points), drawn on the device from the seed.
"""
import ctypes
import math

import numpy as np
import torch

import galpha_b200 as G
from galpha_b200 import api

QUANTILES = (0.1, 0.5, 0.9)
_QUERY = np.dtype([("alpha", "f8"), ("rank", "i4"), ("counts", "i4", 12), ("pad", "i4")])  # galphaQueryResult
_KINDS = ("uniform", "disk", "annulus")
_kept = []


def listed():
    return [
        # the smallest benchmark configuration: one call of 1,000 points, latency and launches only
        {"name": "call_1k", "kind": "call", "n": 1000, "dist": "uniform", "fbo": 512, "lines": 0},
        # an ordinary call at the default texture size
        {"name": "call_50k", "kind": "call", "n": 49999, "dist": "uniform", "fbo": 2048, "lines": 0},
        # a large call with every result copied back to the host
        {"name": "call_1m", "kind": "call", "n": 1048575, "dist": "uniform", "fbo": 4096, "lines": 0},
        # break lines through a terrain: the constrained triangulation at the size of the constraint tests
        {"name": "constrained_20k", "kind": "call", "n": 20011, "dist": "uniform", "fbo": 1024, "lines": 10},
        # the reference program's sequence: alpha shapes and master list of a triangulation the caller holds
        {"name": "mesh_30k", "kind": "mesh", "n": 30011, "dist": "uniform", "fbo": 1024},
        # a small set resident on the device with repeated queries (the viewer's and the request loop's use)
        {"name": "device_12k", "kind": "device", "n": 12289, "dist": "disk", "fbo": 512, "fetch": False},
        # clustered points (half of the request stream), alpha arrays fetched
        {"name": "device_262k_blobs", "kind": "device", "n": 262145, "dist": "blobs", "fbo": 2048, "fetch": True},
        # the headline configuration: 4,194,304 uniform points on the largest ordinary texture
        {"name": "device_4m", "kind": "device", "n": 4194304, "dist": "uniform", "fbo": 8192, "fetch": False},
        # the precision stress: 16,777,216 points with duplicates, cocircular and collinear runs
        {"name": "device_16m_mix", "kind": "device", "n": 16777216, "dist": "mix", "fbo": 8192, "fetch": False},
        # the batched configuration's size range, a quarter of its sets
        {"name": "batch_1024", "kind": "batch", "sets": 1024, "lo": 64, "hi": 65536},
        # a small batch whose results all go back to the host
        {"name": "host_30", "kind": "host", "sets": 30, "lo": 64, "hi": 8192},
        # a micro-batch of the request stream: 1,000 to 1,048,576 points, half of the sets clustered
        {"name": "serve_24", "kind": "serve", "sets": 24, "lo": 1000, "hi": 1048576},
    ]


def _texture(n):
    """The texture the benchmark gives a set of n points."""
    fbo = 256
    while fbo < 8192 and fbo * fbo < 16 * n:
        fbo *= 2
    return fbo


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(("call", "call", "constrained", "mesh", "device", "device", "device", "batch", "host", "serve"))
    if kind in ("call", "constrained"):
        n = size(1000, 1 << 20) if kind == "call" else size(3000, 100000)
        dist = rng.choice(("uniform", "disk", "annulus", "blobs")) if kind == "call" else "uniform"
        lines = 0 if kind == "call" else rng.randint(2, 16)
        return {"kind": "call", "n": n, "dist": dist, "fbo": _texture(n), "lines": lines}
    if kind == "mesh":
        n = size(1000, 200000)
        return {"kind": kind, "n": n, "dist": rng.choice(_KINDS), "fbo": _texture(n)}
    if kind == "device":
        n = size(1000, 1 << 22)
        return {"kind": kind, "n": n, "dist": rng.choice(_KINDS + ("blobs", "mix")), "fbo": _texture(n),
                "fetch": rng.random() < 0.3}
    if kind == "batch":
        return {"kind": kind, "sets": size(32, 1024), "lo": 64, "hi": size(4096, 65536)}
    if kind == "host":
        return {"kind": kind, "sets": rng.randint(4, 30), "lo": 64, "hi": size(1024, 65536)}
    return {"kind": kind, "sets": rng.randint(4, 28), "lo": 1000, "hi": size(65536, 1 << 20)}


# ------------------------------------------------------------------ inputs
def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _blobs(n, g):
    centres = _rand(g, 64, 2)
    pick = torch.randint(0, 64, (n,), generator=g, device="cuda")
    return centres[pick] + 0.01 * torch.randn(n, 2, generator=g, device="cuda", dtype=torch.float64)


def _points(n, dist, g):
    if dist == "uniform":
        return _rand(g, n, 2)
    if dist == "blobs":
        return _blobs(n, g)
    if dist == "mix":  # half blobs, 30 % uniform, 20 % on a 1024 x 1024 lattice
        nb, nu = n // 2, 3 * n // 10
        return torch.cat([_blobs(nb, g), _rand(g, nu, 2), torch.floor(1024.0 * _rand(g, n - nb - nu, 2)) / 1024.0])
    u, th = _rand(g, n), 2.0 * math.pi * _rand(g, n)
    r = torch.sqrt(u) if dist == "disk" else torch.sqrt(0.64 + 0.36 * u)
    return torch.stack([r * torch.cos(th), r * torch.sin(th)], dim=1)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _bounds(p):
    lo, hi = p.amin(0), p.amax(0)
    return tuple(torch.cat([lo, hi]).tolist())


def _pinned(p):
    host = torch.empty(p.shape, dtype=p.dtype, pin_memory=True)
    host.copy_(p)
    return host.numpy()


def _results(n, master=False):
    """Pinned result buffers for n points: rows of the element layouts of galpha.h and gpudt.h."""
    rows = {"tris": (2 * n + 64, 9), "points": (n, 2), "edges": (3 * n + 64, 6), "tri_ranks": (2 * n + 64, 1)}
    if master:
        rows.update(master=(13 * n + 256, 3), pointers=(5 * n + 256, 1))
    out = {k: torch.zeros(v, dtype=torch.int32, pin_memory=True).numpy() for k, v in rows.items()}
    out["spectrum"] = torch.zeros(5 * n + 256, dtype=torch.float64, pin_memory=True).numpy()
    return out


def _sizes(case):
    """Set sizes spread evenly over the logarithm of the range: the same total for every seed."""
    k = (np.arange(case["sets"]) + 0.5) / case["sets"]
    return np.floor(case["lo"] * (case["hi"] / case["lo"]) ** k).astype(np.int64)


def _sets(case, seed):
    g = _generator(seed)
    sizes = _sizes(case)[np.random.RandomState(seed % (1 << 32)).permutation(case["sets"])]
    if case["kind"] == "serve":
        return [_points(int(n), "blobs" if k % 2 else "uniform", g) for k, n in enumerate(sizes)]
    return [_points(int(n), _KINDS[k % 3], g) for k, n in enumerate(sizes)]


def _break_lines(p, lines):
    """Polylines that join consecutive points, by x, of thin horizontal bands: they cross neither each other nor
    a point."""
    n = len(p)
    bands = max(2 * lines, int(round(math.sqrt(n))))
    of = np.floor(p[:, 1] * bands).astype(np.int64)
    out = []
    for b in np.linspace(0, bands - 1, lines).astype(np.int64):
        idx = np.nonzero(of == b)[0]
        idx = idx[np.argsort(p[idx, 0])]
        out.append(np.stack([idx[:-1], idx[1:]], axis=1))
    return np.concatenate(out).astype(np.int32)


def _in_order(dt):
    """The triangulation with its triangles in a fixed order: each from its smallest vertex on, sorted."""
    t = torch.from_numpy(dt.triangles.view(np.int32).reshape(-1, 9)).cuda().long()
    nbr, vtx = t[:, 0:3], t[:, 3:6]
    first = vtx.argmin(1)
    turn = (first[:, None] + torch.arange(3, device="cuda")) % 3
    nbr, vtx = nbr.gather(1, turn), vtx.gather(1, turn)
    order = (vtx[:, 0] * (int(vtx.max()) + 1) + vtx[:, 1]).argsort()
    place = torch.empty_like(order)
    place[order] = torch.arange(len(order), device="cuda")
    to, edge = (nbr >> 2).clamp(min=0), nbr & 3
    nbr = torch.where(nbr < 0, nbr, (place[to] << 2) | ((edge - first[to]) % 3))
    return _pinned(torch.cat([nbr, vtx, torch.zeros_like(vtx)], 1)[order].to(torch.int32))


def _engine():
    """One handle for the life of the program, as a user keeps it."""
    if not _kept:
        _kept.append(G.Engine())
    return _kept[0]


def prepare(case, seed):
    eng, kind = _engine(), case["kind"]
    state = {"eng": eng, "kind": kind}
    if kind in ("call", "mesh"):
        p = _points(case["n"], case["dist"], _generator(seed))
        host, b = _pinned(p), _bounds(p)
        lines = _break_lines(host, case["lines"]) if case.get("lines") else None
        state["params"] = G.GPUDTParams(host, case["fbo"], b[0], b[1], b[2], b[3], constraints=lines)
        state["out"] = _results(case["n"], master=kind == "mesh")
        if kind == "mesh":
            state["tris"] = _in_order(eng.triangulate(state["params"]))
    elif kind == "device":
        p = _points(case["n"], case["dist"], _generator(seed))
        state.update(xy=p, n=case["n"], bounds=_bounds(p), fbo=case["fbo"], fetch=case["fetch"])
        if case["fetch"]:
            state["out"] = _results(case["n"])
    else:
        sets = _sets(case, seed)
        state["bounds"] = np.array([_bounds(p) for p in sets])
        state["sizes"] = np.array([len(p) for p in sets], np.int32)
        if kind == "batch":
            state["xy"] = torch.cat(sets)
        elif kind == "host":
            state["xy"], state["out"] = _pinned(torch.cat(sets)), _results(int(state["sizes"].sum()))
        else:
            state["sets"] = [p.cpu().numpy() for p in sets]
    if "out" not in state:
        n = case["n"] if "n" in case else int(state["sizes"].sum())
        state["classes"] = torch.zeros(n, dtype=torch.uint8, pin_memory=True).numpy()
    torch.cuda.synchronize()  # the engine works on a stream of its own
    return state


# ------------------------------------------------------------------ passes
def _check(status):
    if status:
        raise RuntimeError("galpha status %d: %s" % (status, G.load().galphaLastError().decode()))


def _alpha_out(buf):
    """GAlphaOutput over the caller's buffers, capacities in its counts."""
    o = api._AlphaOut()
    o.spectrum, o.nSpectrum = buf["spectrum"].ctypes.data, len(buf["spectrum"])
    o.point_list, o.nPoints = buf["points"].ctypes.data, len(buf["points"])
    o.edge_list, o.nEdges = buf["edges"].ctypes.data, len(buf["edges"])
    o.tri_list, o.nTris = buf["tri_ranks"].ctypes.data, len(buf["tri_ranks"])
    return o


def _call(state):
    buf, params, o = state["out"], state["params"]._c(), _alpha_out(state["out"])
    dt = api._Output(buf["tris"].ctypes.data, len(buf["tris"]))
    _check(G.load().galphaComputeAll(state["eng"]._h, ctypes.byref(params), ctypes.byref(dt), ctypes.byref(o), None))
    return {"counts": [dt.nTris, o.nEdges, o.nSpectrum], "spectrum": buf["spectrum"], "points": buf["points"]}


def _mesh(state):
    lib, h, buf = G.load(), state["eng"]._h, state["out"]
    params, o = state["params"]._c(), _alpha_out(buf)
    dt = api._Output(state["tris"].ctypes.data, len(state["tris"]))
    _check(lib.galphaCompute(h, ctypes.byref(params), ctypes.byref(dt), ctypes.byref(o)))
    m = api._MasterOut(len(buf["master"]), buf["master"].ctypes.data, len(buf["pointers"]), buf["pointers"].ctypes.data)
    _check(lib.galphaMasterList(h, ctypes.byref(m)))
    return dict({k: buf[k] for k in ("spectrum", "points", "edges", "tri_ranks", "master", "pointers")},
                counts=[o.nEdges, o.nSpectrum, m.nMaster, m.nSpecPointers])


def _set_counts(eng):
    """nPoints, nTris, nEdges, nSpectrum of each set of the last batch."""
    return np.frombuffer(eng.batch_sets(), np.int32).reshape(-1, 8)[:, 0::2]


def _host(state):
    eng, buf = state["eng"], state["out"]
    sizes, bounds = state["sizes"], state["bounds"]
    _check(G.load().galphaRunBatchHost(eng._h, len(sizes), sizes.ctypes.data, state["xy"].ctypes.data,
                                       bounds.ctypes.data, 1, None))
    _check(G.load().galphaBatchCopy(eng._h, *(buf[k].ctypes.data for k in ("tris", "points", "edges", "tri_ranks", "spectrum"))))
    return {"spectrum": buf["spectrum"], "points": buf["points"]}


def _answers(res):
    q = np.frombuffer(res, _QUERY)
    return [q["alpha"], q["rank"], q["counts"]]


def _point_classes(state):
    _check(G.load().galphaCopyClasses(state["eng"]._h, state["classes"].ctypes.data, None, None))
    return state["classes"]


def run(state):
    eng, kind = state["eng"], state["kind"]
    if kind in ("call", "mesh", "host"):
        return {"call": _call, "mesh": _mesh, "host": _host}[kind](state)
    if kind == "device":
        eng.run_device(state["xy"].data_ptr(), state["n"], state["bounds"], state["fbo"])
        if state["fetch"]:
            o = _alpha_out(state["out"])
            _check(G.load().galphaComputeResident(eng._h, ctypes.byref(o)))
            return {"counts": [o.nTris, o.nEdges, o.nSpectrum], "spectrum": state["out"]["spectrum"],
                    "points": state["out"]["points"]}
        out = {"counts": list(eng.counts()), "queries": [_answers(eng.query(quantile=q)) for q in QUANTILES]}
    else:
        if kind == "batch":
            eng.run_batch_device(state["xy"].data_ptr(), state["sizes"], state["bounds"])
        else:
            eng.run_batch(state["sets"], bounds=state["bounds"])
        k = len(state["sizes"])
        queries = [_answers(eng.batch_query([q] * k, by_quantile=True)) for q in QUANTILES]
        out = {"counts": _set_counts(eng), "queries": queries}
    return dict(out, classes=_point_classes(state))


def work(case):
    """Compulsory bytes: the points once, and per point 2 triangles (vertices and links), 3 edge intervals, 2
    triangle ranks, 3.9 spectrum values and 1 point interval once; the mesh case reads the triangles, and writes
    13 master-list entries and 3.9 pointers per point."""
    n = case["n"] if "n" in case else int(_sizes(case).sum())
    per_point = 16 + 2 * 24 + 3 * 24 + 2 * 4 + 3.9 * 8 + 8
    if case["kind"] == "mesh":
        per_point += 13 * 12 + 3.9 * 4
    return {"bytes": per_point * n, "flops": 0}


# ------------------------------------------------------------------ 64-bit results
def _delaunay(p):
    """Triangles (ccw) of points in general position: incremental insertion with a ghost vertex, pure Python."""
    n = len(p)
    ghost, m = n, n + 1
    x, y = p[:, 0].tolist(), p[:, 1].tolist()
    rows = max(1, int(math.sqrt(n / 2)))
    lo, hi = p.min(0), p.max(0)
    cell = np.minimum((rows * (p - lo) / (hi - lo)).astype(np.int64), rows - 1)
    along = np.where(cell[:, 1] % 2 == 0, p[:, 0], -p[:, 0])  # row by row, there and back
    order = np.lexsort((along, cell[:, 1])).tolist()

    def orient(a, b, c):
        return (x[b] - x[a]) * (y[c] - y[a]) - (y[b] - y[a]) * (x[c] - x[a])

    apex = {}  # directed edge a -> b, as a * m + b: the third vertex of the triangle left of it

    def add(a, b, c):
        apex[a * m + b], apex[b * m + c], apex[c * m + a] = c, a, b

    a, b, c = order[:3]
    if orient(a, b, c) < 0:
        b, c = c, b
    add(a, b, c)
    add(b, a, ghost), add(c, b, ghost), add(a, c, ghost)
    last = (a, b)

    def inside(a, b, c, q):
        if a == ghost:
            return orient(b, c, q) > 0
        if b == ghost:
            return orient(c, a, q) > 0
        if c == ghost:
            return orient(a, b, q) > 0
        ax, ay, bx, by, cx, cy = x[a] - x[q], y[a] - y[q], x[b] - x[q], y[b] - y[q], x[c] - x[q], y[c] - y[q]
        return ((ax * ax + ay * ay) * (bx * cy - cx * by) - (bx * bx + by * by) * (ax * cy - cx * ay)
                + (cx * cx + cy * cy) * (ax * by - bx * ay)) > 0

    for q in order[3:]:
        a, b = last
        while True:  # walk to the triangle that holds q, or to a ghost across the hull
            c = apex[a * m + b]
            if c == ghost:
                break
            if orient(c, a, q) < 0:
                a, b = a, c
            elif orient(b, c, q) < 0:
                a, b = c, b
            elif orient(a, b, q) < 0:
                a, b = b, a
            else:
                break
        c = apex[a * m + b]
        for u, v in ((a, b), (b, c), (c, a)):
            del apex[u * m + v]
        todo, rim = [(a, b), (b, c), (c, a)], []
        while todo:
            u, v = todo.pop()
            w = apex.get(v * m + u)
            if w is not None and inside(v, u, w, q):
                del apex[v * m + u], apex[u * m + w], apex[w * m + v]
                todo += [(u, w), (w, v)]
            else:
                rim.append((u, v))
        for u, v in rim:
            add(u, v, q)
        last = next((u, v) for u, v in rim if u != ghost and v != ghost)
    e = np.fromiter(apex.keys(), np.int64, len(apex))
    t = np.stack([e // m, e % m, np.fromiter(apex.values(), np.int64, len(apex))], 1)
    return t[(t.max(1) < ghost) & (t[:, 0] < t[:, 1]) & (t[:, 0] < t[:, 2])]


def _spectrum(p):
    """Sorted squared radii: circumcircles of the triangles and half lengths of the edges no apex is inside of."""
    t, q = _delaunay(p), p.astype(np.longdouble)
    a, b, c = q[t[:, 0]], q[t[:, 1]], q[t[:, 2]]

    def cross(u, v):
        return u[:, 0] * v[:, 1] - u[:, 1] * v[:, 0]

    def sq(u):
        return (u * u).sum(1)

    radii = [sq(a - b) * sq(b - c) * sq(c - a) / (4 * cross(b - a, c - a) ** 2)]
    u = np.concatenate([t[:, 0], t[:, 1], t[:, 2]])
    v = np.concatenate([t[:, 1], t[:, 2], t[:, 0]])
    w = np.concatenate([t[:, 2], t[:, 0], t[:, 1]])
    holds = ((q[u] - q[w]) * (q[v] - q[w])).sum(1) < 0
    key, index = np.unique(np.minimum(u, v) * len(p) + np.maximum(u, v), return_inverse=True)
    attached = np.zeros(len(key), bool)
    attached[index[holds]] = True
    key = key[~attached]
    radii.append(sq(q[key // len(p)] - q[key % len(p)]) / 4)
    return np.concatenate([[0.0], np.sort(np.concatenate(radii)).astype(np.float64)])


def exact(case, seed):
    """The spectra of sets in general position small enough for plain Python; the rest are whole numbers."""
    kind = case["kind"]
    n = case["n"] if "n" in case else int(_sizes(case).sum())
    if kind not in ("call", "mesh", "host", "device") or case.get("lines") or n > 150000 or case.get("dist") in ("blobs", "mix"):
        return None
    if kind == "device" and not case["fetch"]:
        return None
    sets = _sets(case, seed) if kind == "host" else [_points(n, case["dist"], _generator(seed))]
    found = np.concatenate([_spectrum(p.cpu().numpy()) for p in sets])
    spectrum = np.zeros(5 * n + 256)
    spectrum[:len(found)] = found
    return {"spectrum": spectrum}
