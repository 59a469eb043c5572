"""GPU tests of the round loops' device-side counts (shifting, missing sites,
fake removal, flips): clustered input that needs more rounds than a ring of
per-round counts holds, under schedules that read the counters after every
round, after groups of eight, and only at the end, with and without the
in-block flip tail.  The triangulation must be the oracle's every time."""
import numpy as np
import pytest

import galpha_b200 as G
from galpha_b200 import datasets as D
from dtcheck import canon_set, compare_dt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 1023, 20001])
@pytest.mark.parametrize("sched", [(1, 1, 1, 0, 1), (8, 8, 64, 0, 1), (3, 5, 7, 2000, 2001), (0, 0, 0, -1, 0)])
def test_rounds_under_schedules(n, sched):
    pts = D.gaussian_blobs(n, 17, nblobs=3, sigma=0.02)
    pts[::7] = D.uniform_points(len(pts[::7]), 18) * 2.0 - 1.0  # far points: long chains of flips
    eng = G.Engine()
    try:
        eng.set_schedule(*sched)
        for _ in range(2):  # the handle's second call starts from the first one's words
            dt = eng.triangulate(G.GPUDTParams(pts, fboSize=256))
            assert canon_set(dt.vtx) == canon_set(O.dt(pts)[0])
    finally:
        eng.close()
    if n > 20000 and sched[2] == 1:
        assert dt.status.flipRounds > 16 and dt.status.missingRounds > 2


@pytest.mark.parametrize("row", [200, 511, 513, 1000])
def test_hull_vertex_with_a_long_fan(engine, row):
    """A far point over a collinear row sees every segment of it, so its fan on
    the hull is as long as the row; the walks to its hull neighbours must reach
    the ends (they once gave up after 512 triangles)."""
    y = np.arange(row + 1) / 4096.0
    line = np.stack([np.zeros(row + 1), y], axis=1)
    rest = D.uniform_points(4000, row) * [1.0, y[-1]] + [1e-3, 0.0]
    far = np.array([[-0.6 * y[-1], 0.47 * y[-1]], [-0.7 * y[-1], 0.53 * y[-1]]])
    pts = np.concatenate([line, rest, far])
    dt = engine.triangulate(G.GPUDTParams(pts, fboSize=4096))
    ok, rep = compare_dt(pts, dt.vtx, dt.tri)
    assert ok, rep


@pytest.mark.parametrize("limit", [-1, 0])
@pytest.mark.parametrize("n,fbo", [(2500, 1024), (5500, 1024), (6500, 1024), (9500, 4096)])
def test_bad_sites_with_long_fans(engine, n, fbo, limit):
    """Points on a circle: thousands of unshiftable sites side by side, whose fans
    grow with every neighbour removed before them, past 64 triangles (the length
    that removal once had room for).  In one launch and in launches."""
    th = np.linspace(0.0, 2.0 * np.pi, n, endpoint=False) + 0.001
    pts = np.stack([np.cos(th), np.sin(th)], axis=1)
    engine.set_cluster_limit(limit)
    try:
        dt = engine.triangulate(G.GPUDTParams(pts, fboSize=fbo))
    finally:
        engine.set_cluster_limit(-1)
    assert dt.status.nBadShift > 1000
    ok, rep = compare_dt(pts, dt.vtx, dt.tri)
    assert ok, rep


@pytest.mark.parametrize("limit", [-1, 0])
@pytest.mark.parametrize("n,fbo", [(3500, 2048), (5000, 512), (7000, 2048)])
def test_points_in_one_pixel(engine, n, fbo, limit):
    """Three clusters that each fall into a pixel or two: all their points are
    located from the one site that owns the pixel, whose fan grows past 256
    triangles (the length after which location once gave up)."""
    c = D.uniform_points(n, 4) * 0.001
    pts = np.concatenate([c, c + [0.9, 0.9], c * [1, -1] + [0.0, 0.9]])
    engine.set_cluster_limit(limit)
    try:
        dt = engine.triangulate(G.GPUDTParams(pts, fboSize=fbo))
    finally:
        engine.set_cluster_limit(-1)
    assert dt.status.nMissing > 2 * n
    assert canon_set(dt.vtx) == canon_set(O.dt(pts)[0])


@pytest.mark.parametrize("limit", [-1, 0])
@pytest.mark.parametrize("n,fbo", [(300, 512), (1500, 2048), (6000, 4096)])
def test_hub_of_a_ring(engine, n, fbo, limit):
    """A point in the middle of a ring sees every point of it; with others beside
    it, so that it is shifted, and located through, with that fan."""
    th = np.linspace(0.0, 2.0 * np.pi, n, endpoint=False) + 0.01
    ring = np.stack([np.cos(th), np.sin(th)], axis=1) * (1.0 + 1e-5 * np.sin(5.0 * th))[:, None]
    pts = np.concatenate([ring, [[1e-4, 2e-4]], 1e-5 * D.uniform_points(40, n)])
    engine.set_cluster_limit(limit)
    try:
        dt = engine.triangulate(G.GPUDTParams(pts, fboSize=fbo))
    finally:
        engine.set_cluster_limit(-1)
    assert canon_set(dt.vtx) == canon_set(O.dt(pts)[0])
