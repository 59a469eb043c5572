"""GPU tests of the alpha stage at the edges of its tiles (1,024 triangles) and
of the scans' tiles (4,096 elements): triangle counts just below, on and above
one and several tiles, against the CPU oracle; and the same handle back and
forth between sizes, whose scans and tiles must not see one another's words."""
import pytest

import galpha_b200 as G
from galpha_b200 import datasets as D
from alphacheck import compare_alpha

pytestmark = pytest.mark.gpu


def _check(engine, n, want):
    """n points on a convex arc plus interior ones give a chosen triangle count."""
    import numpy as np

    h = 4 + (2 * n - 6 - want)  # hull vertices: 2 n - 2 - h triangles
    th = np.linspace(0.1, 0.1 + 2 * np.pi, h, endpoint=False)
    hull = np.stack([np.cos(th), np.sin(th)], axis=1) * (1.0 + 1e-3 * np.sin(37.0 * th))[:, None]
    pts = np.concatenate([hull, (D.uniform_points(n - h, n) - 0.5) * 0.9])
    dt = engine.triangulate(G.GPUDTParams(pts, fboSize=1024))
    ok, rep = compare_alpha(pts, dt.vtx, dt.tri, engine.alpha_resident(), 4)
    assert ok, rep
    return dt.nTris


@pytest.mark.parametrize("want", [1022, 1023, 1024, 1025, 2048, 2049, 4096, 4097])
def test_alpha_tile_edges(engine, want):
    n = (want + 6) // 2 + 8
    got = _check(engine, n, want)
    assert abs(got - want) <= 8  # a slightly dented arc may lose a few hull vertices
    _check(engine, 20000, 2 * 20000 - 6 - 10)
    assert _check(engine, n, want) == got


@pytest.mark.parametrize("n", [3, 4, 5, 33])
def test_alpha_smallest(engine, n):
    pts = D.uniform_points(n, 7 * n)
    dt = engine.triangulate(G.GPUDTParams(pts, fboSize=256))
    ok, rep = compare_alpha(pts, dt.vtx, dt.tri, engine.alpha_resident(), 4)
    assert ok, rep


@pytest.mark.parametrize("n", [500, 80000])
def test_undecided_predicates(engine, n):
    """Points of an integer grid: right and straight angles and cocircular fours
    everywhere, so the filters of the in-circle and the attached test leave much
    to the exact stage, with one triangle per thread and with four."""
    import numpy as np
    from dtcheck import compare_dt

    side = int(2 * n ** 0.5)
    ids = np.random.default_rng(n).permutation(side * side)[:n]
    pts = np.stack([ids % side, ids // side], axis=1) / 1024.0
    dt = engine.triangulate(G.GPUDTParams(pts, fboSize=1024))
    ok, rep = compare_dt(pts, dt.vtx, dt.tri)
    assert ok, rep
    assert dt.status.exactIncircle > 0
    ok, rep = compare_alpha(pts, dt.vtx, dt.tri, engine.alpha_resident(), 4)
    assert ok, rep


@pytest.mark.parametrize("n", [302000, 304500])
def test_vertex_intervals_by_block(engine, n):
    """Either side of 606,208 triangles, from where a block combines its
    triangles' contributions to a vertex before they go to global memory; a hub
    of high degree and a far cluster make vertices that many blocks share."""
    import numpy as np

    th = np.linspace(0.0, 2.0 * np.pi, 200, endpoint=False)
    ring = np.stack([np.cos(th), np.sin(th)], axis=1) * 0.3
    rest = D.uniform_points(n - 201, n) * 2.0 - 1.0
    rest = rest[np.hypot(rest[:, 0], rest[:, 1]) > 0.31]
    pts = np.concatenate([ring, [[1e-4, 2e-4]], rest, D.uniform_points(n - 201 - len(rest), n + 1) * 0.01 + 0.9])
    dt = engine.triangulate(G.GPUDTParams(pts, fboSize=2048))
    assert (dt.nTris < 606208) == (n < 303000)
    ok, rep = compare_alpha(pts, dt.vtx, dt.tri, engine.alpha_resident(), 4)
    assert ok, rep
