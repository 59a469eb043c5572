"""GPU tests of the mesh stages that run in one launch (a thread-block cluster):
vertex counts just below, on and above the sizes at which the cluster grows, a
stage goes back to launches of its own, or the missing sites are handed back;
fans too long for the shared arrays; constraints between the stages; several
handles at once.  The triangulation must be the oracle's every time."""
import threading

import numpy as np
import pytest

import galpha_b200 as G
from galpha_b200 import datasets as D
from dtcheck import canon_set, compare_dt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(engine, pts, fbo):
    dt = engine.triangulate(G.GPUDTParams(pts, fboSize=fbo))
    assert canon_set(dt.vtx) == canon_set(O.dt(pts)[0])
    return dt.status


# vertices = points + 4 * ceil((fbo - 1) / 16) ring sites
@pytest.mark.parametrize("n,fbo", [(192, 256), (193, 256), (960, 256), (961, 256), (3968, 512), (3969, 512),
                                   (28416, 1024), (28417, 1024)])
def test_cluster_sizes(engine, n, fbo):
    st = _check(engine, D.uniform_points(n, n), fbo)
    assert list(st.ms)[5] > 0.0  # the boundary's time, by the device's clock


@pytest.mark.parametrize("n,sigma", [(6000, 0.02), (40000, 0.02), (40000, 0.05)])
def test_missing_sites_handed_back(engine, n, sigma):
    st = _check(engine, D.gaussian_blobs(n, 23, nblobs=4, sigma=sigma), 256)
    assert st.nMissing > (8192 if n > 10000 else 1000)


@pytest.mark.parametrize("n", [5, 40, 700])
def test_long_fans(engine, n):
    """A few points on a large texture: ring sites whose fans and runs span
    hundreds of triangles once their neighbours are gone."""
    th = np.linspace(0.0, 2.0 * np.pi, n, endpoint=False) + 0.01
    pts = np.stack([np.cos(th), np.sin(th)], axis=1) * (0.02 + 0.98 * (np.arange(n) % 5 == 0))[:, None]
    pts = pts + 1e-3 * D.uniform_points(n, n)
    dt = engine.triangulate(G.GPUDTParams(pts, fboSize=4096))
    ok, rep = compare_dt(pts, dt.vtx, dt.tri)
    assert ok and rep["identical"], rep


def test_lattice_and_duplicates(engine):
    """Cocircular quads, collinear hulls and exact duplicates."""
    g = np.stack(np.meshgrid(np.arange(60.0), np.arange(60.0)), axis=-1).reshape(-1, 2)
    pts = np.concatenate([g, g[::7], g[::7]])
    dt = engine.triangulate(G.GPUDTParams(pts, fboSize=512))
    ok, rep = compare_dt(pts, dt.vtx, dt.tri)
    assert ok, rep
    assert dt.status.nDuplicates == 2 * len(g[::7])


def test_handles_in_parallel():
    """Launches of several handles' clusters overlap on the device."""
    sets = [D.uniform_points(n, n) for n in (900, 5000, 12000, 20000)]
    want = [canon_set(O.dt(p)[0]) for p in sets]
    bad = []

    def work(k):
        eng = G.Engine()
        for _ in range(10):
            if canon_set(eng.triangulate(G.GPUDTParams(sets[k], fboSize=512)).vtx) != want[k]:
                bad.append(k)
        eng.close()

    th = [threading.Thread(target=work, args=(k,)) for k in range(len(sets))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad


@pytest.mark.parametrize("n,fbo", [(8191, 512), (8192, 512), (8193, 512), (8193, 4096), (3000, 16384)])
def test_spatial_sort_sizes(engine, n, fbo):
    """One block sorts up to 8,192 points, digit passes more; odd and even
    numbers of digits."""
    pts = D.uniform_points(n, 3)
    pts[1::3] = pts[::3][:len(pts[1::3])] + 1e-9  # pixels with several sites
    _check(engine, pts, fbo)


@pytest.mark.parametrize("n", [1030, 1034, 1038, 2092, 2098, 2102, 2106, 2112])
def test_ranks_in_one_block(engine, n):
    """Spectrum lengths on both sides of what one block sorts, and of what it
    sorts without a look at the length."""
    from alphacheck import compare_alpha

    pts = D.uniform_points(n, 5)
    dt = engine.triangulate(G.GPUDTParams(pts, fboSize=512))
    ok, rep = compare_alpha(pts, dt.vtx, dt.tri, engine.alpha_resident(), 4)
    assert ok, rep


def test_ties_in_one_block(engine):
    """A lattice (exact ties) with a few points moved by far less than an ulp of
    the radii (near ties whose keys may be out of exact order)."""
    from alphacheck import compare_alpha

    g = np.stack(np.meshgrid(np.arange(20.0), np.arange(20.0)), axis=-1).reshape(-1, 2) / 3.0
    g[21::37] *= 1.0 + 2.0 ** -51
    dt = engine.triangulate(G.GPUDTParams(g, fboSize=256))
    ok, rep = compare_alpha(g, dt.vtx, dt.tri, engine.alpha_resident(), 4)
    assert ok, rep


@pytest.mark.parametrize("n", [3, 700, 1024, 1025, 3000])
def test_degenerate_inputs(engine, n):
    """Copies of one point, and collinear points, with the deciding point first,
    in the first 1,024 or after them: an empty mesh, or a triangulation."""
    for pts in (np.ones((n, 2)), np.stack([np.arange(n) * 0.5, np.arange(n) * 0.25], axis=1)):
        assert engine.triangulate(G.GPUDTParams(pts, fboSize=256)).nTris == 0
        assert len(engine.alpha_resident()["spectrum"]) == 1
        last = pts.copy()
        last[-1] += [0.3, 0.9]
        dt = engine.triangulate(G.GPUDTParams(last, fboSize=256))
        if len(np.unique(last, axis=0)) < 3:
            assert dt.nTris == 0
        else:
            ok, rep = compare_dt(last, dt.vtx, dt.tri)
            assert ok, rep
