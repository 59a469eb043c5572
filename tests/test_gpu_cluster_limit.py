"""GPU tests of the mesh stages where the cluster of the one-launch form cannot
be placed or is not allowed (galphaSetClusterLimit): every stage runs as
launches of its own and the triangulation is the oracle's all the same.  Which
form ran shows in the counter reads: the one launch makes one for all stages,
the launched boundary stage at least two of its own."""
import numpy as np
import pytest

import galpha_b200 as G
from galpha_b200 import datasets as D
from alphacheck import compare_alpha
from dtcheck import canon_set, compare_dt
from oracle import oracle as O

pytestmark = pytest.mark.gpu
SHIFT, MISSING, BOUNDARY, FLIP = 3, 4, 5, 6


@pytest.fixture()
def limited(engine):
    yield engine
    engine.set_cluster_limit(-1)


# vertices = points + 64 ring sites; a cluster has one block per 256, rounded up to a power of two
@pytest.mark.parametrize("n,blocks", [(3, 1), (192, 1), (193, 2), (960, 4), (961, 8), (1984, 8), (1985, 16), (12000, 16)])
def test_limit_chooses_the_form(limited, n, blocks):
    pts = D.uniform_points(n, n)
    want = canon_set(O.dt(pts)[0])
    for limit in (0, blocks // 2, blocks, 16, -1):
        limited.set_cluster_limit(limit)
        dt = limited.triangulate(G.GPUDTParams(pts, fboSize=256))
        assert canon_set(dt.vtx) == want
        reads = list(dt.status.hostReadsStage)
        if limit >= blocks or limit < 0:
            assert [reads[k] for k in (SHIFT, MISSING, BOUNDARY, FLIP)] == [1, 0, 0, 0]
        else:
            assert reads[SHIFT] >= 2 and reads[MISSING] >= 1 and reads[BOUNDARY] >= 2 and reads[FLIP] >= 1
        assert all(dt.status.ms[k] > 0.0 for k in (SHIFT, BOUNDARY, FLIP))


@pytest.mark.parametrize("limit", [0, 4])
def test_clustered_constraints_and_batches(limited, limit):
    limited.set_cluster_limit(limit)
    pts = D.gaussian_blobs(40000, 23, nblobs=4, sigma=0.02)  # bad and missing sites by the thousand
    dt = limited.triangulate(G.GPUDTParams(pts, fboSize=256))
    assert dt.status.nMissing > 8192 and canon_set(dt.vtx) == canon_set(O.dt(pts)[0])
    pts = D.uniform_points(3000, 9)
    order = np.argsort(pts[:, 0])[::40].astype(np.int32)
    cons = np.stack([order[:-1], order[1:]], axis=1)
    got = {}
    for lim in (limit, -1):
        limited.set_cluster_limit(lim)
        dt = limited.triangulate(G.GPUDTParams(pts, fboSize=512, constraints=cons))
        got[lim] = canon_set(dt.vtx)
        assert (dt.status.hostReadsStage[SHIFT] == 1) == (lim < 0)
    assert got[limit] == got[-1]
    limited.set_cluster_limit(limit)
    sets = [D.uniform_points(n, n + 1) for n in (3, 70, 800, 4000)]
    limited.run_batch(sets)
    for s, r in zip(sets, limited.batch_results()):
        vtx = r["triangles"]["vtx"]
        assert canon_set(vtx) == canon_set(O.dt(s)[0])


def test_alpha_after_launched_stages(limited):
    limited.set_cluster_limit(0)
    for n in (5, 900, 9000):
        pts = D.uniform_points(n, 3 * n)
        dt, res = limited.compute_all(G.GPUDTParams(pts, fboSize=512))
        ok, rep = compare_dt(pts, dt.vtx, dt.tri)
        assert ok, rep
        ok, rep = compare_alpha(pts, dt.vtx, dt.tri, res, 4)
        assert ok, rep


@pytest.mark.parametrize("side,spacing,launched", [(60, 3.0, False), (66, 3.0, True), (120, 3.0, True), (120, 1.0, True)])
def test_flips_with_many_exact_tests(engine, side, spacing, launched):
    """A lattice leaves an edge of every triangle to the exact in-circle test: with
    more triangles than the cluster has threads (8,192) the flips are handed back
    to launches.  With constraints they are handed back after those."""
    g = np.stack(np.meshgrid(np.arange(float(side)), np.arange(float(side))), axis=-1).reshape(-1, 2) / spacing
    for cons in (None, np.array([[0, side * (side - 1) + 1], [side - 1, side * (side - 1) + side - 2]], np.int32)):
        dt = engine.triangulate(G.GPUDTParams(g, fboSize=1024, constraints=cons))
        if cons is None:
            assert (dt.status.hostReadsStage[FLIP] >= 1) == launched
            ok, rep = compare_dt(g, dt.vtx, dt.tri)
            assert ok, rep
            assert dt.status.exactIncircle >= (side - 1) ** 2  # a diagonal per cell
        else:
            v = np.concatenate([dt.vtx[:, [0, 1]], dt.vtx[:, [1, 2]], dt.vtx[:, [2, 0]]])
            edges = set(map(tuple, v.tolist())) | set(map(tuple, v[:, ::-1].tolist()))
            assert all(tuple(c) in edges for c in cons.tolist())
            assert dt.nTris == 2 * side * side - 2 - 4 * (side - 1)
    pts = D.uniform_points(12000, 4)  # the same size, nothing undecided
    assert engine.triangulate(G.GPUDTParams(pts, fboSize=512)).status.hostReadsStage[FLIP] == 0


def test_constraint_time_in_the_boundary_stage(engine):
    """gpudtStatus.ms[boundary] holds the constraints' time too, with the fake
    ring in the one launch as with launches (some 500 us against 200)."""
    pts = D.uniform_points(20000, 6)
    band = np.floor(pts[:, 1] * 141).astype(int)
    lines = [np.nonzero(band == b)[0] for b in range(4, 140, 12)]
    lines = [i[np.argsort(pts[i, 0])] for i in lines]
    cons = np.concatenate([np.stack([i[:-1], i[1:]], axis=1) for i in lines]).astype(np.int32)
    ms = {}
    for name, c in (("plain", None), ("constrained", cons)):
        ms[name] = np.median([engine.triangulate(G.GPUDTParams(pts, fboSize=1024, constraints=c)).status.ms[BOUNDARY]
                              for _ in range(5)])
    assert ms["constrained"] > 1.5 * ms["plain"]


# 256 ring sites: 196,608 vertices is the last size that shifts in the one launch
@pytest.mark.parametrize("n,one", [(196352, True), (196353, False)])
def test_shift_size_limit(engine, n, one):
    pts = D.gaussian_blobs(n, 9, nblobs=64, sigma=0.01)
    dt = engine.triangulate(G.GPUDTParams(pts, fboSize=1024))
    reads = list(dt.status.hostReadsStage)
    assert (reads[SHIFT] == 1) == one and reads[BOUNDARY] == 1  # the fake ring is in one launch either way
    assert canon_set(dt.vtx) == canon_set(O.dt(pts)[0])


def test_limit_out_of_range(engine):
    with pytest.raises(G.GpudtError):
        engine.set_cluster_limit(17)
