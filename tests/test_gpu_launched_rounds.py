"""GPU tests of the round loops that run as launches of their own (shifting,
missing sites, fake removal, flips; ring words of per-round counts read by the
host in groups): small clustered sets with the one-launch form turned off, and
sets above the sizes it takes, under schedules that read the counters after
every round, after groups of eight (half a ring, the tightest reuse of its
words) and only at the end, and with a round cap.  The triangulation must be
the oracle's; the counter reads show that the loops under test ran."""
import ctypes

import pytest

import galpha_b200 as G
from galpha_b200 import datasets as D
from dtcheck import canon_set
from oracle import oracle as O

pytestmark = pytest.mark.gpu
SHIFT, MISSING, BOUNDARY, FLIP = 3, 4, 5, 6


def _blobs(n):
    pts = D.gaussian_blobs(n, 17, nblobs=3, sigma=0.02)
    pts[::7] = D.uniform_points(len(pts[::7]), 18) * 2.0 - 1.0  # far points: long chains of flips
    return pts


@pytest.mark.parametrize("n", [4, 1023, 20001])
@pytest.mark.parametrize("sched", [(1, 1, 1, 0, 1), (8, 8, 64, 0, 1), (3, 5, 7, 2000, 2001), (0, 0, 0, -1, 0)])
def test_small_sets(n, sched):
    pts = _blobs(n)
    want = canon_set(O.dt(pts)[0])
    eng = G.Engine()
    try:
        eng.set_cluster_limit(0)
        eng.set_schedule(*sched)
        for _ in range(2):  # the handle's second call starts from the first one's words
            dt = eng.triangulate(G.GPUDTParams(pts, fboSize=256))
            assert canon_set(dt.vtx) == want
    finally:
        eng.close()
    st, reads = dt.status, list(dt.status.hostReadsStage)
    if n > 20000:
        assert st.shiftRounds > 8 and st.missingRounds > 2 and st.nBadShift > 0
        if sched[0] == 1:  # a read per round
            assert reads[SHIFT] >= st.shiftRounds and reads[MISSING] >= st.missingRounds
            assert st.flipRounds > 16 and reads[FLIP] >= st.flipRounds
        if sched[0] == 8:
            assert reads[SHIFT] < st.shiftRounds and reads[MISSING] < st.missingRounds and reads[FLIP] <= 2


@pytest.mark.parametrize("dist", ["uniform", "clustered"])
def test_above_the_one_launch_sizes(dist):
    n = 270000
    pts = D.uniform_points(n, 3) if dist == "uniform" else D.gaussian_blobs(n, 5, nblobs=16, sigma=0.02)
    want = canon_set(O.dt(pts)[0])
    eng = G.Engine()
    reads = {}
    try:
        for sched in ((1, 1, 1, 0, 1), (8, 8, 64, 0, 1), (0, 0, 0, -1, 0)):
            eng.set_schedule(*sched)
            dt = eng.triangulate(G.GPUDTParams(pts, fboSize=1024))
            assert canon_set(dt.vtx) == want
            assert dt.status.nMissing > 10000 and dt.status.nBadShift > 0
            reads[sched[0]] = list(dt.status.hostReadsStage)
    finally:
        eng.close()
    assert reads[1][SHIFT] > reads[0][SHIFT] > 2 and reads[1][MISSING] > reads[8][MISSING]


def test_round_cap(engine):
    """The launched loops stop at the round cap with NOCONVERGE, in each stage
    that needs more rounds than it, and the next call computes the full result."""
    L = G.load()
    L.galphaSetLimits.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int]
    pts = _blobs(20001)
    want = canon_set(O.dt(pts)[0])
    engine.set_cluster_limit(0)
    try:
        stages = set()
        for cap in (1, 4, 16, 64):
            assert L.galphaSetLimits(engine._h, cap, 0, 0) == 0
            try:
                engine.triangulate(G.GPUDTParams(pts, fboSize=256))
            except G.GpudtError as e:
                assert e.code == -5
                stages.add(str(e).split("stage ")[1].split(":")[0])
        assert "shift" in stages
        assert L.galphaSetLimits(engine._h, 0, 0, 0) == 0
        assert canon_set(engine.triangulate(G.GPUDTParams(pts, fboSize=256)).vtx) == want
    finally:
        L.galphaSetLimits(engine._h, 0, 0, 0)
        engine.set_cluster_limit(-1)
