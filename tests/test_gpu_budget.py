"""GPU test of device-memory budgets: the scratch of the one-launch mesh stages
adds nothing to what a call needs, so a budget that held a call with every
stage as launches of its own (the bytes below) holds it in the one-launch form,
also where fans too long for shared memory need that scratch."""
import numpy as np
import pytest

import galpha_b200 as G
from galpha_b200 import datasets as D
from dtcheck import canon_set, compare_dt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,fbo,nbytes", [(3, 256, 1045216), (1000, 256, 2007008), (1000, 512, 4063200),
                                          (5000, 512, 7936480), (20000, 1024, 30553568), (60000, 1024, 69273056)])
def test_budget_holds_the_call(n, fbo, nbytes):
    eng = G.Engine(budget_bytes=nbytes)
    try:
        pts = D.uniform_points(n, 1)
        assert canon_set(eng.triangulate(G.GPUDTParams(pts, fboSize=fbo)).vtx) == canon_set(O.dt(pts)[0])
    finally:
        eng.close()


@pytest.mark.parametrize("n", [600, 3000])
def test_long_fans_in_the_idle_array(engine, n):
    """A diagonal row of points with one either side: ring sites whose fans and
    runs hold up to half of the mesh, several of them in a round."""
    x = np.arange(n) / 4096.0
    pts = np.concatenate([np.stack([x, x], axis=1), [[x[-1] * 0.9375, x[-1] * 0.0625], [x[-1] * 0.0625, x[-1] * 0.9375]]])
    for fbo in (256, 1024):
        dt = engine.triangulate(G.GPUDTParams(pts, fboSize=fbo))
        assert dt.status.hostReadsStage[5] == 0  # the fake ring went in the one launch
        ok, rep = compare_dt(pts, dt.vtx, dt.tri)
        assert ok, rep
