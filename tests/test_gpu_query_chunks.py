"""GPU tests of the query kernels at the edges of their chunks (2,048 entries
of one kind per block): a single set whose points end just before, on and
after a chunk, and batches whose chunks hold one set or many.  Every class and
count must equal the numpy restatement of the interval rule."""
import numpy as np
import pytest

import galpha_b200 as G
from galpha_b200 import datasets as D
from alphacheck import classify_intervals

pytestmark = pytest.mark.gpu


def _counts(c):
    return np.bincount(c, minlength=4).tolist()


@pytest.mark.parametrize("n", [3, 2047, 2048, 2049, 4097])
def test_query_chunk_edges(engine, n):
    engine.triangulate(G.GPUDTParams(D.uniform_points(n, n), fboSize=256))
    res = engine.alpha_resident()
    spec = res["spectrum"]
    for a in (float(spec[1]), float(spec[len(spec) // 2]), float(spec[-1])):
        q = engine.query(alpha=a)
        wp, we, wt, R = classify_intervals(res, a)
        pc, ec, tc = engine.classes()
        assert q.rank == R and q.alpha == a
        for got, want, cnt in ((pc, wp, q.nPoints), (ec, we, q.nEdges), (tc, wt, q.nTris)):
            np.testing.assert_array_equal(got, want)
            assert list(cnt) == _counts(want)


@pytest.mark.parametrize("sizes", [[5] * 700, [2047, 1, 2, 2048, 3, 0, 6200, 4], [9000]])
def test_batch_query_chunk_edges(sizes):
    engine = G.Engine()
    sets = [D.uniform_points(n, 100 + k).reshape(-1, 2) for k, n in enumerate(sizes)]
    engine.run_batch(sets)
    res = engine.batch_results()
    for quantile in (0.0, 0.4, 1.0):
        q = engine.batch_query(quantile, by_quantile=True)
        classes = engine.classes()
        at = [0, 0, 0]
        for k, r in enumerate(res):
            spec = r["spectrum"]
            a = float(spec[int(np.rint(quantile * (len(spec) - 1)))])
            wp, we, wt, R = classify_intervals(r, a)
            assert q[k].alpha == a and q[k].rank == R
            for j, (want, cnt) in enumerate(((wp, q[k].nPoints), (we, q[k].nEdges), (wt, q[k].nTris))):
                np.testing.assert_array_equal(classes[j][at[j]:at[j] + len(want)], want)
                assert list(cnt) == _counts(want)
                at[j] += len(want)
        assert [len(c) for c in classes] == at
    engine.close()
