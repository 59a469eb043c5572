"""GPU tests of the alpha stage at exact triangle counts: on both sides of the
edges of its tiles (256 triangles with one per thread, 1,024 with four), of the
number of tiles whose status words fit the counter block (63), and of the
counts per SM where it goes over to four triangles per thread (1,024) and to
vertex intervals combined per block (4,096).  The mesh is the first triangles
of a triangulation, handed in as the caller's own."""
import numpy as np
import pytest

import galpha_b200 as G
from galpha_b200 import datasets as D
from alphacheck import compare_alpha

pytestmark = pytest.mark.gpu
_kept = {}


def _mesh(engine, want):
    n = next(m for m in (700, 9000, 90000, 320000) if 2 * m - 200 > want)
    if n not in _kept:
        pts = D.uniform_points(n, n)
        _kept[n] = pts, engine.triangulate(G.GPUDTParams(pts, fboSize=1024)).triangles
    pts, tris = _kept[n]
    part = tris[:want].copy()
    nbr = part["tri"]
    nbr[(nbr >= 0) & (nbr >> 2 >= want)] = -1
    return pts, part


def _counts():
    out = [1, 2, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 63 * 256, 63 * 256 + 1, 64 * 256]
    return out + ["%d*%+d" % (k, d) for k in (1024, 4096) for d in (-1, 0, 1)] + ["1025*-1", "1025*+0", "1025*+1"]


@pytest.mark.parametrize("want", _counts())
def test_exact_counts(engine, want):
    if isinstance(want, str):  # per SM; 1025: whole tiles of 1,024 past the change to four per thread
        import torch

        sms = torch.cuda.get_device_properties(0).multi_processor_count
        k, d = want.split("*")
        want = (int(k) * sms if k != "1025" else 1024 * (sms + 1)) + int(d)
    pts, tris = _mesh(engine, want)
    assert len(tris) == want
    params = G.GPUDTParams(pts, fboSize=1024)
    res = engine.alpha_of(params, G.DTOutput(tris, None))
    assert len(res["tri_list"]) == want
    ok, rep = compare_alpha(pts, tris["vtx"], tris["tri"], res, 4)
    assert ok, rep
