"""GPU test of a handle that is moved to a caller's stream right after it is
made: its first scans find cleared status words, although the memory was an
earlier handle's, whose words carry the same scan numbers."""
import pytest

import galpha_b200 as G
from galpha_b200 import datasets as D
from dtcheck import canon_set
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_new_handle_on_a_caller_stream():
    torch = pytest.importorskip("torch")
    sets = [D.uniform_points(n, n) for n in (40000, 5000)]  # scans of several tiles and of one
    want = [canon_set(O.dt(p)[0]) for p in sets]
    stream = torch.cuda.Stream()
    for k in range(12):
        eng = G.Engine()
        try:
            eng.set_stream(stream.cuda_stream)
            for p, w in zip(sets, want):
                assert canon_set(eng.triangulate(G.GPUDTParams(p, fboSize=1024)).vtx) == w
        finally:
            eng.close()
