"""Targets on both sides of the sizes where the Hausdorff search changes its
form, so far away that squared distances pass the 1e30 from which the search
that evaluates every triangle starts: the same distances."""
import numpy as np
import pytest

from conftest import pkg

G, M, T = pkg("meshgen"), pkg("mesh"), pkg("tree")

pytestmark = pytest.mark.gpu


def test_small_targets_far_away():
    cfg = dict(width=3, width2=3, depth=1, nConcaveEdges=0, hullMaxVerts=4096)
    m = G.icosphere(3)
    part = {n: M.Mesh(m.verts, m.tris[:n]) for n in (32, 63, 64, 65, 200, 255)}
    pairs = [(p, M.Mesh(p.verts + np.float32([x, 0, 0]), p.tris)) for p in part.values()
             for x in (5.0, 3e7, 5e15)]
    a, b = T.GpuTree(**cfg).hausdorff(pairs), T.GpuTree(**cfg, hdScreenMinTris=-1).hausdorff(pairs)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (a, b)
