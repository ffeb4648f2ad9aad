"""A level's children can be far larger than every seed: a plane through many
triangles gives each of them its own cut points. Such parts' hulls succeed on
blocks, warps and both, as the oracle's do."""
import numpy as np
import pytest

import parity
from conftest import pkg

M, T = pkg("mesh"), pkg("tree")

pytestmark = pytest.mark.gpu


def fan(n):
    """n thin triangles around the x axis, all crossed by the plane x = 0,
    over n + 2 vertices: a child has about 2 n points of its own."""
    a = 2 * np.pi * np.arange(n) / n
    r = np.where(np.arange(n) % (n // 20) == 0, 1.0, np.random.default_rng(n).uniform(0.3, 0.5, size=n))
    ring = np.stack([np.where(np.arange(n) % 2, 0.5, -0.5), r * np.cos(a), r * np.sin(a)], 1)
    v = np.concatenate([ring, [[-1, 0, 0], [1, 0, 0]]]).astype(np.float32)
    k = np.arange(n, dtype=np.uint32)
    j = (k + 1) % n
    t = [np.stack([k, np.full(n, n, np.uint32), j], 1), np.stack([k, j, np.full(n, n + 1, np.uint32)], 1)]
    return M.Mesh(v, np.concatenate(t))


@pytest.mark.parametrize("warps", [0, 1, 65536])
@pytest.mark.parametrize("n,bound", [(60, 4096), (400, 8), (2000, 64)])
def test_children_larger_than_seeds(oracle, n, bound, warps):
    cfg = dict(width=3, width2=3, depth=1, nConcaveEdges=0, hullMaxVerts=bound, warpMaxNv=warps)
    planes = [np.array([[1, 0, 0, 0.0]], np.float32)]
    g, o = T.GpuTree(**cfg), oracle.OracleTree(**cfg)
    m = fan(n)
    rg, ro = (t.run([m], planes, width=0, n_edge_cuts=1) for t in (g, o))
    assert rg["hullFailCount"] == ro["hullFailCount"]
    parity.compare_level_tables(g, o, rg, ro, 1, label=f"fan {n}")
    parity.compare_seeds(rg, ro, label=f"fan {n}")
    assert max(g.parts(1, 2 * rg["jobsPerLevel"][0])[:, 1]) > 2 * n
