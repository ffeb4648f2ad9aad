"""Parts whose points are far more than their slab's faces (a small hull
bound): the points on the grid lie behind the slab's other words, on warps and
blocks, at sizes on both sides of the slab's spare room, for hulls that fit the
bound and hulls that fail it."""
import numpy as np
import pytest

from test_gpu_hull_lists import CFG, M, NONE, T, sphere

pytestmark = pytest.mark.gpu


def ball(n, seed):
    p = np.random.default_rng(seed).uniform(-1, 1, size=(n, 3))
    return M.Mesh(p.astype(np.float32), NONE)


@pytest.mark.parametrize("warps", [1, 1024, 16384], ids=["blocks", "both", "warps"])
@pytest.mark.parametrize("nv", [129, 1025, 5200])
def test_small_bounds(oracle, nv, warps):
    cfg = dict(CFG, hullMaxVerts=64)
    sets = [ball(nv, 1), ball(nv // 2, 2), sphere(min(nv, 1025), 3), ball(130, 4)]
    rg, sg = T.GpuTree(**cfg, warpMaxNv=warps).hull_meshes(sets)
    ro, so = oracle.OracleTree(**cfg).hull_meshes(sets)
    assert list(sg) == list(so)
    for a, b in zip(rg, ro):
        assert (a is None) == (b is None)
        if a is not None:
            assert np.array_equal(a["tris"], b["tris"]) and a["volume"] == b["volume"]
