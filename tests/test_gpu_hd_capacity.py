"""Sample capacities of large Hausdorff batches, whose areas the device adds:
the scratch they ask for is the host sum's to the word, so a pool of exactly
that size is accepted and one of a word less is refused."""
import numpy as np
import pytest

from conftest import pkg

G, M, T = pkg("meshgen"), pkg("mesh"), pkg("tree")

pytestmark = pytest.mark.gpu


def samples(m):
    """max(1000, floor(2000 * area)) with the area added in triangle order"""
    a, b, c = (m.verts[m.tris[:, k]].astype(np.float64) for k in range(3))
    area = np.cumsum(0.5 * np.linalg.norm(np.cross(b - a, c - a), axis=1))[-1]
    return max(1000, int(np.floor(2000.0 * area)))


def grid_cube(n, size):
    """A cube of n x n squares a side: its area is a whole number where size
    is, so that a bound around it never settles the floor."""
    k = np.arange(n + 1)
    u, w = (x.ravel() for x in np.meshgrid(k[:-1], k[:-1], indexing="ij"))
    verts, tris = [], []
    for ax in range(3):
        for side in (0, n):
            p = np.zeros(((n + 1) ** 2, 3))
            p[:, ax], p[:, (ax + 1) % 3], p[:, (ax + 2) % 3] = side, np.repeat(k, n + 1), np.tile(k, n + 1)
            i = u * (n + 1) + w + sum(map(len, verts))
            q = np.array([[i, i + n + 1, i + n + 2], [i, i + n + 2, i + 1]]).transpose(0, 2, 1).reshape(-1, 3)
            tris.append(q if side else q[:, ::-1])
            verts.append(p)
    return M.Mesh((np.concatenate(verts) * (size / n)).astype(np.float32), np.concatenate(tris))


def meshes(name):
    if name == "sphere":  # 20,480 triangles and more: the smallest batches the device adds
        return [G.noisy_icosphere(5, seed=1)]
    if name == "cubes":
        return [grid_cube(32, s) for s in (1.0, 2.0, 4.0)]
    if name == "slivers":  # edges far longer than the areas they span
        m = G.noisy_icosphere(4, seed=2)
        return [M.Mesh(m.verts * np.float32([1, 1e-5, s]), m.tris) for s in (1, 3, 10, 30)]
    rng = np.random.default_rng(5)
    base = [G.noisy_icosphere(k, seed=k) for k in (0, 1, 2, 3, 4)]
    return [M.Mesh(m.verts * rng.uniform(0.01, 9, size=3).astype(np.float32), m.tris) for m in base * 12]


@pytest.mark.parametrize("name", ["sphere", "cubes", "slivers", "many"])
def test_capacity_is_the_host_sums(name):
    ms = meshes(name)
    need = sum(3 * 2 * max(2 * samples(m) + m.nt + 16 for m in (m, o)) for m, o in zip(ms, ms[::-1]))
    cfg = dict(width=3, depth=1, nConcaveEdges=0, hullMaxVerts=16384)
    pairs = list(zip(ms, ms[::-1]))
    g = T.GpuTree(**cfg, scratchWords=need)
    full = g.hausdorff(pairs)
    assert np.isfinite(full).all()
    with pytest.raises(T.ScratchError):
        T.GpuTree(**cfg, scratchWords=need - 1).hausdorff(pairs)
    need = sum(3 * 2 * (2 * samples(m) + max(m.nt, 2 * m.nv) + 16) for m in ms)
    assert len(T.GpuTree(**cfg, scratchWords=need).hulls_with_hausdorff(ms)) == len(ms)
    with pytest.raises(T.ScratchError):
        T.GpuTree(**cfg, scratchWords=need - 1).hulls_with_hausdorff(ms)
