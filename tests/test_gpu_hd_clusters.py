"""The Hausdorff cluster search at the sizes where its blocks and clusters
end: one triangle, around a cluster of 32, around the area chunk (1,920), the
count and sort chunk (2,048) and their doubles, against the oracle's float32
form and, bit for bit, against the search that evaluates every triangle."""
import importlib

import numpy as np
import pytest

from conftest import pkg

M, G = pkg("mesh"), pkg("meshgen")
T = importlib.import_module("cuacd-web_gb300.tree")

pytestmark = pytest.mark.gpu
SIZES = (1, 31, 32, 33, 63, 64, 65, 1919, 1920, 1921, 2047, 2048, 2049, 4097)


@pytest.fixture(scope="module")
def trees():
    cfg = dict(width=3, width2=3, depth=1, nConcaveEdges=0, hullMaxVerts=4096)
    return T.GpuTree(**cfg, hdScreenMinTris=1), T.GpuTree(**cfg, hdScreenMinTris=-1), T.GpuTree(**cfg)


def piece(n, seed, offset=0.0):
    """n triangles of a noisy icosphere in random order (an open surface),
    every seventh one collapsed to a segment."""
    m = G.noisy_icosphere(4 if n <= 5120 else 5, seed=seed)
    t = m.tris[np.random.default_rng(seed).permutation(m.nt)[:n]].copy()
    t[6::7, 2] = t[6::7, 1]
    return M.Mesh(m.verts + np.float32(offset), t)


@pytest.mark.parametrize("offset", [0.0, 300.0])
def test_cluster_search_sizes(trees, oracle, offset):
    pairs = [(piece(n, 2 * i, offset), piece(SIZES[(5 * i + 3) % len(SIZES)], 2 * i + 1, offset))
             for i, n in enumerate(SIZES)]
    a, b, c = (t.hausdorff(pairs) for t in trees)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (a, b)
    assert np.array_equal(c.view(np.uint32), b.view(np.uint32)), (c, b)
    if offset == 0.0:
        ref = oracle.hausdorff_gpu_form(pairs)
        assert np.all(np.abs(a - ref) <= 1e-5 + 1e-4 * ref), (a, ref)


def test_cluster_search_long_and_mixed_batch(trees):
    """More meshes than one tile-prefix chunk holds (2 x 600), with empty
    meshes among them."""
    base = [piece(n, n) for n in (1, 33, 70, 320)] + [M.Mesh(np.zeros((0, 3), np.float32), np.zeros((0, 3), np.uint32))]
    pairs = [(base[i % 5], base[(i * 7 + 1) % 5]) for i in range(600)]
    a, b = trees[0].hausdorff(pairs), trees[1].hausdorff(pairs)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    for i, (x, y) in enumerate(pairs):
        if x.nt == 0 or y.nt == 0:
            assert a[i] == 0.0


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_cluster_search_slivers(trees, seed):
    """Parts cut again and again hold slivers, whose tri_sq can be far off
    their geometry: the distances are the same on every run, whichever tiles
    finish first; a sliver out of reach does not count, so they are never
    below the search in which every triangle does; and small targets' are
    that search's."""
    cut = pkg("decompose").plane_cut
    rng = np.random.default_rng(seed)
    parts = [G.noisy_icosphere(3, seed=seed), M.normalize(G.blob_mesh(6, 22 + seed, seed=seed))[0]]
    for _ in range(4):
        halves = []
        for m in parts:
            n = np.eye(3)[rng.integers(3)] if rng.random() < 0.5 else rng.normal(size=3)
            n /= np.linalg.norm(n)
            p = m.verts.astype(np.float64) @ n
            try:
                halves += cut(m, [*n, -(p.min() + rng.uniform(0.3, 0.7) * np.ptp(p))])
            except RuntimeError:
                halves.append(m)
        parts = [h for h in halves if h.nt >= 4]
    runs = [[h["hausdorff"] if h else None for h in t.hulls_with_hausdorff(parts)] for t in (trees[2], trees[2], trees[1])]
    assert runs[0] == runs[1]
    for m, x, y in zip(parts, runs[0], runs[2]):
        assert (x is None) == (y is None) and (x is None or x >= y)
    small = [(m, o) for m in parts for o in parts if max(m.nt, o.nt) < 256]
    assert np.array_equal(trees[2].hausdorff(small), trees[1].hausdorff(small))
