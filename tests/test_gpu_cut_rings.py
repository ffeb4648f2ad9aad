"""The GPU cap at the sizes where its forms change, bit for bit against the
host cut: rings around the 32 vertices that a warp holds whole, rings in
shared memory and beyond its 2,048 nodes, tall and flat outlines (ears that
cover many rows of the grid), collinear runs, and boundary vertices with two
out-edges (the sequential walk)."""
import importlib

import numpy as np
import pytest

from conftest import pkg

M = pkg("mesh")
D = importlib.import_module("cuacd-web_gb300.decompose")
T = importlib.import_module("cuacd-web_gb300.tree")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tree():
    return T.GpuTree(width=3, width2=3, depth=1, nConcaveEdges=0)


def prism(outline):
    """A closed prism over a ring of points (z from -1 to 1)."""
    n = len(outline)
    v = np.concatenate([np.c_[outline, np.full(n, -1.0)], np.c_[outline, np.full(n, 1.0)], [[*outline.mean(0), -1.0], [*outline.mean(0), 1.0]]])
    i, j = np.arange(n), (np.arange(n) + 1) % n
    t = np.concatenate([np.c_[i, j, n + j], np.c_[i, n + j, n + i], np.c_[np.full(n, 2 * n), j, i], np.c_[np.full(n, 2 * n + 1), n + i, n + j]])
    return M.Mesh(v.astype(np.float32), t.astype(np.uint32))


def star(n, seed, flat=1.0):
    rng = np.random.default_rng(seed)
    a = 2 * np.pi * np.arange(n) / n
    r = rng.uniform(0.4, 1.0, n)
    return np.stack([r * np.cos(a), flat * r * np.sin(a)], 1)


def comb(n):
    """A comb of n teeth: long thin teeth, collinear tips and gaps."""
    x = np.arange(2 * n + 1, dtype=float) / (2 * n)
    top = [p for k in range(n) for p in ((x[2 * k], 1.0), (x[2 * k + 1], 1.0), (x[2 * k + 1], 0.05), (x[2 * k + 2], 0.05))]
    return np.array([(0.0, 0.0), (1.0, 0.0), *reversed(top)])


def same(tree, meshes, plane):
    got = tree.plane_cuts(meshes, [plane] * len(meshes), None, closed=True)
    for k, (m, (st, pos, neg)) in enumerate(zip(meshes, got)):
        try:
            want = D.plane_cut(m, plane)
        except T.CuacdError:
            assert st != 0, k
            continue
        assert st == 0, (k, st)
        for g, w in zip((pos, neg), want):
            assert np.array_equal(g.verts, w.verts) and np.array_equal(g.tris, w.tris), k


@pytest.mark.parametrize("plane", [[0, 0, 1, 0.1], [0.05, -0.02, 1, 0.03]])
def test_ring_sizes(tree, plane):
    # every wall quad is two triangles: a plane across the walls meets 2 n edges
    sizes = (3, 4, 8, 15, 16, 17, 18, 31, 32, 33, 34, 65, 200, 1020, 1030)
    meshes = [prism(star(n, n)) for n in sizes] + [prism(star(n, n, 0.01)) for n in (16, 33, 100)]
    meshes += [prism(star(n, n)[:, ::-1][::-1] * [0.01, 1.0]) for n in (17, 40, 300)]
    meshes += [prism(comb(n)) for n in (2, 4, 9, 40)]
    same(tree, meshes, plane)


def test_two_out_edges(tree):
    """Boxes meeting in a vertical edge, welded: the cap's vertex there has
    two out-edges."""
    a = M.make_box((0, 0, -1), (1, 1, 1))
    b = M.make_box((1, 1, -1), (2, 2, 1))
    v, inv = np.unique(np.concatenate([a.verts, b.verts]), axis=0, return_inverse=True)
    m = M.Mesh(v, inv.reshape(-1)[np.concatenate([a.tris, b.tris + 8]).astype(np.int64)].astype(np.uint32))
    assert m.nv == 14
    for plane in ([0, 0, 1, 0.25], [0.1, 0.05, 1, 0]):
        same(tree, [m, a, m], plane)
