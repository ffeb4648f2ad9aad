"""GPU concave planes where their kernels' forms change, bit for bit against
the host restatement: vertices of high valence (fans whose rim zigzags, so
that spokes are concave), thresholds on both sides of pi (with and without
the cosine test) and at extreme angles, reservoirs around a warp's width, and
edges that occur twice (boxes welded along an edge)."""
import numpy as np
import pytest

from conftest import pkg

M, G, D, T = pkg("mesh"), pkg("meshgen"), pkg("decompose"), pkg("tree")

pytestmark = pytest.mark.gpu


def zigzag(n):
    """A double cone over a rim of n points that alternate in radius."""
    a = 2 * np.pi * np.arange(n) / n
    r = np.where(np.arange(n) % 2 == 0, 1.0, 0.8)
    v = np.concatenate([np.stack([r * np.cos(a), r * np.sin(a), np.zeros(n)], 1), [[0, 0, 0.5], [0, 0, -0.5]]])
    i, j = np.arange(n), (np.arange(n) + 1) % n
    return M.Mesh(v, np.concatenate([np.c_[i, j, np.full(n, n)], np.c_[j, i, np.full(n, n + 1)]]))


def welded():
    a, b = M.make_box((0, 0, 0), (1, 1, 1)), M.make_box((1, 1, 0), (2, 2, 1))
    v, inv = np.unique(np.concatenate([a.verts, b.verts]), axis=0, return_inverse=True)
    return M.Mesh(v, inv.reshape(-1)[np.concatenate([a.tris, b.tris + 8]).astype(np.int64)])


@pytest.mark.parametrize("n_edges", [1, 31, 32, 33, 100])
@pytest.mark.parametrize("threshold", [2.5, np.pi, 3.15, 3.49, 6.0])
def test_hubs_and_thresholds(n_edges, threshold):
    meshes = [zigzag(n) for n in (4, 12, 64, 1000)] + [welded(), G.noisy_icosphere(3, seed=2), G.staircase(9),
                                                       M.Mesh(np.zeros((3, 3)), np.zeros((0, 3)))]
    seeds = [5 + 77 * k for k in range(len(meshes))]
    got = T.GpuTree(width=3, width2=3, depth=1, nConcaveEdges=0).concave_planes(meshes, n_edges, 0.005, threshold, seeds)
    for k, (m, s, p) in enumerate(zip(meshes, seeds, got)):
        want = D.concave_planes(m, n_edges, 0.005, threshold, s)
        assert np.array_equal(p.view(np.uint32), want.view(np.uint32)), (k, p.shape, want.shape)
