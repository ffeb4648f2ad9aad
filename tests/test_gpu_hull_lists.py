"""Block hulls (candidates in per-face lists) and the warps' handing on, at
the sizes where their forms change, against the oracle's faces and volumes:
part sizes around a warp's and a block's width, convex position (every point
inserted, so the candidate pool is compacted), lattices (coplanar points,
exact signs), duplicates, and low hats on m-gon prisms, whose insertion sees
the whole m-gon cap: within a walk's 32 faces, beyond it, and beyond the 128
faces of the single-pick step."""
import importlib

import numpy as np
import pytest

from conftest import pkg

M = pkg("mesh")
T = importlib.import_module("cuacd-web_gb300.tree")

pytestmark = pytest.mark.gpu
CFG = dict(width=3, width2=3, depth=1, nConcaveEdges=0, hullMaxVerts=4096)
NONE = np.zeros((0, 3), np.uint32)


def sphere(n, seed, noise=0.0):
    rng = np.random.default_rng(seed)
    p = rng.normal(size=(n, 3))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    return M.Mesh((p * (1.0 - noise * rng.uniform(size=(n, 1)))).astype(np.float32), NONE)


def lattice(n, seed):
    p = np.random.default_rng(seed).integers(0, 7, size=(n, 3))
    return M.Mesh(p.astype(np.float32), NONE)


def twice(n, seed):
    p = sphere((n + 1) // 2, seed).verts
    return M.Mesh(np.concatenate([p, p])[:n], NONE)


def hat(m, height=1e-5):
    a = 2 * np.pi * np.arange(m) / m
    ring = np.stack([np.cos(a), np.sin(a)], 1)
    p = [np.concatenate([ring, np.full((m, 1), z)], 1) for z in (-0.5, 0.5)] + [[[0, 0, 0.5 + height], [0, 0, -0.5 - height]]]
    return M.Mesh(np.concatenate(p).astype(np.float32), NONE)


def check(tree, oracle, sets):
    rg, sg = tree.hull_meshes(sets)
    ro, so = oracle.OracleTree(**CFG).hull_meshes(sets)
    assert list(sg) == list(so)
    for i, (a, b) in enumerate(zip(rg, ro)):
        assert (a is None) == (b is None), i
        if a is not None:
            assert np.array_equal(a["tris"], b["tris"]) and a["volume"] == b["volume"], (i, sets[i].nv)


SIZES = (4, 5, 8, 31, 32, 33, 34, 64, 96, 128, 129, 255, 256, 257, 511, 513, 1023, 1024, 1025)


@pytest.mark.parametrize("cfg", [{}, dict(warpMaxNv=1), dict(warpMaxNv=4096)], ids=["handed on", "blocks", "warps"])
@pytest.mark.parametrize("make", [sphere, lattice, twice])
def test_sizes(oracle, make, cfg):
    check(T.GpuTree(**CFG, **cfg), oracle, [make(n, n) for n in SIZES])


@pytest.mark.parametrize("count", [1, 153, 305])
def test_hats_on_every_block_width(oracle, count):
    """1, 153 and 305 parts: 1024-, 512- and 256-thread blocks on 152 SMs."""
    sets = [hat(m) for m in (12, 30, 33, 34, 60, 126, 131, 200, 700)]
    sets = sets if count > 1 else sets[-2:]
    pad = [sphere(5, k) for k in range(max(0, count - len(sets)))]
    check(T.GpuTree(**CFG, warpMaxNv=1), oracle, sets + pad)


def test_convex_position_compacts_pool(oracle):
    check(T.GpuTree(**CFG), oracle, [sphere(3500, 1), sphere(3500, 2, 0.01), sphere(700, 3)])


def test_tree_levels_hand_on(oracle):
    """A tree whose children fall on both sides of every rule: its tables
    equal the oracle's under each trial schedule."""
    import parity

    gen = pkg("meshgen")
    cfg = dict(CFG, width=3, depth=2)
    seeds = [gen.noisy_icosphere(2, seed=1), M.normalize(gen.blob_mesh(6, 14, seed=3))[0], gen.staircase(5)]
    g, o = T.GpuTree(**cfg), oracle.OracleTree(**cfg)
    ro = o.run(seeds)
    for k in range(4):
        rg = g.run(seeds)
        parity.compare_level_tables(g, o, rg, ro, len(seeds), label=f"run {k}")
        parity.compare_seeds(rg, ro, label=f"run {k}")
