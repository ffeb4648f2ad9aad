"""The GPU cap where an ear covers many rows of the ring's grid, with few and
with many nodes a row (either way of going through them, and both in one
ring), bit for bit against the host cut."""
import importlib

import numpy as np
import pytest

from conftest import pkg
from test_gpu_cut_rings import prism, same, star

T = importlib.import_module("cuacd-web_gb300.tree")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tree():
    return T.GpuTree(width=3, width2=3, depth=1, nConcaveEdges=0)


def spiral(n, turns, seed):
    """A band wound into itself: ears across it cover the rows of every turn."""
    rng = np.random.default_rng(seed)
    a = np.linspace(0, 2 * np.pi * turns, n)
    r = 0.2 + 0.8 * a / a[-1]
    w = 0.25 * 0.8 / turns
    out = np.stack([(r + w) * np.cos(a), (r + w) * np.sin(a)], 1)
    back = np.stack([(r - w * rng.uniform(0.2, 1.0, n)) * np.cos(a), (r - w) * np.sin(a)], 1)[::-1]
    return np.concatenate([out, back])


@pytest.mark.parametrize("n", [40, 300, 1100, 2600])
def test_ears_over_many_rows(tree, n):
    meshes = [prism(star(n, n)), prism(star(n, n + 1, 0.1)), prism(spiral(n // 2, 3, n)), prism(spiral(n // 2, 9, n))]
    same(tree, meshes, [0, 0, 1, 0.1])
