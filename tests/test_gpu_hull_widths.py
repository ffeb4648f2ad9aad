"""Hull blocks of 256, 512 and 1024 threads, chosen by the batch's largest part
and its count: the oracle's faces and volumes of small parts, of hats around
the walks' limits and of the large part itself, on both sides of each rule."""
import numpy as np
import pytest

from test_gpu_hull_lists import CFG, M, NONE, T, check, hat, lattice, sphere

pytestmark = pytest.mark.gpu


def ball(n, seed):
    return M.Mesh(np.random.default_rng(seed).uniform(-1, 1, size=(n, 3)).astype(np.float32), NONE)


@pytest.mark.parametrize("largest", [1024, 1025, 2048, 2049])
@pytest.mark.parametrize("count", [152, 153, 304, 305])
def test_widths(oracle, count, largest):
    """152 SMs hold 152 blocks of 1024 threads, 304 of 512."""
    sets = [ball(largest, 1), sphere(600, 2), lattice(300, 3)] + [hat(m) for m in (12, 31, 33, 60, 131, 400)]
    sets += [sphere(5 + k % 30, k) for k in range(count - len(sets))]
    check(T.GpuTree(**CFG, warpMaxNv=1), oracle, sets)
