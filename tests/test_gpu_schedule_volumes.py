"""A tree's tables under each of the autotuner's schedules, bit for bit: seeds
of 2,049-4,096 points, above the size from which a part's flux is added over a
block's lanes and below the largest parent a schedule leaves to a warp, and
sizes around it, far from the origin, where the faces' flux cancels most."""
import numpy as np
import pytest

from conftest import pkg

G, M, T = pkg("meshgen"), pkg("mesh"), pkg("tree")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,depth,n", [(26, 1, 4), (34, 1, 12), (34, 2, 2), (44, 2, 2)])
def test_schedules_give_the_same_volumes(grid, depth, n):
    seeds = [M.normalize(G.blob_mesh(10, grid, seed=k))[0] for k in range(3, 3 + n)]
    seeds = [M.Mesh(m.verts + np.float32([1000, -700, 400]), m.tris) for m in seeds]
    g = T.GpuTree(width=6, width2=3, depth=depth, nConcaveEdges=64, hullMaxVerts=8192, vertexCap=128 << 20,
                  triCap=128 << 20, edgeCap=8 << 20, scratchWords=128 << 20, hullBudgetBytes=2 << 30)
    planes = [G.random_planes(m, 256, seed=k) for k, m in enumerate(seeds)]
    runs, schedules = [], set()
    for _ in range(4):
        r = g.run(seeds, planes)
        assert not r["overflow"]
        s = g.schedule()
        schedules.add((s["warpMaxNv"], s["bigJobNv"]))
        runs.append((r["seeds"], np.asarray(g.parts(0, len(seeds) + 2 * r["validJobs"]))[:, :8].tobytes()))
    assert len(schedules) == 4, schedules
    assert len(runs[0][1]) > 32 * 200 * n
    assert all(x == runs[0] for x in runs[1:])
