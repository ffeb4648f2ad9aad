"""Plan and emit on warps, on blocks with a warp's flux sums, and on blocks with
their own: the same tables as the oracle's on both sides of each rule (few
jobs, many jobs of small parents, mid-sized parents, large parents)."""
import pytest

import parity
from conftest import pkg

G, M, T = pkg("meshgen"), pkg("mesh"), pkg("tree")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,depth,width", [
    ("few small", 2, 3), ("many small", 3, 6), ("middle", 2, 3), ("middle many", 2, 6), ("large", 1, 3)])
def test_forms_match_oracle(oracle, name, depth, width):
    seeds = {"few small": [G.staircase(3), M.unit_cube()],
             # 36 x (6 + 32) = 1,368, 4,104 and 12,312 jobs, on both sides of 16 per SM, parents of 20 points
             "many small": [G.staircase(3)] * 36,
             "middle": [G.noisy_icosphere(2, seed=1), M.normalize(G.blob_mesh(6, 24, seed=2))[0]],
             "middle many": [G.noisy_icosphere(2, seed=k) for k in range(40)],
             "large": [M.normalize(G.blob_mesh(10, 42, seed=3))[0]]}[name]
    planes = [G.random_planes(m, 32, seed=k) for k, m in enumerate(seeds)] if "many" in name else None
    cfg = dict(width=width, width2=3, depth=depth, nConcaveEdges=8, hullMaxVerts=4096, autotune=0,
               vertexCap=64 << 20, triCap=64 << 20, edgeCap=4 << 20, scratchWords=64 << 20, hullBudgetBytes=2 << 30)
    g, o = T.GpuTree(**cfg), oracle.OracleTree(**cfg)
    rg, ro = g.run(seeds, planes), o.run(seeds, planes)
    assert not rg["overflow"]
    parity.compare_level_tables(g, o, rg, ro, len(seeds), label=name)
    parity.compare_seeds(rg, ro, label=name)
