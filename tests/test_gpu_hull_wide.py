"""Block hulls whose insertion sees more faces than a walk or the single-pick
step holds (low hats on m-gon prisms), in batches with a part above 2,048
points, so that one wave of 1024- and 512-thread blocks and more than one wave
all occur: the oracle's faces and volumes."""
import pytest
import torch

from test_gpu_hull_lists import CFG, check, hat, sphere
from conftest import pkg

T = pkg("tree")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("waves", [0, 1, 2])
def test_hats_in_wide_blocks(oracle, waves):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sets = [hat(m) for m in (1100, 700, 200, 131, 33)]
    assert sets[0].nv > 2048
    count = 1 if waves == 0 else waves * sms + 1
    pad = [sphere(5, k) for k in range(max(0, count - len(sets)))]
    check(T.GpuTree(**CFG, warpMaxNv=1), oracle, (sets[:1] if waves == 0 else sets) + pad)
