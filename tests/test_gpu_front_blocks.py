"""As many blocks of the persistent front end fit an SM as its tuning can ask for."""
from __future__ import annotations

import pytest

from przm_b200 import gpu

from .launch_graph import LaunchGraph
from .test_gpu_front import tuning  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [1, 2, 3])
def test_blocks_that_the_tuning_asks_for_are_resident(comp, tuning, blocks):  # noqa: F811
    for k in range(4):
        comp.SetTuning(k, 1, blocks, 2048)
    b = gpu.DeviceBatch(comp, [1 << 20] * 4, gpu.PROFILE_ANS)
    try:
        assert b.info()["front"] == 1 and b.info()["ctas_per_sm"] == blocks
        g = LaunchGraph(lambda s: b.enqueue(s, graph=False))
    finally:
        b.close()
    (front,) = g.named("k_front")
    assert g.blocks_per_sm(front) >= blocks
    g.close()
