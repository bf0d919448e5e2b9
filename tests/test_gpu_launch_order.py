"""What the kernels of a batch wait for: the Mode 12 chains run beside the rANS
launches, which wait for the walks of their own segments alone."""
from __future__ import annotations

import pytest

from przm_b200 import gpu

from .launch_graph import LaunchGraph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("profile", [gpu.PROFILE_ANS, gpu.PROFILE_ANS_DIST, gpu.PROFILE_ANS_SHEAF])
def test_rans_waits_for_its_walks_and_no_chain(comp, profile):
    b = gpu.DeviceBatch(comp, [2_500_007, 900_001], profile)
    try:
        g = LaunchGraph(lambda s: b.enqueue(s, graph=False))
    finally:
        b.close()
    walks = {int(x) for x in g.named("k_seg_walk")}
    chains = {int(x) for x in g.named("k_m12_")}
    assert len(walks) == 2 and bool(chains) == (profile >= gpu.PROFILE_ANS_DIST)
    for part in ("k_seg_resolve", "k_rans"):
        (x,) = g.named(part)
        assert walks <= g.waits_for(x)
        assert not chains & g.waits_for(x), part
    (plan,) = g.named("k_plan")
    assert walks | chains <= g.waits_for(plan)
    g.close()
