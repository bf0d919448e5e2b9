"""The gather of many short inputs, and of inputs whose tiles several blocks
share: streams as the oracle's, and a short input costs it no more than the
assembly of its frame does."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import devmem, gpu
from przm_b200 import workloads as W

from .gpu_profile import kernels, total

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [1, 7, 8, 15, 16, 17, 63, 65])
@pytest.mark.parametrize("count", [1, 3])
def test_tiles_shared_by_blocks(comp, oracle, tiles, count):
    # parts of a frame: its tiles / 8, as long as the blocks are at most two an SM
    xs = [W.gen("markov", tiles + i, tiles * 32_768 - 5 * i) for i in range(count)]
    b = gpu.DeviceBatch(comp, [len(x) for x in xs], gpu.PROFILE_ANS)
    try:
        for x, o in zip(xs, b.in_offs):
            devmem.upload_to(b.d_in + int(o), x)
        b.enqueue(graph=False)
        for x, o, n in zip(xs, b.out_offs, b.frame_sizes()):
            assert devmem.download(b.d_out + int(o), int(n)) == oracle.compress_p1(x)
    finally:
        b.close()


def test_short_inputs_do_not_wait_for_divisions(comp):
    # the assembly of these frames: 397 us, the gather 483
    n, count = 200, 20_000
    b = gpu.DeviceBatch(comp, [n] * count, gpu.PROFILE_D2D)
    try:
        b.upload(np.concatenate([W.mixture(9 + i % 40, n)[0] for i in range(count)]))
        ks = kernels(lambda: b.enqueue(0, graph=False))
    finally:
        b.close()
    assert total(ks, "k_gather") < 1.4 * total(ks, "k_assemble"), ks
