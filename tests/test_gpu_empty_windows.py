"""Inputs where whole windows of match descriptors are empty, alone and beside
others, tokenize to the oracle's streams, and a window without a descriptor
costs the tokenizer no more than its loads."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import gpu
from przm_b200 import workloads as W

from .gpu_profile import kernels, total

pytestmark = pytest.mark.gpu


def some_matches(n: int, where: list[int]) -> np.ndarray:
    """Random bytes with a run of 60 equal bytes and a copy of the 40 bytes before, at each place."""
    a = W.gen("uniform", n, n)
    for p in where:
        a[p:p + 60] = 7
        a[p + 61:p + 101] = a[p - 41:p - 1]
    return a


CASES = [(1000, []), (33_000, []), (65_536, []), (65_537, []), (200_000, []),
         (65_536, [1000]), (65_536, [32_768 - 30, 50_000]), (40_000, [1024 - 50, 3 * 1024 + 31]), (200_000, [8192 * 3 - 8, 150_001])]


@pytest.mark.parametrize("n,where", CASES)
def test_streams_with_empty_windows(comp, oracle, n, where):
    a = some_matches(n, where)
    assert tuple(comp.Tokenize(a)[:3]) == tuple(oracle.tokenize(a))
    assert comp.Compress(a, gpu.PROFILE_D2D)[0] == oracle.compress_p0(a)


def test_windows_without_a_descriptor_cost_only_their_loads(comp):
    # k_tile_find looks at the same bytes: 100 us for these, the tokenizer 45
    n, count = 65_536, 148
    b = gpu.DeviceBatch(comp, [n] * count, gpu.PROFILE_D2D)
    try:
        b.upload(np.concatenate([W.gen("uniform", i, n) for i in range(count)]))
        ks = kernels(lambda: b.enqueue(0, graph=False))
    finally:
        b.close()
    assert total(ks, "k_tokenize") < 0.65 * total(ks, "k_tile_find"), ks
