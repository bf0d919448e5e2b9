"""Literal runs at the lengths where another number of lanes copies them, one
and several of them in a group of records, at every alignment; and a long run
costs the tokenizer no more than its bytes do elsewhere."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import gpu
from przm_b200 import workloads as W

from .gpu_profile import kernels, total

pytestmark = pytest.mark.gpu

LENS = [127, 128, 129, 143, 511, 2047, 2048, 2049, 2063, 5000]


def runs(lens: list[int], seed: int) -> np.ndarray:
    """Random bytes of each length, a copy of the first 64 bytes after each."""
    r = np.random.default_rng(seed)
    head = r.integers(0, 256, 64, np.uint8)
    return np.concatenate([head] + [np.concatenate([r.integers(0, 256, n, np.uint8), head]) for n in lens])


@pytest.mark.parametrize("n", LENS)
@pytest.mark.parametrize("count", [1, 2, 5])
def test_runs_of_one_length(comp, oracle, n, count):
    for skip in (0, 1, 3):  # where the runs start
        a = runs([7 + skip] + [n] * count, n + skip)
        assert tuple(comp.Tokenize(a)[:3]) == tuple(oracle.tokenize(a))


@pytest.mark.parametrize("seed", range(6))
def test_runs_of_mixed_lengths(comp, oracle, seed):
    a = runs(list(np.random.default_rng(seed).choice(LENS + [3, 20], 40)), seed)
    assert tuple(comp.Tokenize(a)[:3]) == tuple(oracle.tokenize(a))
    assert comp.Compress(a, gpu.PROFILE_D2D)[0] == oracle.compress_p0(a)


def test_long_runs_are_copied_by_the_warp(comp):
    # 32 KiB of literals a tile; the radix sort reads the same bytes: 101 us, the tokenizer 74
    n, count = 1 << 20, 148
    b = gpu.DeviceBatch(comp, [n] * count, gpu.PROFILE_D2D)
    try:
        b.upload(np.concatenate([W.gen("uniform", i % 8, n) for i in range(count)]))
        ks = kernels(lambda: b.enqueue(0, graph=False))
    finally:
        b.close()
    assert total(ks, "k_tokenize") < 0.95 * total(ks, "k_rx_sort"), ks
