"""Chains of Mode 12 codes of one segment beside those of several: the oracle's
sections and frames, and short ones take no launch for their totals."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import devmem, gpu
from przm_b200 import workloads as W

from .gpu_profile import kernels
from .test_gpu_mode12 import KINDS, sections

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1], [6144], [6144, 3, 0, 512], [6145, 1, 6144, 20_000, 2]])
def test_chains_of_one_segment_beside_longer_ones(comp, oracle, sizes):
    parts = [np.clip(KINDS["log"](n), 1, 1 << 24).astype(np.uint32) for n in sizes if n]
    for p, g in zip(parts, sections(comp, parts)):
        assert g == oracle.package_offsets(p), len(p)


def test_frames_with_and_without_segments(comp, oracle):
    xs = [W.gen("records", 1, 300_000), W.gen("markov", 2, 5000), W.gen("table", 3, 100), W.gen("markov", 4, 900_000)]
    for x, f in zip(xs, comp.CompressBatch(xs, gpu.PROFILE_ANS_DIST)[0]):
        assert f == oracle.compress_p2(x)


def test_launches_of_short_chains(comp):
    d = np.array([5], np.uint32)
    d_in, d_out = devmem.upload(d), devmem.alloc(64)
    ks = [n for n, _ in kernels(lambda: comp.PackageOffsetsBatch(d_in.ptr, [0], [1], d_out.ptr, [0], [64]))]
    assert len(ks) == 5, ks  # codes, chain, its stream, plan, section
    b = gpu.DeviceBatch(comp, [5000] * 3, gpu.PROFILE_ANS_DIST)
    try:
        b.upload(np.concatenate([W.gen("markov", i, 5000) for i in range(3)]))
        ks = [n for n, _ in kernels(lambda: b.enqueue(0, graph=False))]
    finally:
        b.close()
    assert not any(n.startswith("k_m12_sum") for n in ks), ks
