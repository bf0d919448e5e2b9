"""The Mode 12 chains in segments: sections at the sizes where the split
begins, at segment and stitch edges, and of distances whose walkers do not
meet (one distance, two in turn, a slow drift), against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import devmem

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 33, 63, 64, 6144, 6145, 8191, 8192, 8193, 16_383, 16_384, 16_385, 40_001]
KINDS = {
    "log": lambda n: np.exp(np.random.default_rng(n).uniform(0, np.log(1 << 20), n)),
    "one": lambda n: np.full(n, 96), "two": lambda n: np.where(np.arange(n) & 1, 5, 70_000),
    "drift": lambda n: 1 + np.arange(n) * 3, "near": lambda n: np.random.default_rng(n).integers(1, 9, n),
}


def sections(comp, parts):
    counts = [len(p) for p in parts]
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint64)
    caps = [5 * n + 64 for n in counts]
    outs = np.concatenate([[0], np.cumsum([(c + 15) // 16 * 16 for c in caps])]).astype(np.uint64)
    d_in, d_out = devmem.upload(np.concatenate(parts)), devmem.alloc(int(outs[-1]) + 64)
    got = comp.PackageOffsetsBatch(d_in.ptr, offs[:-1], counts, d_out.ptr, outs[:-1], caps)
    return [devmem.download(d_out.ptr + int(o), int(n)) for o, n in zip(outs, got)]


@pytest.mark.parametrize("kind", sorted(KINDS))
def test_sections_at_segment_edges(comp, oracle, kind):
    parts = [np.clip(KINDS[kind](n), 1, (1 << 24)).astype(np.uint32) for n in SIZES]
    for p, g in zip(parts, sections(comp, parts)):
        assert g == oracle.package_offsets(p), (kind, len(p))


def test_one_long_section(comp, oracle):
    p = np.clip(KINDS["log"](700_003), 1, 1 << 24).astype(np.uint32)
    assert sections(comp, [p]) == [oracle.package_offsets(p)]
