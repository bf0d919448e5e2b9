"""The tokenizer's walk by precomputed successors, at the edges of its windows
(1024 descriptors), with runs, lookahead, extended matches and more distances
than repeat slots; and frames whose streams several blocks gather."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def runs(n, every, length):
    """Noise with a run of one byte every `every` bytes."""
    a = np.random.default_rng(every).integers(0, 256, n, np.uint8)
    for i, o in enumerate(range(every - length // 2, n - length, every)):
        a[o:o + length] = i & 255
    return a


def periods(n, *ps):
    """Stretches repeated at alternating distances."""
    rng = np.random.default_rng(sum(ps))
    a = rng.integers(0, 256, n, np.uint8)
    o, i = max(ps), 0
    while o + 40 < n:
        p, m = ps[i % len(ps)], 8 + (i * 7) % 30
        for k in range(m):
            a[o + k] = a[o + k - p]
        o += m + (i % 5)
        i += 1
    return a


INPUTS = {
    "runs-1024": lambda n: runs(n, 1024, 40), "runs-8192": lambda n: runs(n, 8192, 300), "runs-11": lambda n: runs(n, 64, 11),
    "runs-12": lambda n: runs(n, 64, 12), "zeros": lambda n: np.zeros(n, np.uint8),
    "far": lambda n: np.resize(np.random.default_rng(3).integers(0, 256, 9000, np.uint8), n),
    "two": lambda n: periods(n, 96, 160), "four": lambda n: periods(n, 16, 64, 256, 1000),
    "records": lambda n: W.gen("records", n, n), "text": lambda n: W.gen("markov", n, n),
}


@pytest.mark.parametrize("kind", sorted(INPUTS))
@pytest.mark.parametrize("n", [1023, 1025, 8191, 32_769, 65_536, 65_537, 300_001])
def test_streams_match_oracle(comp, oracle, kind, n):
    a = INPUTS[kind](n)
    cmd, off, lit, _ = comp.Tokenize(a)
    want = oracle.tokenize(a)
    assert (cmd, off, lit) == tuple(bytes(x) for x in want[:3])


@pytest.mark.parametrize("profile,want", [(0, "compress_p0"), (1, "compress_p1")])
def test_frames_gathered_in_parts(comp, oracle, profile, want):
    for n in (8 * 32_768, 16 * 32_768 - 1, 1_700_003):
        a = W.gen("records", n, n)
        assert comp.Compress(a, profile)[0] == getattr(oracle, want)(a)
