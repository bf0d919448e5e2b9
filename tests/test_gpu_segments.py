"""Long rANS tasks coded as independent segments: the containers and frames
must be the oracle's bytes at the sizes where the split begins, at segment and
stitch edges, at every source alignment, and on symbols whose walkers never
meet (runs of one symbol, two symbols, a nearly constant stream)."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import devmem, gpu
from przm_b200 import workloads as W

pytestmark = pytest.mark.gpu

WARM, SEG = 4096, 2048            # rounds walked above a segment, shortest segment
FIRST = 4 * 2 * (WARM + SEG) + 1   # symbols of the shortest split task


def skewed(n: int) -> np.ndarray:
    return np.minimum(np.random.default_rng(n).geometric(0.97, n) - 1, 255).astype(np.uint8)


def runs(n: int) -> np.ndarray:
    return np.repeat(np.array([7, 200, 7, 9], np.uint8), -(-n // 4))[:n]


KINDS = {
    "zipf": lambda n: W.zipf(n, n), "uniform": lambda n: W.gen("uniform", n, n), "skewed": skewed, "runs": runs,
    "constant": lambda n: np.full(n, 65, np.uint8), "two": lambda n: (np.arange(n) // 3 & 1).astype(np.uint8),
    "records": lambda n: W.gen("records", n, n),
}
SIZES = [FIRST - 1, FIRST, FIRST + 1, FIRST + 3, 4 * (WARM + 3 * SEG) - 1, 4 * (WARM + 3 * SEG), 4 * (WARM + 3 * SEG) + 2,
         16 * 4096, 16 * 4096 + 5, 300_001]


def encode(comp, parts, gap=0):
    """The containers of the streams, one call; stream i starts gap * i bytes past a 64-byte boundary."""
    lens = [len(p) for p in parts]
    offs, o = [], 0
    for i, n in enumerate(lens):
        offs.append(o + gap * i % 64)
        o += (n + 127) // 64 * 64
    host = np.zeros(o + 64, np.uint8)
    for p, a in zip(parts, offs):
        host[a:a + len(p)] = p
    outs = np.concatenate([[0], np.cumsum([2 * n + 1024 for n in lens])]).astype(np.uint64)
    d_in, d_out = devmem.upload(host), devmem.alloc(int(outs[-1]))
    got = comp.VANSEncodeBatch(d_in.ptr, offs, lens, gpu.NORM_CPU, d_out.ptr, outs[:-1])
    return [devmem.download(d_out.ptr + int(a), int(n)) for a, n in zip(outs, got)]


@pytest.mark.parametrize("kind", sorted(KINDS))
def test_containers_at_segment_edges(comp, oracle, kind):
    parts = [KINDS[kind](n) for n in SIZES]
    for gap in (0, 1):  # aligned sources, then every alignment in turn
        for p, g in zip(parts, encode(comp, parts, gap)):
            assert g == oracle.adaptive_vans(p), (kind, len(p), gap)


@pytest.mark.parametrize("kind", ["zipf", "skewed"])
def test_one_long_stream(comp, oracle, kind):
    p = KINDS[kind](3_000_005)
    assert encode(comp, [p]) == [oracle.adaptive_vans(p)]


def test_many_streams_take_longer_segments(comp, oracle):
    # together far more segments than one call may have at the shortest length
    parts = [W.gen("records" if i % 3 else "uniform", i, 600_000 + 17 * i) for i in range(40)]
    for p, g in zip(parts, encode(comp, parts)):
        assert g == oracle.adaptive_vans(p)


@pytest.mark.parametrize("profile,want", [(1, "compress_p1"), (3, "compress_p3")])
def test_frames_with_long_command_streams(comp, oracle, profile, want):
    # records: op, meta and var streams long enough to be split, as Meta8 and adaptive tasks
    a = W.gen("records", 21, 2_500_007)
    assert comp.Compress(a, profile)[0] == getattr(oracle, want)(a)


@pytest.mark.parametrize("graph", [False, True])
def test_meta8_walk_beside_the_adaptive_one(comp, oracle, graph):
    # new bytes in the same buffers: a walk not waited for would leave the last call's states
    b = gpu.DeviceBatch(comp, [2_500_007, 900_001], gpu.PROFILE_ANS)
    try:
        for seed in (21, 22, 23):
            xs = [W.gen("records", seed, 2_500_007), W.gen("records", seed + 50, 900_001)]
            for x, o in zip(xs, b.in_offs):
                devmem.upload_to(b.d_in + int(o), x)
            b.enqueue(graph=graph)
            for x, o, n in zip(xs, b.out_offs, b.frame_sizes()):
                assert devmem.download(b.d_out + int(o), int(n)) == oracle.compress_p1(x)
    finally:
        b.close()
