"""Command execution by blocks of 1024 threads (a frame an SM or fewer) and of
512, on the same frames: rounds trips at the edges of both tiles and chunks,
what is left to the walk after whole chunks, and damaged frames."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import gpu
from przm_b200 import workloads as W

from .gpu_profile import kernels
from .test_gpu_exec import decode, flat_frame, inputs, period

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def filled(frames, caps, threads, sms):
    """The frames in calls that take blocks of `threads`: a long frame behind them, repeated past the SM count for 512."""
    long = flat_frame(b"\xfa" + b"\x00" * 1250, b"", bytes(range(8)), 8 + 5000)
    if threads == 1024:
        step = sms - 1
        return [(frames[i:i + step] + [long], caps[i:i + step] + [5008]) for i in range(0, len(frames), step)]
    extra = max(1, sms + 1 - len(frames))
    return [(frames + [long] * extra, caps + [5008] * extra)]


def run(comp, frames, caps, threads, sms, shift=0):
    st, outs = [], []
    for f, c in filled(frames, caps, threads, sms):
        s, o = decode(comp, f, c, shift)
        keep = min(len(frames) - len(st), len(f))
        keep -= keep == len(f)  # (the long one behind)
        st += [int(x) for x in s[:keep]]
        outs += o[:keep]
        assert s[-1] == 0
    return st, outs


@pytest.mark.parametrize("threads", [1024, 512])
def test_the_calls_take_the_block_size(comp, sms, threads):
    f = comp.Compress(period(5, 9000), 1)[0]
    (call, caps), = filled([f], [9000], threads, sms)
    names = [n for n, _ in kernels(lambda: decode(comp, call, caps))]
    assert [n for n in names if n.startswith("k_dec_exec<")] == [f"k_dec_exec<{threads}u>"], names


@pytest.mark.parametrize("threads", [1024, 512])
@pytest.mark.parametrize("profile", [0, 1, 2, 3])
@pytest.mark.parametrize("shift", [0, 3])
def test_round_trips(comp, sms, threads, profile, shift):
    xs = inputs() + [period(p, n, p) for p in (8191, 8192, 8193) for n in (8192, 8193, 16_384, 40_001)]
    st, outs = run(comp, [comp.Compress(x, profile)[0] for x in xs], [len(x) for x in xs], threads, sms, shift)
    assert st == [0] * len(xs)
    bad = [i for i, (x, o) in enumerate(zip(xs, outs)) if x.tobytes() != o]
    assert not bad, bad


@pytest.mark.parametrize("threads", [1024, 512])
def test_hand_over_after_whole_chunks(comp, sms, threads):
    lits = bytes(range(8))
    frames, want = [], []
    for k in (0, 1, 510, 511, 512, 1022, 1023, 1024, 1025, 2047, 2048, 3000):  # repeats before the opcode
        head, body = b"\xfa" + b"\x00" * k, lits + bytes([7]) * (4 * k)
        d = len(body)
        frames.append(flat_frame(head + b"\xc7\x0c", b"", lits, d + 16))  # 16 bytes from four back
        want.append((0, body + (body[-4:] * 4)))
        frames.append(flat_frame(head + b"\xe0\x01", b"", lits, d + 16))  # a dictionary word: not taken
        frames.append(flat_frame(head + b"\xf2", b"", lits, d + 16))      # no opcode
        frames.append(flat_frame(head + b"\x8f", b"\x08", lits, d + 40))  # its varint is missing
        frames.append(flat_frame(head, b"", lits, d + 1))                 # commands end early
        want += [(None, None)] * 4
    st, outs = run(comp, frames, [max(int.from_bytes(f[5:8], "little"), 1) for f in frames], threads, sms)
    unsupported, corrupt = st[1], st[2]
    assert unsupported != 0 and corrupt not in (0, unsupported)
    for i in range(0, len(frames), 5):
        assert st[i:i + 5] == [0, unsupported, corrupt, corrupt, corrupt]
        assert outs[i] == want[i][1]


def test_damaged_frames_alike_in_both(comp, sms):
    rng = np.random.default_rng(41)
    frames = []
    for p in (1, 2, 3):
        for x in (W.gen("records", 6, 60_000), W.gen("markov", 5, 20_000), W.gen("table", 4, 30_000)):
            fr = comp.Compress(x, p)[0]
            frames += [fr[:-1], fr[:len(fr) // 2]]
            for _ in range(60):
                b = bytearray(fr)
                b[int(rng.integers(8, len(b)))] ^= 1 << int(rng.integers(0, 8))
                frames.append(bytes(b))
    caps = [60_000] * len(frames)
    a, b = run(comp, frames, caps, 1024, sms), run(comp, frames, caps, 512, sms)
    assert a[0] == b[0]
    assert 20 < sum(s == 0 for s in a[0]) < len(frames)
    assert [o for s, o in zip(*a) if s == 0] == [o for s, o in zip(*b) if s == 0]
