"""The decoder's parallel command execution at the edges of its chunks (512
commands), tiles (4096 bytes) and output alignments, on long self-overlapping
matches, and the frames it leaves to the serial walk."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import devmem, gpu
from przm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def decode(comp, frames, caps, shift=0):
    """One device call; frame i's output starts shift * i bytes past a 16-byte boundary."""
    so, do, o, d = [], [], 0, 0
    for i, (f, c) in enumerate(zip(frames, caps)):
        so.append(o)
        do.append(d + shift * i % 16)
        o += len(f) + 16
        d += (c + 47) // 16 * 16
    src = np.zeros(o + 64, np.uint8)
    for f, x in zip(frames, so):
        src[x:x + len(f)] = np.frombuffer(f, np.uint8)
    d_src, d_dst = devmem.upload(src), devmem.alloc(d + 64)
    st, ln = comp.DecompressBatchDevice(d_src.ptr, so, [len(f) for f in frames], d_dst.ptr, do, caps)
    return list(st), [devmem.download(d_dst.ptr + x, int(n)) for x, n in zip(do, ln)]


def period(p, n, seed=1):
    return np.resize(np.random.default_rng(seed).integers(0, 256, p, np.uint8), n)


def inputs():
    xs = [period(p, n, p) for p in (1, 2, 3, 7, 100, 4095, 4096, 4097) for n in (4095, 4096, 4097, 12_289, 70_000)]
    xs += [W.gen(k, 40 + n, n) for k in ("records", "table", "markov") for n in (1, 2047, 8192, 65_536, 65_537, 250_003)]
    return xs


@pytest.mark.parametrize("profile", [0, 1, 2, 3])
@pytest.mark.parametrize("shift", [0, 1])
def test_round_trips(comp, profile, shift):
    xs = inputs()
    frames = [comp.Compress(x, profile)[0] for x in xs]
    st, outs = decode(comp, frames, [len(x) for x in xs], shift)
    assert st == [0] * len(xs)
    bad = [i for i, (x, o) in enumerate(zip(xs, outs)) if x.tobytes() != o]
    assert not bad, bad


def flat_frame(cmds: bytes, offs: bytes, lits: bytes, n: int) -> bytes:
    """A frame with flat sections and a 16-bit directory."""
    return (b"PRZM\x00" + n.to_bytes(3, "little") + (len(cmds) + 5).to_bytes(2, "little") +
            (len(offs) + 5).to_bytes(2, "little") + bytes(8) + b"\x00" + len(cmds).to_bytes(4, "little") + cmds +
            b"\x00" + len(offs).to_bytes(4, "little") + offs + lits)


def test_plain_distance_opcodes_and_what_is_around_them(comp):
    lits = bytes(range(8))
    run = b"\xfa"  # eight literals
    frames = [
        flat_frame(run + b"\xc7\x0c", b"", lits, 24),                      # 16 bytes from four back
        flat_frame(run + b"\x00" * 600 + b"\xc4\x05", b"", lits, 8 + 600 * 4 + 9),  # after a whole chunk of repeats
        flat_frame(run + b"\x8f\x7d", b"\x08", lits, 8 + 19 + 0x7d),       # explicit distance, extended length
        flat_frame(run + b"\xf1\x05", b"", lits + b"Z", 13),               # a byte run
        flat_frame(run + b"\xe0\x01", b"", lits, 24),                      # a dictionary word: not taken
        flat_frame(run + b"\xf2", b"", lits, 24),                          # no opcode
        flat_frame(run + b"\x8f", b"\x08", lits, 40),                      # its varint is missing
        flat_frame(run + b"\x84", b"\x09", lits, 16),                      # a distance before the output
        flat_frame(run + b"\x84", b"\x00", lits, 16),                      # a distance of nothing
        flat_frame(run, b"", lits, 9),                                     # commands end early
        flat_frame(run + b"\xfa", b"", lits, 16),                          # literals run out
    ]
    one = bytes([7]) * (600 * 4)
    want = [lits + (lits[4:] * 4), lits + one + bytes([7]) * 9, lits + (lits * 20)[:19 + 0x7d], lits + b"Z" * 5]
    st, outs = decode(comp, frames, [max(int.from_bytes(f[5:8], "little"), 1) for f in frames])
    assert st[:4] == [0] * 4
    for o, w in zip(outs, want):
        assert o == w
    assert st[4] not in (0, st[5]) and st[5] != 0 and st[6:] == [st[5]] * 5


@pytest.mark.parametrize("copies", [1, 12])
def test_edges_of_both_block_sizes(comp, copies):
    # 14 frames take 1024 threads each, 168 frames 512
    lits = bytes(range(8))
    counts = (510, 511, 512, 1022, 1023, 1024)  # commands after the first
    frames = [flat_frame(b"\xfa" + b"\x00" * k, b"", lits, 8 + 4 * k) for k in counts]
    want = [lits + bytes([7]) * (4 * k) for k in counts]
    xs = [x for n in (8191, 8192, 8193, 16_385) for x in (period(5, n), W.gen("records", n, n))]
    frames += [comp.Compress(x, gpu.PROFILE_ANS)[0] for x in xs]
    want += [x.tobytes() for x in xs]
    st, outs = decode(comp, frames * copies, [len(w) for w in want] * copies, 1)
    assert st == [0] * len(outs)
    bad = [i for i, (w, o) in enumerate(zip(want * copies, outs)) if w != o]
    assert not bad, bad
