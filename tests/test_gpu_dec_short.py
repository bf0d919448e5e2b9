"""Short frames are decoded by a warp each: the same bytes and statuses as by
the command blocks (which a longer frame in the call brings on), at the sizes
and frame counts where one goes over to the other, and no slower than the
other stages of the call."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import devmem, gpu
from przm_b200 import workloads as W

from .gpu_profile import kernels, total
from .test_gpu_exec import flat_frame

pytestmark = pytest.mark.gpu


def layout(frames, caps):
    so = np.concatenate([[0], np.cumsum([len(f) for f in frames])]).astype(np.uint64)
    do = np.concatenate([[0], np.cumsum([(c + 15) // 16 * 16 for c in caps])]).astype(np.uint64)
    d_src = devmem.upload(np.frombuffer(b"".join(frames) + bytes(64), np.uint8))
    return d_src, devmem.alloc(int(do[-1]) + 64), so, do


def decode(comp, frames, caps):
    d_src, d_dst, so, do = layout(frames, caps)
    st, ln = comp.DecompressBatchDevice(d_src.ptr, so[:-1], [len(f) for f in frames], d_dst.ptr, do[:-1], caps)
    host = devmem.download(d_dst.ptr, int(do[-1]))
    return [int(x) for x in st], [host[int(a):int(a) + int(n)] for a, n in zip(do, ln)]


def frames_up_to(comp, cap, profile):
    xs = [W.gen(k, 3 * n + profile, n) for k in ("records", "markov", "table", "uniform") for n in (1, 7, 100, cap // 2, cap - 1, cap)]
    xs += [np.zeros(cap, np.uint8), np.resize(np.arange(5, dtype=np.uint8), cap)]
    return [comp.Compress(x, profile)[0] for x in xs], [len(x) for x in xs], [x.tobytes() for x in xs]


@pytest.mark.parametrize("profile", [0, 1, 2, 3])
@pytest.mark.parametrize("count,cap", [(1, 768), (148, 768), (149, 768), (296, 769), (297, 1536), (1184, 1537), (1185, 2304), (1300, 2305)])
def test_same_bytes_at_the_borders(comp, profile, count, cap):
    fr, caps, want = frames_up_to(comp, cap, profile)
    pick = [i % len(fr) for i in range(count - 1)] + [len(fr) - 3]  # (the last: `cap` bytes)
    st, outs = decode(comp, [fr[i] for i in pick], [caps[i] for i in pick])
    assert st == [0] * count
    bad = [i for i, o in zip(pick, outs) if o != want[i]]
    assert not bad, bad


def test_damaged_short_frames_as_in_a_call_with_a_long_one(comp):
    rng = np.random.default_rng(5)
    base = [comp.Compress(W.gen(k, 9, 700), p)[0] for k in ("records", "markov") for p in (0, 1, 2)]
    lits = bytes(range(8))
    frames = [flat_frame(b"\xfa" + t, o, lits, n) for t, o, n in (
        (b"\xc7\x0c", b"", 24), (b"\xe0\x01", b"", 24), (b"\xf2", b"", 24), (b"\x8f", b"\x08", 40), (b"\x84", b"\x09", 16), (b"", b"", 9))]
    for fr in base:
        for _ in range(20):
            b = bytearray(fr)
            b[int(rng.integers(8, len(b)))] ^= 1 << int(rng.integers(0, 8))
            frames.append(bytes(b))
    caps = [700] * len(frames)
    short = decode(comp, frames, caps)
    big = comp.Compress(W.gen("records", 2, 20_000), 1)[0]
    st, outs = decode(comp, frames + [big], caps + [20_000])
    assert st[-1] == 0
    assert short[0] == st[:-1]
    assert [o for s, o in zip(*short) if s == 0] == [o for s, o in zip(st[:-1], outs) if s == 0]


def test_flat_frames_of_a_call_of_many(comp):
    # more than 8 frames an SM, one of them long: flat streams of short commands are walked, the others are not
    xs = [W.gen(("records", "uniform", "table")[i % 3], i, 300 + 37 * (i % 90)) for i in range(1200)] + [W.gen("records", 1, 40_000)]
    frames = [comp.Compress(x, i % 2)[0] for i, x in enumerate(xs)]
    st, outs = decode(comp, frames, [len(x) for x in xs])
    assert st == [0] * len(xs)
    assert [o == x.tobytes() for o, x in zip(outs, xs)] == [True] * len(xs)


def test_launches_of_a_short_frame(comp):
    fr = np.frombuffer(comp.Compress(W.gen("records", 1, 100), 1)[0], np.uint8)
    ks = [n for n, _ in kernels(lambda: comp.Decompress(fr))]
    assert len(ks) == 6, ks  # parse, static models, adaptive bodies, prefix, sheaf, commands


@pytest.mark.parametrize("count,listed", [(19, False), (512, False), (513, True)])
def test_short_bodies_need_no_list(comp, count, listed):
    x = W.gen("markov", 1, 700)
    fr = comp.Compress(x, 1)[0]
    ks = [n for n, _ in kernels(lambda: decode(comp, [fr] * count, [700] * count))]
    assert ("k_dec_lists" in ks) == listed, ks
    st, outs = decode(comp, [fr] * count, [700] * count)
    assert st == [0] * count and outs == [x.tobytes()] * count


@pytest.mark.parametrize("profile", [0, 1])
def test_many_short_frames_cost_less_than_empty_slots(comp, profile):
    # k_dec_static only finds that these frames' 160 000 slots have no static body: 112 us
    n, count = 200, 20_000
    xs = [W.gen("records", i, n) for i in range(40)]
    fr = [comp.Compress(x, profile)[0] for x in xs]
    frames = [fr[i % 40] for i in range(count)]
    d_src, d_dst, so, do = layout(frames, [n] * count)
    ln = [len(f) for f in frames]
    ks = kernels(lambda: comp.DecompressBatchDevice(d_src.ptr, so[:-1], ln, d_dst.ptr, do[:-1], [n] * count))
    assert total(ks, "k_dec_exec", "k_dec_adaptive") < total(ks, "k_dec_static"), ks


@pytest.mark.parametrize("profile", [0, 1])
def test_frames_of_byte_runs_are_walked(comp, profile):
    # k_dec_static only finds that the 20 000 slots have no static body: 16 us
    xs = [np.full(60_000 + i % 7, i % 3, np.uint8) for i in range(2500)]
    frames = [comp.Compress(x, profile)[0] for x in xs[:21]]
    frames = [frames[i % 21] for i in range(len(xs))]
    caps = [len(x) for x in xs]
    st, outs = decode(comp, frames[:60], caps[:60])
    assert st == [0] * 60 and outs == [x.tobytes() for x in xs[:60]]
    d_src, d_dst, so, do = layout(frames, caps)
    ln = [len(f) for f in frames]
    ks = kernels(lambda: comp.DecompressBatchDevice(d_src.ptr, so[:-1], ln, d_dst.ptr, do[:-1], caps))
    assert total(ks, "k_dec_exec<") < 2 * total(ks, "k_dec_static"), ks


@pytest.mark.parametrize("count,way", [(1, 0), (18, 0), (19, 1), (407, 1), (408, 2), (900, 2)])
def test_ways_to_the_adaptive_bodies(comp, count, way):
    # a block per slot up to one an SM, then in the list's order, then blocks that stay (148 SMs, eight slots a frame)
    xs = [W.gen("markov", i, 5000 + 13 * i) for i in range(20)]
    fr = [comp.Compress(x, 1)[0] for x in xs]
    pick = [i % 20 for i in range(count)]
    frames, caps = [fr[i] for i in pick], [len(xs[i]) for i in pick]
    st, outs = decode(comp, frames, caps)
    assert st == [0] * count and [o == xs[i].tobytes() for o, i in zip(outs, pick)] == [True] * count
    ks = [n for n, _ in kernels(lambda: decode(comp, frames, caps))]
    assert f"k_dec_adaptive<{way}>" in ks, ks


@pytest.mark.parametrize("profile", [0, 1])
@pytest.mark.parametrize("count,n", [(297, 2400), (600, 6000), (1300, 12_000), (1300, 3000), (4400, 2400)])
def test_frames_of_few_commands_in_calls_of_many(comp, profile, count, n):
    # some walked, some by blocks in the same call: rare ones among zeros, a short period, digits, records, text
    rng = np.random.default_rng(n)
    xs = []
    for i in range(5):
        m = n - 7 * i
        xs += [(rng.random(m) < 0.003).astype(np.uint8), np.resize(rng.integers(0, 256, 37).astype(np.uint8), m),
               np.frombuffer(b"0123456789abcdef", np.uint8)[rng.integers(0, 16, m)], W.gen("records", i, m), W.gen("markov", i, m)]
    fr = [comp.Compress(x, profile)[0] for x in xs]
    pick = [i % len(xs) for i in range(count)]
    st, outs = decode(comp, [fr[i] for i in pick], [len(xs[i]) for i in pick])
    assert st == [0] * count and [o == xs[i].tobytes() for o, i in zip(outs, pick)] == [True] * count


def test_rare_ones_are_walked(comp):
    # 3000 frames of 3000 bytes, each a few matches: 123 us in blocks, 16 walked and 12 for the blocks that leave them
    x = (np.random.default_rng(1).random(3000) < 0.003).astype(np.uint8)
    fr = comp.Compress(x, 1)[0]
    ks = kernels(lambda: decode(comp, [fr] * 3000, [3000] * 3000))
    assert total(ks, "k_dec_exec") < 3 * total(ks, "k_dec_static"), ks  # (which only finds that there is nothing for it: 19 us)
