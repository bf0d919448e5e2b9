"""Which rANS tasks are coded as segments: the rule by rounds, and its estimate
of the rounds that stay apart against walkers restated here.  (CPU)"""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "przm_b200", "csrc")
SHIM = """
#include "split.h"
extern "C" uint32_t apart(const uint32_t* w, uint32_t n) {
    uint32_t most = 0, off = 0;
    for (uint32_t k = 0; k < n; k++) {
        most = w[k] > most ? w[k] : most;
        off += pz::seg_off_power(w[k]);
    }
    return pz::seg_apart(most, n, off / 4096);
}
extern "C" uint32_t cut(const uint32_t* rounds, const uint32_t* apart, uint32_t n, uint32_t weight) {
    unsigned long long walk[pz::kSegSizes] = {};
    uint32_t most[pz::kSegSizes] = {}, longest = 0;
    for (uint32_t k = 0; k < n; k++) {
        const int i = pz::seg_cut_below(rounds[k]);
        longest = rounds[k] > longest ? rounds[k] : longest;
        if (i < 0) continue;
        walk[i] += pz::seg_walk_cost(rounds[k], apart[k], weight);
        const uint32_t a = pz::seg_apart_rounds(rounds[k], apart[k]);
        most[i] = a > most[i] ? a : most[i];
    }
    return pz::best_cut(walk, most, longest);
}
"""
WHOLE = 0xFFFFFFFF
M = 1 << 18  # rounds of a stream of 1 MiB


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("split")
    (d / "shim.cpp").write_text(SHIM)
    so = d / "shim.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", so, d / "shim.cpp"], check=True)
    lib = C.CDLL(str(so))
    lib.apart.restype = lib.cut.restype = C.c_uint32
    return lib


def apart(rule, weights) -> int:
    f = np.array([w for w in weights if w], np.uint32)
    assert f.sum() == 4096
    return rule.apart(f.ctypes.data_as(C.POINTER(C.c_uint32)), len(f))


def cut(rule, tasks, weight=1) -> int:
    r = np.array([t[0] for t in tasks], np.uint32)
    a = np.array([t[1] for t in tasks], np.uint32)
    p = lambda x: x.ctypes.data_as(C.POINTER(C.c_uint32))
    return rule.cut(p(r), p(a), len(r), weight)


def one(p: float, others: int = 1) -> list[int]:
    """Weights of a symbol of probability p and of others of equal ones."""
    rest = max(others, round(4096 * (1 - p)))
    w = [rest // others + (i < rest % others) for i in range(others)]
    return [4096 - sum(w)] + w


def test_models_of_a_bit_and_more_are_not_held_back(rule):
    for w in ([16] * 256, [1024] * 4, one(0.8, 15), one(0.7), [4096]):
        assert apart(rule, w) & 0xFFFF == 0


@pytest.mark.parametrize("tasks,weight,split", [
    # the figures beside the rule: text as before the models counted
    ([(M, 0)] * 64, 1, True), ([(M, 0)] * 64, 3, True), ([(M, 0)] * 256, 1, True), ([(M, 0)] * 256, 3, False),
    ([(4 * M, 0)], 1, True), ([(12_288, 0)], 1, False), ([(15_000, 0)], 1, False), ([(24_000, 0)], 1, True),
    # 64 streams of 1 MiB, by the probability of their first symbol: whole from where segments take longer
    ([(M, 0.95)] * 64, 1, True), ([(M, 0.99)] * 64, 1, True), ([(M, 0.995)] * 64, 1, False), ([(M, 0.999)] * 64, 1, False),
    ([(M, 0.9999)] * 64, 1, False), ([(M, 0.99)] * 64, 3, False),
    # 64 frames of hexadecimal digits, other batches beside them
    ([(M, "hex")] * 64, 3, True),
    # one stream of 4 MiB
    ([(4 * M, 0.99)], 1, True), ([(4 * M, 0.999)], 1, True), ([(4 * M, 0.9999)], 1, False),
    # one stream of 256 KiB
    ([(M // 4, 0.99)], 1, True), ([(M // 4, 0.995)], 1, True), ([(M // 4, 0.9999)], 1, False),
    # one long stream of text among short ones that stay apart: it alone is split
    ([(4 * M, 0)] + [(20_000, 0.999)] * 200, 1, True),
])
def test_what_is_split(rule, tasks, weight, split):
    t = [(r, apart(rule, near(16, 2) if p == "hex" else one(p)) if p else 0) for r, p in tasks]
    c = cut(rule, t, weight)
    assert (c != WHOLE) == split
    if split and len(set(t)) > 1:
        assert 20_000 <= c < 4 * M


def near(k: int, off: int = 1) -> list[int]:
    """Weights of k equally likely symbols, half of them `off` above and half below."""
    return [4096 // k + off] * (k // 2) + [4096 // k - off] * (k // 2)


TEXT = [205] * 16 + [51] * 16


@pytest.mark.parametrize("count,rounds,weights,split", [
    # the table beside the rule, from where whole chains are the shorter call
    (256, M // 4, TEXT, True), (96, M // 8, TEXT, True), (64, M, TEXT, True), (256, M, TEXT, True),
    (256, M // 4, one(0.9, 15), False), (64, M, one(0.9, 15), True), (256, M, one(0.9, 15), True),
    (256, M // 4, one(0.95, 15), False), (96, M // 8, one(0.95, 15), False), (64, M, one(0.95, 15), True), (256, M, one(0.95, 15), False),
    (256, M // 4, one(0.97, 15), False), (96, M // 8, one(0.97, 15), False), (64, M, one(0.97, 15), True), (256, M, one(0.97, 15), False),
    (256, M // 4, near(2), False), (96, M // 8, near(2), False), (64, M, near(2), True), (256, M, near(2), False),
    (256, M // 4, near(16), False), (64, M, near(16), True), (256, M, near(16), False),
    (64, M, near(16, 2), True),
    # exact powers of two: few walkers meet, none is missed
    (256, M // 4, [2048] * 2, False), (200, M, [2048] * 2, True), (1, 4 * M, [2048] * 2, True),
])
def test_streams_of_one_kind(rule, count, rounds, weights, split):
    w = weights[:-1] + [weights[-1] + 4096 - sum(weights)]
    assert (cut(rule, [(rounds, apart(rule, w))] * count) != WHOLE) == split


def step(x, f, c):
    """The encoder's step, on arrays of states."""
    x = np.where(x >= f << 20, x >> 16, np.where(x >= f << 12, x >> 8, x))
    return (x // f << 12) + x % f + c


def share_apart(weights: list[int], seed: int, streams: int = 160) -> float:
    """The share of segments of 2048 rounds whose true first state no walker has."""
    w = np.array(weights, np.int64)
    cum = np.concatenate([[0], np.cumsum(w)[:-1]])
    rng = np.random.default_rng(seed)
    k = np.arange(64)
    x = np.concatenate([np.full((streams, 1), 65536, np.int64),
                        np.tile((np.exp2(k % 8 / 8) * 65536).astype(np.int64) << (k // 8), (streams, 1))], 1)
    for i in range(6000 + 4096):
        s = rng.choice(len(w), streams, p=w / 4096)
        f, c = w[s][:, None], cum[s][:, None]
        if i < 6000:  # the true state alone
            x[:, :1] = step(x[:, :1], f, c)
            continue
        x = step(x, f, c)
        if (i - 6000) % 512 == 511 and (i - 6000) // 512 == 5:  # 32 of what is left, in ring order
            for row in x:
                r = row[1:]
                d = r[r != np.roll(r, 1)] if (r != np.roll(r, 1)).any() else r[:1]
                pick = d[np.minimum(np.arange(32), len(d) - 1)] if len(d) <= 32 else d[np.arange(32) * len(d) // 32]
                row[1:] = np.concatenate([pick, pick])
    return float((x[:, 1:] != x[:, :1]).all(1).mean())


@pytest.mark.parametrize("weights", [one(0.999), one(0.99), one(0.98), one(0.95), one(0.9), one(0.99, 15), one(0.8, 15), [16] * 256],
                         ids=["999", "99", "98", "95", "90", "99 of 16", "80 of 16", "uniform"])
def test_the_estimate_against_the_walk(rule, weights):
    # it stands for the slowest of many lanes: not below the mean share by more
    # than 160 segments tell (three standard deviations, 0.12), and above by 0.2 at most
    share, told = share_apart(weights, 3), (apart(rule, weights) & 0xFFFF) / 256
    assert share - 0.12 <= told <= share + 0.2, (share, told)


@pytest.mark.parametrize("weights", [near(2), near(2, 2), near(4), near(16), [2048, 1024, 513, 255, 256], near(2, 32), [2048, 2048], [1024] * 4, [2048, 1024, 512, 256, 256]],
                         ids=["2", "2 by 2", "4", "16", "unequal", "2 by 32", "exact 2", "exact 4", "exact unequal"])
def test_the_estimate_near_powers_of_two(rule, weights):
    # not below the mean share, as above; above it by what the slowest lane takes
    # more (0.8 where the mean is 0.2 to 0.45), and nothing where none is missed
    share, told = share_apart(weights, 4), (apart(rule, weights) & 0xFFFF) / 256
    assert share - 0.12 <= told <= (0.8 if share > 0.1 else share + 0.2), (share, told)
