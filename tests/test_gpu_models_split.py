"""Streams of symbols of very few bits: the oracle's containers, split or whole,
and not walked one segment after another where whole chains are shorter."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import devmem, gpu

from .gpu_profile import kernels, total
from .test_gpu_segments import encode

pytestmark = pytest.mark.gpu


def rare(n: int, p: float, others: int, seed: int) -> np.ndarray:
    r = np.random.default_rng(seed)
    return np.where(r.random(n) < p, 0, 1 + r.integers(0, others, n)).astype(np.uint8)


@pytest.mark.parametrize("p,others", [(0.9999, 1), (0.999, 3), (0.99, 15), (0.95, 1), (0.5, 1)])
def test_containers(comp, oracle, p, others):
    for parts in ([rare(400_003, p, others, 1)], [rare(200_000 + i, p, others, i) for i in range(12)]):
        for x, g in zip(parts, encode(comp, parts)):
            assert g == oracle.adaptive_vans(x)


def test_user_table_of_few_bits(comp, oracle):
    x = rare(300_000, 0.999, 1, 5)
    freq = np.zeros(256, np.uint16)
    freq[:2] = 4092, 4
    cdf = np.concatenate([[0], np.cumsum(freq)]).astype(np.uint16)
    d_in, d_out = devmem.upload(x), devmem.alloc(2 * len(x) + 1024)
    n, _, _ = comp.VANSEncode4xGPU(d_in.ptr, d_out.ptr, len(x), freq, cdf, b"")
    body = devmem.download(d_out.ptr, n)[8:]
    xs = [int.from_bytes(body[4 * l:4 * l + 4], "little") for l in range(4)]
    at, out = 16, np.zeros(len(x), np.uint8)
    for i in range(len(x)):  # the decoder's step
        l = i & 3
        slot = xs[l] & 4095
        s = int(slot >= 4092)
        out[i] = s
        xs[l] = int(freq[s]) * (xs[l] >> 12) + slot - int(cdf[s])
        while xs[l] < 65536:
            xs[l] = xs[l] << 8 | body[at]
            at += 1
    assert (out == x).all() and at == len(body)


def test_streams_whose_walkers_stay_apart_are_coded_whole(comp):
    # one symbol of 99.9 %: segments were walked one after another for 6.0 ms, and coded in 0.33
    n, count = 1 << 20, 64
    d_in = devmem.upload(np.concatenate([rare(n, 0.999, 1, i) for i in range(count)]))
    d_out = devmem.alloc(count * (2 * n + 1024))
    io, oo = np.arange(count, dtype=np.uint64) * n, np.arange(count, dtype=np.uint64) * (2 * n + 1024)
    ks = kernels(lambda: comp.VANSEncodeBatch(d_in.ptr, io, [n] * count, gpu.NORM_CPU, d_out.ptr, oo), warm=1)
    assert total(ks, "k_seg_") < 0.1 * total(ks, "k_rans"), ks
