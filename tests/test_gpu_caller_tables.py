"""VANSEncode4xGPU with tables no normaliser makes: weights above 4096, sums
that are not 4096, symbols of weight 0 and cumulative weights in any order give
the states and bytes of the step as its fields define it."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import devmem

pytestmark = pytest.mark.gpu


def encode(x: np.ndarray, freq: np.ndarray, cdf: np.ndarray) -> bytes:
    """Four lanes from the last symbol down, and their bytes in the container's order."""
    state, bytes_of = [65536] * 4, [[] for _ in range(len(x))]
    for i in range(len(x) - 1, -1, -1):
        f, c, l = int(freq[x[i]]), int(cdf[x[i]]), i & 3
        v = state[l]
        if f == 0:  # no step, no byte
            continue
        t1 = 4096 * f
        k = (v >= t1) + (v >= min(256 * t1, 0xFFFFFFFF))
        bytes_of[i] = [v >> 8 * b & 0xFF for b in range(k)]
        v >>= 8 * k
        w = c | ((4096 - f) & 0xFFFFFFFF) << 13 & 0xFFFFFFFF  # cumulative weight, 4096 - f, (shift)
        q = 0 if f > 4096 else v // f
        state[l] = v + (w & 0x1FFF) + q * (w >> 13 & 0xFFF)
        assert state[l] < 1 << 31
    out = b"".join(s.to_bytes(4, "little") for s in state)
    return out + bytes(b for bs in bytes_of for b in reversed(bs))


def tables(kind: str, rng) -> tuple[np.ndarray, np.ndarray]:
    f = rng.integers(2, 4096, 256)
    c = rng.integers(0, 4097, 256)
    if kind == "large weights":
        f[::2] = rng.integers(4097, 65536, 128)
        f[::16] = [4097, 8191, 8192, 8193, 16_384, 32_768, 65_535, 5000] * 2
    elif kind == "only large weights":  # a state grows until it gives off bytes at such a weight
        f = rng.integers(4097, 4200, 256)
    elif kind == "zero weights":
        f[::3] = 0
    elif kind == "large cumulative weights":
        c = rng.integers(0, 65_536, 256)
    elif kind == "ones and 4096":
        f[::2] = 1
        f[1::4] = 4096
    return f.astype(np.uint16), np.concatenate([c, [4096]]).astype(np.uint16)


@pytest.mark.parametrize("kind", ["any sum", "large weights", "only large weights", "zero weights", "large cumulative weights", "ones and 4096"])
@pytest.mark.parametrize("n", [1, 5, 1000, 60_001])
def test_containers_of_any_table(comp, kind, n):
    rng = np.random.default_rng(n + len(kind))
    freq, cdf = tables(kind, rng)
    x = rng.integers(0, 256, n).astype(np.uint8)
    d_in, d_out = devmem.upload(x), devmem.alloc(2 * n + 1024)
    size, _, _ = comp.VANSEncode4xGPU(d_in.ptr, d_out.ptr, n, freq, cdf, b"")
    assert devmem.download(d_out.ptr, size)[8:] == encode(x, freq, cdf), kind
