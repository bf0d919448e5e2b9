"""Models of histograms whose symbols lie in one to eight groups of 32, with
many equal counts: the containers are the oracle's, and small alphabets cost
the normaliser less than large ones."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import devmem, gpu
from przm_b200 import workloads as W

from .gpu_profile import kernels, total
from .test_gpu_segments import encode

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [(0,), (7,), (0, 7), (1, 2, 3), (0, 2, 5, 7), (1, 3, 4, 6), (0, 1, 3, 6, 7), (0, 1, 2, 4, 5, 6), tuple(range(8))])
def test_models_by_groups_of_symbols(comp, oracle, groups):
    rng = np.random.default_rng(sum(1 << g for g in groups))
    parts = []
    for per in (1, 2, 5, 32):  # symbols of a group
        sym = np.concatenate([32 * g + rng.choice(32, per, replace=False) for g in groups]).astype(np.uint8)
        for n in (64, 65, 101, 4096, 4099, 30_000):
            parts.append(rng.choice(sym, n))                                   # near-equal counts
            parts.append(np.resize(sym, n))                                    # equal ones
            p = 0.6 ** np.arange(len(sym))
            parts.append(rng.choice(sym, n, p=p / p.sum()).astype(np.uint8))   # falling ones
    for p, g in zip(parts, encode(comp, parts)):
        assert g == oracle.adaptive_vans(p), (groups, len(p))


def test_small_alphabets_cost_less(comp):
    # 2000 streams of text (three groups) beside as many of all 256 symbols
    n, count = 300, 2000

    def norm_us(kind):
        host = np.concatenate([np.pad(W.gen(kind, 5 + i % 40, n), (0, 84)) for i in range(count)])
        d_in, d_out = devmem.upload(host), devmem.alloc(count * 2048)
        io, oo = np.arange(count, dtype=np.uint64) * 384, np.arange(count, dtype=np.uint64) * 2048
        return total(kernels(lambda: comp.VANSEncodeBatch(d_in.ptr, io, [n] * count, gpu.NORM_CPU, d_out.ptr, oo)), "k_stream_norm")

    assert norm_us("markov") < 0.75 * norm_us("uniform")
