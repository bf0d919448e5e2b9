"""A batch that is laid out once pins no memory for its tables; one that is laid
out again gives the same frames from the kept buffer."""
from __future__ import annotations

import numpy as np
import pytest

from przm_b200 import devmem, gpu
from przm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_creating_a_batch_pins_nothing(comp):
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.zeros(1, device="cuda")
    gpu.DeviceBatch(comp, [1000], gpu.PROFILE_ANS).close()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        for sizes, profile_ in (([1000], gpu.PROFILE_D2D), ([1 << 20] * 4 + [3], gpu.PROFILE_ANS), ([70_000] * 3, gpu.PROFILE_ANS_SHEAF)):
            gpu.DeviceBatch(comp, sizes, profile_).close()
        torch.cuda.synchronize()
    names = [e.name for e in p.events()]
    assert any("cudaMalloc" in n for n in names)
    assert not [n for n in names if "HostAlloc" in n or "MallocHost" in n]


def test_tables_of_batches_and_of_calls_laid_out_again(comp, oracle):
    xs = [W.gen("records", i, n) for i, n in enumerate((5, 40_000, 70_000, 300_000))]
    for _ in range(2):
        b = gpu.DeviceBatch(comp, [len(x) for x in xs], gpu.PROFILE_ANS)
        try:
            for x, o in zip(xs, b.in_offs):
                devmem.upload_to(b.d_in + int(o), x)
            b.enqueue(graph=False)
            for x, o, n in zip(xs, b.out_offs, b.frame_sizes()):
                assert devmem.download(b.d_out + int(o), int(n)) == oracle.compress_p1(x)
        finally:
            b.close()
        frames, sizes = comp.CompressPacked(np.concatenate(xs), [len(x) for x in xs], gpu.PROFILE_ANS)
        assert bytes(frames) == b"".join(oracle.compress_p1(x) for x in xs)
        for x in xs:
            assert comp.Compress(x, gpu.PROFILE_ANS)[0] == oracle.compress_p1(x)
