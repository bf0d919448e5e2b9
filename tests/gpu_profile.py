"""Kernels that a call launches and the time each takes on the device."""
from __future__ import annotations


def kernels(fn, warm: int = 2) -> list[tuple[str, float]]:
    """(name without arguments and namespace, microseconds) of every kernel of one call of fn, in order."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    for _ in range(warm):
        fn()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    out = []
    for e in sorted(p.events(), key=lambda e: e.time_range.start):
        name = e.name.split("(")[0].replace("void ", "").replace("pz::", "")
        if name.startswith("k_"):
            out.append((name, e.time_range.elapsed_us()))
    return out


def total(ks: list[tuple[str, float]], *prefixes: str) -> float:
    return sum(t for n, t in ks if n.startswith(prefixes))
