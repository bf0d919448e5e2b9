"""Kernels that a call launches and the time each takes on the device."""
from __future__ import annotations


def kernels(fn, warm: int = 2) -> list[tuple[str, float]]:
    """(name without arguments and namespace, microseconds) of every kernel of one call of fn, in order."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    for _ in range(warm):
        fn()
    mark = torch.zeros(1024, device="cuda")
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        fn()  # (a trace may begin without its first kernels: this call's are not looked at)
        torch.cuda.synchronize()
        mark.add_(1.0)
        torch.cuda.synchronize()
        fn()
        torch.cuda.synchronize()
    out, marked = [], False
    for e in sorted(p.events(), key=lambda e: e.time_range.start):
        name = e.name.split("(")[0].replace("void ", "").replace("pz::", "")
        if "at::native" in e.name:
            out, marked = [], True
        elif name.startswith("k_"):
            out.append((name, e.time_range.elapsed_us()))
    assert marked and out
    return out


def total(ks: list[tuple[str, float]], *prefixes: str) -> float:
    return sum(t for n, t in ks if n.startswith(prefixes))
