"""The work that is timed: calls of przm_b200 as a program makes them.

Inputs are the seeded synthetic data of przm_b200.workloads (order-1 text with
copies, tables of integers, mutated records, uniform bytes, Zipf streams), so a
case, a seed and the generators give the same bytes everywhere.

A case names one entry point ("path"), its frame profile (0: flat sections,
1: entropy coded, 2: and coded distances, 3: and the literal foliations), how
many inputs one call takes ("count") and their sizes: "lo" to "hi" bytes each,
log-uniform, the same list for every seed.
"""
from __future__ import annotations

import math
import random
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from przm_b200 import gpu
from przm_b200 import workloads as W

KiB, MiB = 1 << 10, 1 << 20


def _case(name, path, **kw):
    c = {"path": path, "profile": 1, "count": 1, "lo": MiB, "hi": MiB, "data": "mixture", "graph": False}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small file or message through the one-call host API: latency only
        _case("compress_small", "compress", lo=12_345, hi=12_345, data="records"),
        # the flat frame of the reference's own GPU call (CompressD2D), an odd size
        _case("compress_flat", "compress", profile=0, lo=1_000_003, hi=1_000_003, data="table"),
        # one 4 MiB text input in one call (the one-frame workload)
        _case("compress_text_4m", "compress", lo=4 * MiB, hi=4 * MiB, data="markov"),
        # a bulk job: inputs of one size resident on the device, the pipeline
        # replayed as a graph, several batches in turn on streams of their own
        _case("batch_1m", "batch", count=64, graph=True),
        # a directory of files of all sizes through the packed host API
        _case("packed_uneven", "packed", count=256, lo=KiB, hi=4 * MiB),
        # the same bulk job with every section coded, the smallest frames
        _case("batch_sheaf", "batch", profile=3, count=48, lo=200_000, hi=700_000),
        # a bulk read: frames resident on the device decoded in one call
        _case("decode_1m", "decode", count=128),
        # one frame read through the host API
        _case("decode_one", "decompress", lo=300_001, hi=300_001),
        # frames with every section coded, read in one call
        _case("decode_sheaf", "decode", profile=3, count=32, lo=100_000, hi=400_000),
        # entropy coding alone: many device streams, histogram to container
        _case("vans_streams", "vans", count=64, data="zipf"),
        # distance coding alone: sections of 20 000 distances
        _case("offset_sections", "offsets", count=256, lo=20_000, hi=20_000, data="log"),
        # literal coding alone: the best of raw, adaptive and four foliations
        _case("literal_sections", "literals", count=64, lo=256 * KiB, hi=256 * KiB, data="markov"),
    ]


# per path: (count range, input size range, total bytes at most, data kinds, profiles)
_RANGES = {
    "compress": ((1, 1), (KiB, 4 * MiB), 4 * MiB, ("mixture", "markov", "table", "records", "uniform"), (0, 1, 2, 3)),
    "batch": ((2, 512), (4 * KiB, 2 * MiB), 48 * MiB, ("mixture", "markov", "records"), (0, 1, 1, 2, 3)),
    "packed": ((2, 512), (KiB, 4 * MiB), 64 * MiB, ("mixture",), (0, 1, 1, 2, 3)),
    "decode": ((2, 640), (4 * KiB, MiB), 48 * MiB, ("mixture", "markov", "records"), (0, 1, 1, 2, 3)),
    "decompress": ((1, 1), (KiB, MiB), MiB, ("mixture", "markov", "table", "records"), (0, 1, 2, 3)),
    "vans": ((1, 256), (KiB, MiB), 48 * MiB, ("zipf", "markov", "uniform"), (1,)),
    "offsets": ((1, 256), (64, 20_000), 5_000_000, ("log",), (1,)),
    "literals": ((1, 64), (KiB, 256 * KiB), 12 * MiB, ("markov", "mixture"), (1,)),
}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(sorted(_RANGES))
    counts, sizes, total, data, profiles = _RANGES[path]
    count = _log(rng, *counts)
    a, b = sorted((_log(rng, *sizes), _log(rng, *sizes)))
    if count == 1 or rng.random() < 0.4:
        a = b
    b = max(a if a < total // count else 1, min(b, total // count))
    a = min(a, b)
    return _case("", path, count=count, lo=a, hi=b, data=rng.choice(data), profile=rng.choice(profiles),
                 graph=path == "batch" and rng.random() < 0.5)


def _sizes(case):
    r = random.Random(case["count"] * 1_000_003 + case["lo"] * 31 + case["hi"])
    return [_log(r, case["lo"], case["hi"]) for _ in range(case["count"])]


def _inputs(case, seed):
    def one(a):
        i, n = a
        s = W.SEED + 1_000_003 * (seed + 1) + 7919 * i
        k = case["data"]
        if k == "mixture":
            return W.mixture(s, n)[0]
        if k == "zipf":
            return W.zipf(s, n)
        if k == "log":  # distances, log-uniform up to the 1 MiB window
            return np.exp(np.random.default_rng(s).uniform(0, math.log(MiB - 1), n)).astype(np.uint32)
        return W.gen(k, s, n)

    W.gen("records", 1, 16)  # the generator library is loaded before the threads use it
    with ThreadPoolExecutor(8) as ex:
        return list(ex.map(one, enumerate(_sizes(case))))


def _offsets(sizes, align=64):
    """Start of every region and the end of the last, regions `align` bytes apart at least."""
    o = np.zeros(len(sizes) + 1, np.uint64)
    o[1:] = np.cumsum([(int(s) + align - 1) // align * align for s in sizes])
    return o[:-1], int(o[-1])


def _to_device(parts):
    """The arrays back to back, each from a 64-byte boundary, and where each starts."""
    offs, total = _offsets([p.nbytes for p in parts])
    host = np.zeros(total + 64, np.uint8)
    for o, p in zip(offs, parts):
        host[int(o):int(o) + p.nbytes] = p.view(np.uint8)
    return torch.from_numpy(host).cuda(), offs


class _Batch:
    """A resident batch and its stream, freed with the last tensor of its memory."""

    def __init__(self, comp, parts, profile):
        self.b = gpu.DeviceBatch(comp, [len(p) for p in parts], profile)
        self.stream = torch.cuda.Stream()
        self.frame_bytes = int(self.b.out_offs[-1]) + gpu.FrameBound(len(parts[-1]))
        host = torch.from_numpy(np.concatenate(parts)).pin_memory()
        self.b.upload(host.numpy())
        torch.cuda.synchronize()

    def __del__(self):
        try:
            torch.cuda.synchronize()
            self.b.close()
        except Exception:
            pass


class _View:
    """A batch's frames as a tensor's source: the tensor keeps it, and it the batch."""

    def __init__(self, batch):
        self.batch = batch
        self.__cuda_array_interface__ = {"data": (batch.b.d_out, False), "shape": (batch.frame_bytes,),
                                         "typestr": "|u1", "version": 3}


def prepare(case, seed):
    comp = gpu.GetGlobalCompressor()
    path, profile = case["path"], case["profile"]
    parts = _inputs(case, seed)
    s = {"path": path, "profile": profile, "comp": comp, "graph": case["graph"]}
    if path == "compress":
        s["src"] = parts[0]
        s["dst"] = np.zeros(gpu.FrameBound(len(parts[0])), np.uint8)
    elif path == "batch":
        s["batch"] = _Batch(comp, parts, profile)
        s["frames"] = torch.as_tensor(_View(s["batch"]), device="cuda")
        s["frames"].zero_()
    elif path == "packed":
        s["sizes"] = [len(p) for p in parts]
        s["src"] = torch.from_numpy(np.concatenate(parts)).pin_memory()
        s["dst"] = torch.zeros(sum(gpu.FrameBound(n) for n in s["sizes"]) + 64, dtype=torch.uint8).pin_memory()
    elif path == "decompress":
        s["frame"] = np.frombuffer(comp.Compress(parts[0], profile)[0], np.uint8)
    elif path == "decode":
        packed, lens = comp.CompressPacked(np.concatenate(parts), [len(p) for p in parts], profile)
        cuts = np.concatenate([[0], np.cumsum(lens, dtype=np.int64)])
        s["src"], s["src_offs"] = _to_device([packed[cuts[i]:cuts[i + 1]] for i in range(len(lens))])
        s["src_lens"] = lens.copy()
        s["dst_offs"], total = _offsets([len(p) for p in parts])
        s["caps"] = [len(p) for p in parts]
        s["dst"] = torch.zeros(total + 64, dtype=torch.uint8, device="cuda")
    else:
        s["src"], s["src_offs"] = _to_device(parts)
        s["lens"] = [len(p) for p in parts]
        wide = 5 if path == "offsets" else 2
        s["caps"] = [wide * n + 1024 for n in s["lens"]]
        s["dst_offs"], total = _offsets(s["caps"])
        s["dst"] = torch.zeros(total + 64, dtype=torch.uint8, device="cuda")
        s["src_offs"] = s["src_offs"] // 4 if path == "offsets" else s["src_offs"]
    return s


def run(s):
    comp, path = s["comp"], s["path"]
    if path == "compress":
        frame, _ = comp.CompressD2D(s["src"]) if s["profile"] == gpu.PROFILE_D2D else comp.Compress(s["src"], s["profile"])
        s["dst"][:len(frame)] = np.frombuffer(frame, np.uint8)  # where the program collects its frames
        return {"frames": s["dst"], "sizes": len(frame)}
    if path == "batch":
        b = s["batch"]
        b.b.enqueue(b.stream.cuda_stream, graph=s["graph"])
        return s["frames"]
    if path == "packed":
        frames, sizes = comp.CompressPacked(s["src"].numpy(), s["sizes"], s["profile"], s["dst"].numpy())
        return {"frames": s["dst"], "total": len(frames), "sizes": sizes.astype(np.int64)}
    if path == "decompress":
        return np.frombuffer(comp.Decompress(s["frame"]), np.uint8)
    d_src, d_dst = s["src"].data_ptr(), s["dst"].data_ptr()
    if path == "decode":
        status, sizes = comp.DecompressBatchDevice(d_src, s["src_offs"], s["src_lens"], d_dst, s["dst_offs"], s["caps"])
        return {"bytes": s["dst"], "status": status, "sizes": sizes.astype(np.int64)}
    if path == "vans":
        sizes = comp.VANSEncodeBatch(d_src, s["src_offs"], s["lens"], gpu.NORM_CPU, d_dst, s["dst_offs"])
        return {"bytes": s["dst"], "sizes": sizes.astype(np.int64)}
    if path == "offsets":
        sizes = comp.PackageOffsetsBatch(d_src, s["src_offs"], s["lens"], d_dst, s["dst_offs"], s["caps"])
        return {"bytes": s["dst"], "sizes": sizes.astype(np.int64)}
    sizes, nibbles = comp.PackageLiteralsBatch(d_src, s["src_offs"], s["lens"], d_dst, s["dst_offs"], s["caps"])
    return {"bytes": s["dst"], "sizes": sizes.astype(np.int64), "nibbles": nibbles}


# bytes out per byte in of these data: frames and containers
_RATIO = {"mixture": 0.62, "markov": 0.68, "table": 0.84, "records": 0.25, "uniform": 1.0, "zipf": 0.75}


def work(case):
    n = sum(_sizes(case))
    if case["data"] == "log":  # four bytes a distance in, about 1.7 out
        return {"bytes": 4 * n + 1.7 * n, "flops": 0}
    return {"bytes": n + _RATIO[case["data"]] * n, "flops": 0}


def exact(case, seed):
    return None  # every output is bytes or whole numbers, equal or not
