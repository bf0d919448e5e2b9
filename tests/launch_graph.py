"""The launches that a call enqueues on a stream, as a captured graph: kernel
names, what each kernel waits for, and its occupancy."""
from __future__ import annotations

from cuda.bindings import driver as D
from cuda.bindings import runtime as R


def _ok(r):
    assert int(r[0]) == 0, r[0]
    return r[1] if len(r) == 2 else r[1:]


class LaunchGraph:
    """fn(stream) captured, and not run."""

    def __init__(self, fn):
        s = _ok(R.cudaStreamCreateWithFlags(R.cudaStreamNonBlocking))
        _ok(R.cudaStreamBeginCapture(s, R.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed))
        try:
            fn(int(s))
        finally:
            self.graph = _ok(R.cudaStreamEndCapture(s))
            R.cudaStreamDestroy(s)
        g = D.CUgraph(int(self.graph))
        count = _ok(D.cuGraphGetNodes(g))[1]
        self.nodes = list(_ok(D.cuGraphGetNodes(g, count))[0])
        n = _ok(D.cuGraphGetEdges(g))[2]
        a, b = _ok(D.cuGraphGetEdges(g, n))[:2]
        self.before = {int(x): set() for x in self.nodes}
        for x, y in zip(a, b):
            self.before[int(y)].add(int(x))
        self.kernels = [x for x in self.nodes if _ok(D.cuGraphNodeGetType(x)) == D.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL]

    def _params(self, node):
        return _ok(D.cuGraphKernelNodeGetParams(node))

    def name(self, node) -> str:
        n = _ok(D.cuFuncGetName(self._params(node).func))
        return n.decode() if isinstance(n, bytes) else str(n)

    def named(self, part: str) -> list:
        return [x for x in self.kernels if part in self.name(x)]

    def waits_for(self, node) -> set[int]:
        """Every node that comes before `node`."""
        seen, todo = set(), [int(node)]
        while todo:
            for x in self.before[todo.pop()] - seen:
                seen.add(x)
                todo.append(x)
        return seen

    def blocks_per_sm(self, node) -> int:
        p = self._params(node)
        return _ok(D.cuOccupancyMaxActiveBlocksPerMultiprocessor(p.func, p.blockDimX * p.blockDimY * p.blockDimZ, p.sharedMemBytes))

    def close(self):
        R.cudaGraphDestroy(self.graph)
