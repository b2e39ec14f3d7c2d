"""What a call launches: its kernels in order, read from a CUDA graph that the call is captured into.

A size chosen to reach a kernel falls out of a test unnoticed when the rule of a dispatch moves; with this the test says
which kernel it means.
"""
import ctypes as C
import re

import torch
from cuda.bindings import driver


class Kernel:
    """`name` without namespaces and template arguments, `ints` the whole numbers and truth values among the latter, in order."""

    def __init__(self, mangled, grid):
        m = re.search(r"\d+(qk_\w+?kernel)I", mangled) or re.search(r"\d+(qk_\w+?kernel)", mangled)
        self.name = m.group(1) if m else mangled
        self.fmt = (re.search(r"kernelIN?S?_?\d*\w*?(Dec\w+?)E", mangled) or [None, ""])[1]
        self.ints = [int(v) for v in re.findall(r"L[ib](\d+)E", mangled)]
        self.mangled, self.grid = mangled, grid

    def __repr__(self):
        return f"{self.name}<{self.fmt} {self.ints}> x {self.grid}"


def _ok(r):
    assert int(r[0]) == 0, r[0]
    return r[1:]


def _graph(call):
    call()  # what is set up once is set up
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        call()
    return g


def launched(call):
    """The kernels of one call(), which launches on torch's current stream."""
    g = _graph(call)
    h = driver.CUgraph(g.raw_cuda_graph())
    (_, n), = [_ok(driver.cuGraphGetNodes(h))]
    nodes = _ok(driver.cuGraphGetNodes(h, n))[0]
    n_edges = _ok(driver.cuGraphGetEdges_v2(h))[-1]
    before, after = _ok(driver.cuGraphGetEdges_v2(h, n_edges))[:2] if n_edges else ([], [])
    follows = {int(b): int(a) for a, b in zip(before, after)}

    def depth(k):
        d = 0
        while k in follows:
            k, d = follows[k], d + 1
        return d

    out = []
    for node in sorted(nodes, key=lambda k: depth(int(k))):
        if _ok(driver.cuGraphNodeGetType(node))[0] != driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        p = _ok(driver.cuGraphKernelNodeGetParams(node))[0]
        name = _ok(driver.cuFuncGetName(p.func))[0] if int(p.func) else _ok(driver.cuKernelGetName(p.kern))[0]
        out.append(Kernel(name.decode(), (p.gridDimX, p.gridDimY, p.gridDimZ)))
    del g
    return out


def programmatic_edges(call):
    """How many launches of call() may start before the one ahead of them has ended, and how many edges there are."""
    g = _graph(call)
    get, n = C.CDLL("libcuda.so.1").cuGraphGetEdges_v2, C.c_size_t()  # (cuda.bindings 12.9 gives edge data of freed memory)
    h = C.c_void_p(g.raw_cuda_graph())
    assert get(h, None, None, None, C.byref(n)) == 0
    before, after, data = (C.c_void_p * n.value)(), (C.c_void_p * n.value)(), (C.c_uint8 * (8 * n.value))()
    assert get(h, before, after, data, C.byref(n)) == 0
    del g
    return sum(data[8 * i + 2] == 1 for i in range(n.value)), n.value  # {from port, to port, type, 5 reserved}; 1: programmatic


def sm_count():
    return torch.cuda.get_device_properties(0).multi_processor_count
