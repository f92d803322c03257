"""What a trace puts on the stream, read from a capture: one kernel, behind
one clear of its work counter where it has one."""
import ctypes as C

import pytest
import torch

from kiraray_gb300 import scenes
from kiraray_gb300.accel import Accel
from tests import helpers as H
from tests.test_oracle import _instanced_scene

pytestmark = pytest.mark.gpu

KERNEL, MEMSET = 0, 2   # cudaGraphNodeType


def _nodes(fn):
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.stream(s):
        fn()
        s.synchronize()
        graph.capture_begin(capture_error_mode="thread_local")
        try:
            fn()
        finally:
            graph.capture_end()
    rt = C.CDLL("libcudart.so.13")
    raw = C.c_void_p(graph.raw_cuda_graph())
    n = C.c_size_t()
    assert rt.cudaGraphGetNodes(raw, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert rt.cudaGraphGetNodes(raw, nodes, C.byref(n)) == 0
    kinds = []
    for node in nodes:
        kind = C.c_int()
        assert rt.cudaGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        kinds.append(kind.value)
    return sorted(kinds)


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("n", [100, 400000])
def test_two_levels(krr_lib, cuda, n, any_hit):
    geos, insts = _instanced_scene(seed=5, n_inst=30)
    acc = Accel.instanced(geos, insts)
    rays = torch.from_numpy(H.random_rays(n, 3, box=5.0)).cuda()
    trace = acc.trace_any if any_hit else acc.trace_closest
    out = trace(rays)
    assert _nodes(lambda: trace(rays, out)) == [KERNEL, MEMSET]


@pytest.mark.parametrize("n,kinds", [(100, [KERNEL]), (400000, [KERNEL, MEMSET])])
def test_one_level(krr_lib, cuda, n, kinds):
    acc = Accel(scenes.cornell_box(16, 16).world_triangles())
    rays = torch.from_numpy(H.random_rays(n, 3)).cuda()
    out = acc.trace_closest(rays)
    assert _nodes(lambda: acc.trace_closest(rays, out)) == kinds
