"""Every kernel that a clustering call launches is counted, and nothing else: the counter against the kernel nodes of the
captured call."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _counted_and_launched(call):
    from reskv_b200 import _extension as ext

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        before = ext.launch_count
        call()
        counted = ext.launch_count - before
    cudart, raw = ctypes.CDLL("libcudart.so.12"), ctypes.c_void_p(graph.raw_cuda_graph())
    count = ctypes.c_size_t()
    assert cudart.cudaGraphGetNodes(raw, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert cudart.cudaGraphGetNodes(raw, nodes, ctypes.byref(count)) == 0
    kernels = 0
    for node in nodes:
        kind = ctypes.c_int(-1)
        assert cudart.cudaGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        kernels += kind.value == 0  # cudaGraphNodeTypeKernel
    return counted, kernels


@pytest.mark.parametrize("iterations", [1, 3])
@pytest.mark.parametrize("form", ["pair", "default", "exact", "warp_mma", "many centres", "misaligned"])
def test_clustering(form, iterations):
    from reskv_b200._extension import load_extension
    from reskv_b200.synthetic import mixture

    ops = load_extension("compression")
    k, v = (mixture(1, 2, 300, seed=i, device=DEV) for i in range(2))
    if form == "misaligned":
        buf = torch.zeros(k.numel() + 1, dtype=k.dtype, device=DEV)
        buf[1:] = k.flatten()
        k = buf[1:].view(k.shape)
    calls = {"pair": lambda: ops.kmeans_pair(k, v, 16, iterations),
             "many centres": lambda: ops.kmeans(k, 40, iterations, False),
             "misaligned": lambda: ops.kmeans(k, 16, iterations, False)}
    options = {form: True} if form in ("exact", "warp_mma") else {}
    counted, launched = _counted_and_launched(calls.get(form) or (lambda: ops.kmeans(k, 16, iterations, False, **options)))
    assert counted == launched
