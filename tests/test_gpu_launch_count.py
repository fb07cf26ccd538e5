"""convgpu_launch_count counts the kernels that a call launches: the kernel nodes of the same call
captured into a graph."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _kernel_nodes(graph):
    cu = ctypes.CDLL("libcuda.so.1")
    count = ctypes.c_size_t(0)
    assert cu.cuGraphGetNodes(ctypes.c_void_p(graph), None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert cu.cuGraphGetNodes(ctypes.c_void_p(graph), nodes, ctypes.byref(count)) == 0
    kind, kernels = ctypes.c_int(), 0
    for n in nodes:
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(n), ctypes.byref(kind)) == 0
        kernels += kind.value == 0
    return kernels


@pytest.mark.parametrize("n,b", [(16, 3), (32, 1), (64, 1), (64, 4), (128, 1), (128, 5), (256, 1), (512, 1)])
@pytest.mark.parametrize("filt", ["shared", "real", "spectrum", "split"])
@pytest.mark.parametrize("xy", [0, 1, 3])
def test_kernels(gpu, n, b, filt, xy):
    if xy and gpu.plan_variant(n, 4) != 3 and n != 512:
        pytest.skip("one plan only")
    keep = {k: gpu.plan_variant(n, k) for k in (4, 7)}
    gpu.plan_variant(n, 4, xy)
    gpu.plan_variant(n, 7, 1 if n == 512 else 0)
    s = torch.zeros((b, n, n, n), dtype=torch.complex64, device="cuda")
    o = torch.empty_like(s)
    f = torch.zeros((n, n, n), dtype=torch.float32 if filt == "real" else torch.complex64, device="cuda")
    flags = {"shared": 0, "real": gpu.FILTER_REAL, "spectrum": gpu.FILTER_IS_SPECTRUM, "split": gpu.TENSOR_SPLIT}[filt]
    try:
        gpu.conv3d_device(n, s, f, o, b, flags)  # allocations
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph(keep_graph=True)
        before = gpu.launch_count()
        with torch.cuda.graph(g):
            gpu.conv3d_device(n, s, f, o, b, flags, torch.cuda.current_stream())
        counted = gpu.launch_count() - before
        assert counted == _kernel_nodes(g.raw_cuda_graph())
    finally:
        for k, v in keep.items():
            gpu.plan_variant(n, k, v)
