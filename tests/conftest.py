import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu on a B200)")


class CapturedLaunch:
    """A kernel of a captured CUDA graph: its grid, the CTAs of a cluster, its static shared memory, and its arguments by position."""

    def __init__(self, node):
        driver = pytest.importorskip("cuda.bindings.driver")
        err, self._p = driver.cuGraphKernelNodeGetParams(node)
        assert err == driver.CUresult.CUDA_SUCCESS
        self.grid = (self._p.gridDimX, self._p.gridDimY, self._p.gridDimZ)
        err, value = driver.cuGraphKernelNodeGetAttribute(node, driver.CUlaunchAttributeID.CU_LAUNCH_ATTRIBUTE_CLUSTER_DIMENSION)
        assert err == driver.CUresult.CUDA_SUCCESS
        self.cluster = max(1, value.clusterDim.x)
        err, self.static_shared = driver.cuFuncGetAttribute(driver.CUfunction_attribute.CU_FUNC_ATTRIBUTE_SHARED_SIZE_BYTES, self._p.func)
        assert err == driver.CUresult.CUDA_SUCCESS

    def argument(self, i, ctype):
        import ctypes
        at = ctypes.cast(int(self._p.kernelParams), ctypes.POINTER(ctypes.c_void_p))[i]
        return ctypes.cast(at, ctypes.POINTER(ctype))[0]


def launches_of(graph):
    """The kernels of a torch.cuda.CUDAGraph(keep_graph=True) in the order of their capture. Valid as long as the graph."""
    driver = pytest.importorskip("cuda.bindings.driver")
    raw = driver.CUgraph(graph.raw_cuda_graph())
    err, _, n = driver.cuGraphGetNodes(raw, 0)
    assert err == driver.CUresult.CUDA_SUCCESS
    err, nodes, n = driver.cuGraphGetNodes(raw, n)
    assert err == driver.CUresult.CUDA_SUCCESS
    kernel = driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL
    return [CapturedLaunch(node) for node in nodes[:n] if driver.cuGraphNodeGetType(node)[1] == kernel]


@pytest.fixture
def launches_in():
    return launches_of


@pytest.fixture
def captured():
    """captured(call): the kernels that call() launches, seen by capturing it: which form of a kernel a size is given."""
    import torch
    kept = []

    def capture(call):
        call()  # first-use work stays outside
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g, stream=torch.cuda.Stream()):
            call()
        kept.append(g)
        return launches_of(g)

    return capture


@pytest.fixture(scope="session")
def golden():
    """Byte fixtures produced by the reference's own code (see tests/golden/make_golden.py)."""
    with np.load(os.path.join(ROOT, "tests", "golden", "ggml_path_golden.npz")) as z:
        return {k: z[k] for k in z.files}


@pytest.fixture(scope="session")
def port():
    from oracle import oracle as O
    return O.port()


@pytest.fixture(scope="session")
def ref():
    from oracle import oracle as O
    if not O.ref_available():
        pytest.skip("oracle/_ref not built (needs a reference checkout at build time)")
    return O.ref()
