"""What a call launches, read from a capture of it."""
import ctypes

import pytest


def capture(call, between=lambda: None):
    """The graph of call(), the second time on a stream of its own, its kernels, and the stream."""
    import torch
    from cuda.bindings import runtime as rt
    st, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.stream(st):
        assert call() == 0                   # scratch for this stream
        st.synchronize()
        between()
        with torch.cuda.graph(graph, stream=st):
            assert call() == 0
    nodes = rt.cudaGraphGetNodes(rt.cudaGraph_t(init_value=graph.raw_cuda_graph()), 16)[1]
    return graph, [n for n in nodes if int(n) and rt.cudaGraphNodeGetType(n)[1] == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel], st


def launches(call, between=lambda: None):
    """The CTAs per cluster of each kernel that call() launches; the captured launches have run once."""
    import torch
    from cuda.bindings import runtime as rt
    graph, kernels, _ = capture(call, between)
    out = []
    for node in kernels:
        err, value = rt.cudaGraphKernelNodeGetAttribute(node, rt.cudaLaunchAttributeID.cudaLaunchAttributeClusterDimension)
        assert int(err) == 0
        out.append(max(1, value.clusterDim.x))
    graph.replay()
    torch.cuda.synchronize()
    return out


def pointer_argument(node, index):
    """(By the driver's call: the runtime that asks is not the one that launched.)"""
    from cuda.bindings import driver
    err, params = driver.cuGraphKernelNodeGetParams(driver.CUgraphNode(init_value=int(node)))
    assert int(err) == 0, err
    return ctypes.c_void_p.from_address((ctypes.c_void_p * (index + 1)).from_address(int(params.kernelParams))[index]).value


@pytest.fixture
def scratch_given_back(gpu):
    """For tests that capture mat-muls: the graphs hold the scratch of their streams, of which a device has sixteen, until it is released."""
    import torch
    yield
    torch.cuda.synchronize()
    assert gpu.gemm_release() == 0
