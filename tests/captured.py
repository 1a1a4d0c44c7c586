"""What a call launches, read from a capture of it."""
import pytest


def launches(call, between=lambda: None):
    """The CTAs per cluster of each kernel that call() launches, the second time on a stream of its own; the captured launches have run once."""
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
    out = []
    for node in nodes:
        if int(node) and rt.cudaGraphNodeGetType(node)[1] == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel:
            err, value = rt.cudaGraphKernelNodeGetAttribute(node, rt.cudaLaunchAttributeID.cudaLaunchAttributeClusterDimension)
            assert int(err) == 0
            out.append(max(1, value.clusterDim.x))
    graph.replay()
    torch.cuda.synchronize()
    return out


@pytest.fixture
def scratch_given_back(gpu):
    """For tests that capture mat-muls: the graphs hold the scratch of their streams, of which a device has sixteen, until it is released."""
    import torch
    yield
    torch.cuda.synchronize()
    assert gpu.gemm_release() == 0
