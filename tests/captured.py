"""What a call puts on its stream, from a captured graph that is not run."""
import torch


def kernels_of(call):
    """How many kernels `call()` launches on the current stream."""
    from cuda.bindings import runtime
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        call()
    raw = runtime.cudaGraph_t(graph.raw_cuda_graph())
    _, _, count = runtime.cudaGraphGetNodes(raw, 0)
    _, nodes, _ = runtime.cudaGraphGetNodes(raw, count)
    kinds = [runtime.cudaGraphNodeGetType(n)[1] for n in nodes]
    return sum(k == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)
