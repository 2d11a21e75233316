"""The kernels of a captured launch sequence, read from its CUDA graph: which
ones they are and what they were compiled to."""
from collections import namedtuple

import torch
from cuda.bindings import driver

Kernel = namedtuple('Kernel', 'name grid threads registers local_bytes')


def _value(result):
    assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
    return result[1]


def captured_kernels(launch):
    """The kernels that ``launch(stream)`` puts on a stream (called once
    before, so that nothing is built or loaded while it is captured)."""
    launch(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        launch(torch.cuda.current_stream().cuda_stream)
    handle = driver.CUgraph(init_value=graph.raw_cuda_graph())
    count = driver.cuGraphGetNodes(handle, 0)
    assert count[0] == driver.CUresult.CUDA_SUCCESS
    nodes = driver.cuGraphGetNodes(handle, count[2])
    assert nodes[0] == driver.CUresult.CUDA_SUCCESS
    attribute = driver.CUfunction_attribute
    out = []
    for node in nodes[1][:nodes[2]]:
        if _value(driver.cuGraphNodeGetType(node)) != driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        params = _value(driver.cuGraphKernelNodeGetParams(node))
        func = params.func if int(params.func) else _value(driver.cuKernelGetFunction(params.kern))
        out.append(Kernel(_value(driver.cuFuncGetName(func)).decode(), params.gridDimX, params.blockDimX,
                          _value(driver.cuFuncGetAttribute(attribute.CU_FUNC_ATTRIBUTE_NUM_REGS, func)),
                          _value(driver.cuFuncGetAttribute(attribute.CU_FUNC_ATTRIBUTE_LOCAL_SIZE_BYTES, func))))
    return out
