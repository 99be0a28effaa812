"""Which kernel a launcher picks where another one was measured to be slower: read from a captured graph that never runs."""
import pytest
import torch
from cuda.bindings import driver

from bare_metal_b200 import igemm as ig
from _gpu import dev

pytestmark = pytest.mark.gpu


def ok(result):
    assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
    return result[1]


def captured_kernels(call):
    """Mangled names of the kernels that `call` launches."""
    call()                                             # scratch and kernel attributes are set up outside of a capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    err, _, count = driver.cuGraphGetNodes(raw, 0)
    assert err == driver.CUresult.CUDA_SUCCESS
    names = []
    for node in driver.cuGraphGetNodes(raw, count)[1]:
        if ok(driver.cuGraphNodeGetType(node)) == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            params = ok(driver.cuGraphKernelNodeGetParams(node))
            name = driver.cuKernelGetName(params.kern) if int(params.kern) else driver.cuFuncGetName(params.func)
            names.append(ok(name).decode())
    return names


# rows that four 16-byte pieces a thread of 512 threads do not hold: still 512 threads, three rows of them on an SM (1024
# threads with two pieces each need 50 registers and leave one)
@pytest.mark.parametrize("M,K,pieces", [(200, 16400, 4), (149, 32768, 4), (200, 16384, 4), (148, 16400, 2), (16, 8192, 1)])
def test_pieces_a_thread_of_the_quantiser(M, K, pieces):
    x = torch.zeros((M, K), dtype=torch.float16, device=dev())
    names = captured_kernels(lambda: ig.quantize_rows(x, M, K))
    assert len(names) == 1 and f"quantize_rows_f16_kernelILi{pieces}E" in names[0]
