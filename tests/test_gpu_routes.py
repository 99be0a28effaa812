"""Which kernel a launcher picks where another one was measured to be slower: read from a captured graph that never runs."""
import pytest
import torch

from bare_metal_b200 import igemm as ig
from _gpu import dev

pytestmark = pytest.mark.gpu
driver = pytest.importorskip("cuda.bindings.driver")


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


# three waves of lone CTAs against two of pairs; the same with a pitch and with a base that TMA cannot store; a K long
# enough for pairs all the same; fourteen waves of pairs; one wave either way
@pytest.mark.parametrize("M,N,K,pad,shift,pairs", [(3200, 1808, 224, 0, 0, True), (3200, 1808, 224, 1, 0, False),
                                                   (3200, 1808, 224, 0, 1, False), (560, 7792, 6880, 1, 0, True),
                                                   (8192, 8192, 32, 1, 0, True), (1600, 1200, 256, 0, 0, False)])
def test_sparse_operand_on_the_left_with_outputs_that_tma_cannot_store(M, N, K, pad, shift, pairs):
    def zeros(*shape, dtype, value=0):
        return torch.full(shape, value, dtype=dtype, device=dev())
    out = zeros(shift + M * (N + pad), dtype=torch.int32)[shift:].view(M, N + pad)[:, :N]
    comp, B, meta = zeros(M, K // 2, dtype=torch.int8), zeros(K, N, dtype=torch.int8), zeros(M, K // 8, dtype=torch.uint8, value=0x44)
    tiled = ig.sp_pack_meta(meta, ig.BM_META_ROWS, M, K)
    names = captured_kernels(lambda: ig.igemm_sparse_i32(comp, tiled, ig.BM_META_TILED, B, out, M, N, K, ig.BM_B_KN))
    assert len(names) == 1 and ("igemm_sparse_pair_kernel" in names[0]) == pairs
    if K < 4096:                                       # half the K: the same bytes of an fp16 operand
        half, dense = zeros(M, K // 4, dtype=torch.float16), zeros(K // 2, N, dtype=torch.float16)
        f16_meta = ig.sp_pack_meta(zeros((M // 16) * (K // 32) * 8, dtype=torch.int32, value=0x44444444), ig.BM_META_REF_F16, M, K // 2)
        c = out.view(torch.float32)
        names = captured_kernels(lambda: ig.hgemm_sparse_tiled(half, dense, c, f16_meta, M, N, K // 2, ig.BM_META_TILED))
        assert len(names) == 1 and ("igemm_sparse_pair_kernel" in names[0]) == pairs


# 16 tokens and few channels or a short K: the wide tiles; from 17 tokens on weights whose rows are off the 128-byte lines: wide
# tiles where all SMs pull both operands
@pytest.mark.parametrize("M,N,K,lanes", [(16, 1024, 64, False), (1, 512, 256, False), (8, 2048, 768, False), (16, 1024, 272, False),
                                         (16, 4096, 512, True), (1, 16384, 768, True), (16, 64, 1024, True), (16, 1024, 1040, True),
                                         (1, 22016, 272, True), (16, 8192, 256, False),
                                         (32, 1024, 1040, False), (64, 2048, 2064, False), (96, 1024, 4112, False),
                                         (128, 22016, 4112, False), (17, 64, 4112, True), (32, 4096, 4112, True)])
def test_few_tokens(M, N, K, lanes):
    x, w = torch.zeros((M, K), dtype=torch.int8, device=dev()), torch.zeros((N, K), dtype=torch.int8, device=dev())
    c = torch.zeros((M, N), dtype=torch.int32, device=dev())
    names = captured_kernels(lambda: ig.igemm_i32(x, w, c, M, N, K, ig.BM_B_NK))
    assert len(names) == 1 and ("igemm_dense_decode_kernel" in names[0]) == lanes


# 296 CTAs of 512 threads are in flight at once on 148 SMs; more run as CTAs of 256
@pytest.mark.parametrize("M,N,K,threads", [(256, 256, 256, 512), (4096, 16, 2048, 512), (4096, 4096, 1024, 512),
                                           (4096, 4096, 2048, 256), (8192, 512, 4096, 256)])
def test_threads_of_the_quantiser_of_fp16_operands(M, N, K, threads):
    a, b = torch.zeros((M, K), dtype=torch.float16, device=dev()), torch.zeros((K, N), dtype=torch.float16, device=dev())
    c = torch.zeros((M, N), dtype=torch.float32, device=dev())
    names = captured_kernels(lambda: ig.igemm_online_quant(a, b, c, M, N, K))
    assert len(names) == 2 and any(f"oq_quantize_kernelILi{threads}E" in n for n in names)
