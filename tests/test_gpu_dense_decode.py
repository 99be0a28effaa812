"""Few-token dense GEMM (output channels on the accumulator lanes, K folded for short tiles) against the CPU oracle."""
import numpy as np
import pytest
import torch

import oracle
from bare_metal_b200 import igemm as ig
from _gpu import T, assert_clean_status, dev, options, ulp_diff_f16

pytestmark = pytest.mark.gpu

# one channel group, ragged groups, one tile per SM, a second wave; one K block, ragged K, K stages that end in chunks
# that do not exist; token counts at the 16- and 32-column borders up to the largest
SHAPES = [(1, 8, 16), (1, 9, 128), (16, 1184, 144), (17, 2368, 1024), (31, 1192, 2064), (33, 4096, 528), (48, 300, 4112),
          (64, 4104, 1024), (65, 640, 256), (100, 12296, 272), (127, 1000, 1152), (128, 4096, 640), (129, 96, 2048),
          (255, 2376, 400), (256, 19000, 160),
          # the ragged K block after folded ones: one, a part of a group, whole groups
          (5, 64, 144), (16, 600, 432), (16, 1024, 1040), (64, 2048, 2064), (3, 1184, 1136)]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_integers_are_exact_and_nothing_is_written_outside(M, N, K):
    X = oracle.gen_int8((M, K), 5, 1)
    W = oracle.gen_int8((N, K), 5, 2)
    buf = torch.full((M + 2, N + 3), 0x5A5A5A5A, dtype=torch.int32, device=dev())
    C = buf[1:M + 1, 1:N + 1]
    with options(dense_decode=1):
        ig.igemm_i32(T(X), T(W), C, M, N, K, ig.BM_B_NK)
        assert_clean_status()
    got = buf.cpu().numpy()
    assert np.array_equal(got[1:M + 1, 1:N + 1], oracle.igemm_nt(X, W))
    got[1:M + 1, 1:N + 1] = 0x5A5A5A5A
    assert (got == 0x5A5A5A5A).all(), "store outside the output"


@pytest.mark.parametrize("M,N,K", [(1, 4096, 1024), (20, 2400, 1040), (64, 520, 4096), (200, 1192, 272)])
def test_every_epilogue_gives_the_bits_of_the_wide_tiles(M, N, K):
    X, W = T(oracle.gen_int8((M, K), 6, 1)), T(oracle.gen_int8((N, K), 6, 2))
    sa, sw = T(oracle.gen_scales(M, 6, 3)), T(oracle.gen_scales(N, 6, 4))
    zp = torch.arange(N, dtype=torch.int32, device=dev()) % 17 - 8
    got = []
    for decode in (1, 0):
        with options(dense_decode=decode):
            f32, ch = (torch.zeros((M, N), dtype=torch.float32, device=dev()) for _ in range(2))
            f16 = torch.zeros((M, N), dtype=torch.float16, device=dev())
            ig.igemm_wmma(X, W, f32, M, N, K, 0.011, 0.007, ig.BM_B_NK)
            ig.igemm_pipelined_cpasync_perchannel(X, W, ch, M, N, K, sw, zp, ig.BM_B_NK)
            ig.w8a8_linear(X, W, f16, sa, sw, M, N, K)
            assert_clean_status()
            got.append((f32, ch, f16))
    assert all(torch.equal(a, b) for a, b in zip(*got))
    want = oracle.dequant_w8a8_f16(oracle.igemm_nt(X.cpu().numpy(), W.cpu().numpy()), sa.cpu().numpy(), sw.cpu().numpy())
    assert ulp_diff_f16(got[0][2].cpu().numpy().view(np.uint16), want.view(np.uint16)) <= 1
