"""Quantiser of the FP16-in GEMM: chunks that end inside the matrices, and infinities and NaNs beyond the first K tile."""
import numpy as np
import pytest
import torch

import oracle
from bare_metal_b200 import igemm as ig
from _gpu import T, assert_clean_status, dev

pytestmark = pytest.mark.gpu


def quantise(x, axis_block, first_k, k_axis):
    """q and the factors of the reference's rule in float32: one factor per block of the other axis, from the first K tile."""
    other = 1 - k_axis
    q = np.zeros(x.shape, np.int8)
    scale = np.zeros(x.shape[other], np.float32)
    for b in range(0, x.shape[other], axis_block):
        blk = np.take(x, range(b, min(b + axis_block, x.shape[other])), other).astype(np.float32)
        m = np.float32(np.abs(np.take(blk, range(first_k), k_axis)).max())
        inv = np.float32(127.0) / m if m > 0 else np.float32(1)
        with np.errstate(invalid="ignore", over="ignore"):
            y = np.rint(blk * inv)
        part = np.where(np.isnan(y), 0, np.clip(y, -128, 127)).astype(np.int8)
        sl = slice(b, min(b + axis_block, x.shape[other]))
        if other == 0: q[sl] = part
        else: q[:, sl] = part
        scale[sl] = m / np.float32(127.0)
    return q, scale


# K of half a tile, below and above a chunk of A (256); rows and columns around the blocks and the rows of a chunk
@pytest.mark.parametrize("M,N,K,col_block", [(1, 16, 16, 128), (127, 144, 48, 128), (129, 272, 256, 256), (130, 400, 272, 128),
                                             (257, 112, 528, 256),
                                             # more CTAs than fit at once: chunks of half the size
                                             (130, 4112, 2320, 128), (2500, 272, 4112, 256)])
def test_block_quantised_product_with_outliers(M, N, K, col_block):
    rng = np.random.default_rng(M * N + K)
    A = rng.uniform(-1, 1, (M, K)).astype(np.float16)
    B = rng.uniform(-1, 1, (K, N)).astype(np.float16)
    if K > 32:                                            # beyond the tile that sets the factors: clamped, or 0 for a NaN
        A[M // 2, 40], A[0, 33], A[M - 1, K - 1] = np.inf, 300.0, np.nan
        B[K - 2, N - 1], B[35, 0], B[K - 1, N // 2] = -np.inf, np.nan, -200.0
    kt = min(K, 32)
    qa, sa = quantise(A, 128, kt, 1)
    qb, sb = quantise(B, col_block, kt, 0)
    want = (oracle.igemm(qa, qb).astype(np.float32) * (sa[:, None] * sb[None, :])).astype(np.float32)
    C = torch.full((M, N), -1.0, device=dev())
    ig.igemm_online_quant(T(A), T(B), C, M, N, K, col_block)
    assert_clean_status()
    assert np.array_equal(C.cpu().numpy().view(np.uint32), want.view(np.uint32))
