"""Sparse operand on the left on CTA pairs: several tiles per pair, so that the two accumulators, which share 32
columns of tensor memory, are refilled while their neighbour is being drained."""
import numpy as np
import pytest
import torch

import oracle
from bare_metal_b200 import igemm as ig
from _gpu import T, assert_clean_status, dev, forced_bn, options

pytestmark = pytest.mark.gpu


def sparse_left(M, K, seed):
    W = oracle.gen_int8((M, K), seed, 1)
    comp, nib = ig.prune_2_4(T(W), M, K)
    return comp, nib, oracle.decompress_rows(comp.cpu().numpy(), nib.cpu().numpy())


# K of one stage and less (the drain is then longer than the MMAs), of several ring turns; columns that end inside the
# first chunk, the middle and the last chunk of a tile; rows that end inside a CTA's half
@pytest.mark.parametrize("M,N,K", [(2304, 6160, 64), (2064, 6384, 256), (1040, 12288, 288), (2560, 4080, 1056), (1040, 6160, 320)])
@pytest.mark.parametrize("tma_store", [1, 0])
def test_integers_are_exact_over_several_tiles_per_pair(M, N, K, tma_store):
    comp, nib, dense = sparse_left(M, K, 4)
    B = oracle.gen_int8((K, N), 4, 2)
    tiled = ig.sp_pack_meta(nib, ig.BM_META_ROWS, M, K)
    buf = torch.full((M + 2, N + 16), 0x5A5A5A5A, dtype=torch.int32, device=dev())
    with options(force_bn=224, tma_store=tma_store):
        ig.igemm_sparse_i32(comp, tiled, ig.BM_META_TILED, T(B), buf[1:M + 1, :N], M, N, K, ig.BM_B_KN)
        assert_clean_status()
    got = buf.cpu().numpy()
    assert np.array_equal(got[1:M + 1, :N], oracle.igemm(dense, B, threads=0))
    got[1:M + 1, :N] = 0x5A5A5A5A
    assert (got == 0x5A5A5A5A).all(), "store outside the output"


@pytest.mark.parametrize("M,N,K", [(2304, 6160, 32), (2064, 6384, 144)])
def test_fp16_sums_of_small_integers_are_exact_over_several_tiles_per_pair(M, N, K):
    """Integers up to 15 make every product and partial sum exact in fp32: any order gives the same bits."""
    g = torch.Generator(device=dev()).manual_seed(3)
    comp = torch.randint(-15, 16, (M, K // 2), device=dev(), generator=g).half()
    B = torch.randint(-15, 16, (K, N), device=dev(), generator=g).half()
    words = torch.full(((M // 16) * (K // 16) * 8,), 0x9CE4 | (0x9CE4 << 16), dtype=torch.int64, device=dev())
    words = torch.where(words >= 2 ** 31, words - 2 ** 32, words).to(torch.int32)
    out = []
    for bn in (224, 128):
        C = torch.full((M, N), -1.0, device=dev())
        with forced_bn(bn):
            ig.hgemm_sparse_tiled(comp, B, C, words, M, N, K)
        assert_clean_status()
        out.append(C)
    # nibbles of a word, lowest first: 0x4 (positions 0, 1), 0xE (2, 3), 0xC (0, 3), 0x9 (1, 2)
    pos = torch.tensor([(0, 1), (2, 3), (0, 3), (1, 2)], device=dev()).repeat(K // 16, 1)
    cols = (torch.arange(K // 4, device=dev())[:, None] * 4 + pos).reshape(-1)
    want = comp.double() @ B.double()[cols]
    assert torch.equal(out[0].double(), want) and torch.equal(out[1], out[0])


# the borders of a 256 x 256 tile and of a CTA's 128 columns and rows, and one 16-column step to either side
@pytest.mark.parametrize("M,N", [(256, 256), (240, 240), (272, 272), (512, 128), (144, 512), (400, 496), (1024, 2304)])
def test_tile_borders(M, N):
    K = 544
    comp, nib, dense = sparse_left(M, K, 9)
    B = oracle.gen_int8((K, N), 9, 2)
    tiled = ig.sp_pack_meta(nib, ig.BM_META_ROWS, M, K)
    C = torch.full((M, N), -1, dtype=torch.int32, device=dev())
    with options(force_bn=224):
        ig.igemm_sparse_i32(comp, tiled, ig.BM_META_TILED, T(B), C, M, N, K, ig.BM_B_KN)
        assert_clean_status()
    assert np.array_equal(C.cpu().numpy(), oracle.igemm(dense, B, threads=0))


# the launcher's own choice behind the reference ABI: 225 pair tiles on 74 pairs (four ring stages, stores in boxes of 16
# columns), 108 (three stages, boxes of 32), few enough for lone CTAs
@pytest.mark.parametrize("M,N,K", [(2064, 6384, 64), (2064, 6384, 320), (2304, 2832, 96), (1040, 1040, 96)])
def test_scaled_fp32_results_where_the_launcher_chooses(M, N, K):
    dense = oracle.gen_sparse_2_4_ref(M, K, 5)
    comp, meta = oracle.compress_2_4_ref(dense)
    B = oracle.gen_int8((K, N), 5, 2)
    buf = torch.full((M + 2, N), -1.0, device=dev())
    ig.igemm_sparse_tiled(T(comp), T(B), buf[1:M + 1], T(meta.view(np.int32)), M, N, K, 0.011, 0.007)
    assert_clean_status()
    got = buf.cpu().numpy()
    assert (got[0] == -1).all() and (got[-1] == -1).all(), "store outside the output"
    want = oracle.dequant_per_tensor(oracle.igemm(dense, B, threads=0), np.float32(0.011), np.float32(0.007))
    assert np.array_equal(got[1:M + 1].view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("pad,shift", [(1, 0), (0, 1), (2, 3)])
def test_integers_are_exact_where_outputs_leave_element_by_element(pad, shift):
    """A pitch or base off 16 bytes, several tiles per pair: the chunk that both accumulators share leaves first."""
    M, N, K = 2064, 6384, 96
    comp, nib, dense = sparse_left(M, K, 6)
    B = oracle.gen_int8((K, N), 6, 2)
    tiled = ig.sp_pack_meta(nib, ig.BM_META_ROWS, M, K)
    flat = torch.full((shift + M * (N + pad) + 8,), 0x5A5A5A5A, dtype=torch.int32, device=dev())
    C = flat[shift:shift + M * (N + pad)].view(M, N + pad)[:, :N]
    with options(force_bn=224):
        ig.igemm_sparse_i32(comp, tiled, ig.BM_META_TILED, T(B), C, M, N, K, ig.BM_B_KN)
        assert_clean_status()
    assert np.array_equal(C.cpu().numpy(), oracle.igemm(dense, B, threads=0))
    C.fill_(0x5A5A5A5A)
    assert bool((flat == 0x5A5A5A5A).all()), "store outside the output"
