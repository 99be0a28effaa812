"""Per-token quantiser: every shape of its thread groups, and rows that hold infinities or NaNs."""
import numpy as np
import pytest
import torch

import oracle
from bare_metal_b200 import igemm as ig
from _gpu import T, assert_clean_status

pytestmark = pytest.mark.gpu


# one-warp groups (several rows a CTA), groups of 1, 2 and 4 pieces a thread, rows longer than a group holds
@pytest.mark.parametrize("M,K", [(1, 16), (3, 256), (149, 272), (150, 1024), (151, 1040), (148, 8192), (149, 8208), (200, 16384),
                                 (150, 16400), (2, 32768), (3, 33040), (149, 24592)])
def test_all_group_sizes_match_the_reference_quantiser(M, K):
    rng = np.random.default_rng(M + 7 * K)
    x = (rng.standard_normal((M, K)) * np.exp2(rng.uniform(-14, 6, (M, 1)))).astype(np.float16)
    x[:, ::5] = np.rint(x[:, ::5].astype(np.float32) * 2).astype(np.float16) / np.float16(2)      # ties and zeros of both signs
    x[0, K - 1] = np.float16(-127)
    q, s = ig.quantize_rows(T(x), M, K)
    assert_clean_status()
    x32 = x.astype(np.float32)
    want_s = np.array([oracle.compute_scale(r) for r in x32], np.float32)
    assert np.array_equal(s.cpu().numpy(), want_s)
    assert np.array_equal(q.cpu().numpy(), np.stack([oracle.quantize_symmetric(r, a) for r, a in zip(x32, want_s)]))


@pytest.mark.parametrize("K", [256, 4096])
def test_infinities_and_nans_quantise_as_before(K):
    """An infinity makes the row's scale infinite and its values 0; a NaN counts for nothing and becomes 0."""
    x = np.linspace(-3, 5, 4 * K).astype(np.float16).reshape(4, K)
    x[1, 7], x[2, K - 3] = np.inf, np.nan
    x[3, :] = np.nan
    q, s = (t.cpu().numpy() for t in ig.quantize_rows(T(x), 4, K))
    assert np.isinf(s[1]) and not q[1].any()
    clean = x[2].astype(np.float32)
    clean[K - 3] = 0
    assert s[2] == oracle.compute_scale(clean) and np.array_equal(q[2], oracle.quantize_symmetric(clean, s[2]))
    assert s[3] == 1 and not q[3].any()
    assert s[0] == oracle.compute_scale(x[0].astype(np.float32))
