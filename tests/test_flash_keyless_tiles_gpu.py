"""Causal calls with far more queries than keys: long runs of query tiles that see no key, between tiles that
do, in the order the persistent forward works through them."""
import pytest
import torch

import flagattention_b200 as fa
from flagattention_b200 import _C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,M,N", [(4, 16, 2048, 128), (2, 40, 1300, 200), (1, 64, 4096, 1)])
def test_runs_of_tiles_without_keys(B, H, M, N, D):
    gen = torch.Generator().manual_seed(M + N)
    q, k, v = (torch.randn((B, H, n, D), generator=gen).half().cuda() for n in (M, N, N))
    with _C.kernel_family("one_cta_per_tile"):
        want = fa.flash_attention(q, k, v, True, return_log_normalizer=True)[:2]
    for _ in range(3):
        junk = [torch.full_like(t, float("nan")) for t in want]   # the outputs come from this memory
        del junk
        o, lse = fa.flash_attention(q, k, v, True, return_log_normalizer=True)[:2]
        assert torch.equal(o, want[0]) and torch.equal(lse, want[1])
    assert not o[:, :, :M - N].any() and torch.isinf(lse[:, :, :M - N]).all()
