"""Forward calls whose query tiles are too few for the SMs: a cluster of 2, 4 or 8 CTAs shares the walk of each.  Sizes
around the lines of the rule, with ranks that get no key tile that a row sees, rows that see no key at all, padded
head_dims and piecewise lists that switch branch inside a rank, against the oracle."""
import pytest
import torch

import flagattention_b200 as fa
import oracle
from flagattention_b200 import _C
from helpers import assert_within_2x, make_qkv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,H,Hk,M,N,D,causal", [
    (1, 32, 8, 512, 3000, 128, True),     # 2 CTAs a tile
    (2, 16, 16, 64, 2900, 128, False),    # 8
    (1, 8, 2, 1024, 1024, 128, True),     # 4: ranks past the diagonal of the first rows
    (1, 9, 3, 700, 520, 64, True),        # the first 180 rows see no key, whole tiles among them
    (3, 16, 4, 130, 1217, 64, True),
    (1, 8, 8, 1030, 2100, 32, True), (1, 8, 8, 1030, 2100, 16, False),
    (1, 4, 4, 512, 513, 64, True),
    # calls that the split-KV kernels took: P with its remainder
    (1, 8, 8, 32, 2000, 128, True), (1, 4, 2, 300, 1000, 64, True), (2, 2, 1, 45, 40, 128, False), (1, 3, 3, 250, 77, 64, True)])
def test_split_walks(B, H, Hk, M, N, D, causal, dtype):
    q, k, v, _ = make_qkv(B, H, Hk, M, N, D, dtype, "cuda", 2.0, seed=M + N)
    junk = torch.full_like(q, float("nan"))   # the outputs come from this memory
    del junk
    o, lse = fa.flash_attention(q, k, v, causal, return_log_normalizer=True)[:2]
    r, t = (oracle.flash_attention(q, k, v, causal, return_log_normalizer=True, upcast=up)[:2] for up in (True, False))
    assert_within_2x(o, r[0], t[0], "o")
    assert_within_2x(lse, r[1], t[1], "lse")
    assert torch.equal(o, fa.flash_attention(q, k, v, causal))
    with _C.kernel_family("one_cta_per_tile"):
        one = fa.flash_attention(q, k, v, causal)
    # both round P to 16 bits against a reference that may lag the maximum by 2^8, and o once: two roundings each
    ulp = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    assert (o.float() - one.float()).norm() <= 4 * ulp * one.float().norm()


@pytest.mark.parametrize("B,H,L,D,w,causal", [(1, 4, 1000, 128, 300, True), (1, 3, 777, 64, 900, True),
                                              (1, 2, 1500, 64, 100, False), (1, 5, 1100, 32, 500, True),
                                              (1, 2, 2050, 128, 1, True)])
def test_split_piecewise_lists(B, H, L, D, w, causal):
    gen = torch.Generator().manual_seed(L)
    x = [torch.randn((B, H, L, D), generator=gen).to(torch.bfloat16).cuda() for _ in range(5)]
    o = fa.piecewise_attention(*x, w, causal=causal)
    r, t = (oracle.piecewise_attention(*x, w, causal=causal, upcast=up) for up in (True, False))
    assert_within_2x(o, r, t, "o")


def test_values_at_the_edges_of_the_range():
    """Infinite and NaN values reach the output where the unsplit kernel lets them, and nowhere else."""
    q, k, v, _ = make_qkv(1, 4, 4, 512, 2048, 64, torch.bfloat16, "cuda", seed=3)
    k[0, 0, 1500, 0], v[0, 1, 100, 5], v[0, 2, 2000, 7] = float("nan"), float("inf"), float("-inf")
    o = fa.flash_attention(q, k, v, True)
    with _C.kernel_family("one_cta_per_tile"):
        one = fa.flash_attention(q, k, v, True)
    assert torch.equal(torch.isnan(o), torch.isnan(one)) and torch.equal(torch.isinf(o), torch.isinf(one))
    assert not torch.isfinite(o).all() and torch.isfinite(o[0, 3]).all()


@pytest.mark.parametrize("B,H,M,N,D,std", [(1, 8, 32, 3000, 128, 1.0), (1, 4, 200, 1500, 64, 2.0), (1, 4, 64, 400, 128, 2.0)])
def test_few_rows_are_no_less_precise_than_the_split_kv_kernels(B, H, M, N, D, std):
    from flagattention_b200 import flash, split_kv
    q, k, v, _ = make_qkv(B, H, H, M, N, D, torch.bfloat16, "cuda", std, seed=M)
    s = (q.double() @ k.double().transpose(2, 3)) * D ** -0.5
    s.masked_fill_(torch.ones(M, N, dtype=torch.bool, device="cuda").triu(N - M + 1), float("-inf"))
    want = torch.softmax(s, 3) @ v.double()
    few = flash._few_rows_forward(q, k, v, True, D ** -0.5)
    split = split_kv._splitkv_forward(q, k, v, True, D ** -0.5, 4)
    errors = [((x[0].double() - want).norm() / want.norm()).item() for x in (few, split)]
    assert errors[0] <= errors[1] * 1.02, errors     # (both end in the same rounding of o)
    assert (few[1].double() - torch.logsumexp(s, 3)).abs().max() <= 2e-5
    assert flash._few_rows_forward(q[:, :, :31], k, v, True, 0.1) is None
