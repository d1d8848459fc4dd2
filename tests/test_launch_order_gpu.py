"""The order in which the blocks of all (batch, head) pairs are handed out: every pair and block once, in one group of
all pairs (causal, up to 64 pairs in the one-pass backward, shared operands within L2 in the forward) and in groups with
a short last one."""
import pytest
import torch

import flagattention_b200 as fa
import oracle
from flagattention_b200 import _C
from helpers import assert_within_2x, make_qkv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Hk,M,N,D,causal", [
    (16, 8, 4, 300, 300, 64, True),     # 64 pairs of the backward: one group
    (13, 5, 5, 300, 333, 64, True),     # 65: two groups of 32 and one of 1
    (3, 8, 2, 515, 515, 128, True),     # one group, more blocks than fit a wave with a partial last block
    (13, 5, 5, 200, 200, 64, False),    # not causal: groups
    (1, 3, 1, 130, 700, 128, True)])
def test_every_block_is_visited_once(B, H, Hk, M, N, D, causal):
    q, k, v, do = make_qkv(B, H, Hk, M, N, D, torch.bfloat16, "cuda", seed=B * H)
    for x in (q, k, v):
        x.requires_grad_()
    o, lse, tot = fa.flash_attention(q, k, v, causal, return_log_normalizer=True, return_total_attention=True)[:3]
    got = (o, lse, tot) + torch.autograd.grad(o, (q, k, v), do)
    outs = {}
    for up in (True, False):
        r = oracle.flash_attention(q, k, v, causal, return_log_normalizer=True, return_total_attention=True, upcast=up)[:3]
        outs[up] = r + torch.autograd.grad(r[0], (q, k, v), do)
    for name, x, r, t in zip(("o", "lse", "total", "dq", "dk", "dv"), got, outs[True], outs[False]):
        assert_within_2x(x, r, t, name)


@pytest.mark.parametrize("pairs,N", [(192, 672), (200, 672), (512, 300)])
def test_forward_of_many_short_walks(pairs, N):
    """Around 64 MB of keys and values in walks of at most 6 blocks: one group and groups, the same bits as a call for some
    of the heads alone."""
    q, k, v, _ = make_qkv(1, pairs, pairs, N, N, 128, torch.float16, "cuda", seed=pairs)
    with _C.kernel_family("one_cta_per_tile"):
        o = fa.flash_attention(q, k, v, True)
        for h in (0, 33, pairs - 40):   # (40: fewer would go to the split-KV kernels)
            some = slice(h, h + 40)
            assert torch.equal(o[:, some], fa.flash_attention(q[:, some], k[:, some], v[:, some], True)), h


@pytest.mark.parametrize("H,N", [(22, 8192), (23, 8192)])
def test_forward_at_the_l2_line(H, N):
    """22 x 8192 keys at head_dim 128 are 88 MiB and one group, 23 heads go in groups of 8: the same bits as a call
    for some of the heads alone."""
    q, k, v, _ = make_qkv(1, H, H, N, N, 128, torch.float16, "cuda", seed=H)
    with _C.kernel_family("one_cta_per_tile"):   # (one head alone would be split over a cluster)
        o = fa.flash_attention(q, k, v, True)
        for h in (0, 9, H - 1):
            assert torch.equal(o[:, h:h + 1], fa.flash_attention(q[:, h:h + 1], k[:, h:h + 1], v[:, h:h + 1], True)), h
