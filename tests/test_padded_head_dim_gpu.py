"""head_dim 16 and 32 on the tcgen05 kernels, which run them as 64 with zero columns: sizes around a tile,
grouped heads, keys and queries of different length, views of a fused projection whose neighbouring columns
hold NaN (they lie past the tensor map's extent and must never enter a product).  Short calls run on the
shape-generic kernels in part; the last three run on the padded ones at both head_dims: the forward with few query
tiles (one CTA a tile) and with more than two an SM (the persistent form), the backward, and total_attention where
there are 1024 queries or more."""
import pytest
import torch

import flagattention_b200 as fa
import oracle
from helpers import assert_within_2x

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [16, 32])
@pytest.mark.parametrize("B,H,Hk,M,N,causal", [
    (32, 8, 8, 64, 64, True), (16, 16, 4, 127, 129, True), (8, 16, 16, 385, 385, False), (4, 16, 2, 1000, 700, True),
    (2, 8, 4, 200, 1100, True), (2, 8, 4, 200, 2100, True), (4, 16, 8, 640, 2056, True), (1, 4, 2, 1100, 2050, True)])
def test_forward_backward_against_oracle(B, H, Hk, M, N, D, causal):
    gen = torch.Generator().manual_seed(M + N + D)

    def make(heads, length):   # a slice of a wider row, NaN on either side of it
        x = torch.full((B, length, heads, 3 * D), float("nan"), dtype=torch.bfloat16, device="cuda")
        x[..., D:2 * D] = torch.randn((B, length, heads, D), generator=gen).to(torch.bfloat16).cuda()
        return x[..., D:2 * D].transpose(1, 2).requires_grad_()

    q, k, v, do = make(H, M), make(Hk, N), make(Hk, N), make(H, M).detach()
    o, lse, tot = fa.flash_attention(q, k, v, causal, return_log_normalizer=True, return_total_attention=True)[:3]
    grads = torch.autograd.grad(o, (q, k, v), do)
    outs = {}
    for up in (True, False):
        ro, rl, rt = oracle.flash_attention(q, k, v, causal, return_log_normalizer=True, return_total_attention=True,
                                            upcast=up)
        outs[up] = (ro, rl, rt) + torch.autograd.grad(ro, (q, k, v), do)
    for name, x, r, t in zip(("o", "lse", "total", "dq", "dk", "dv"), (o, lse, tot) + grads, outs[True], outs[False]):
        seen = torch.isfinite(r)
        assert torch.equal(torch.isfinite(x), seen), name   # -inf of the rows that see no key
        assert_within_2x(torch.where(seen, x, 0), torch.where(seen, r, 0), torch.where(seen, t, 0), name)
