"""Dropout decisions kept from the forward: the backward that reads them against the one that draws them again."""
import pytest
import torch

import flagattention_b200 as fa
from flagattention_b200 import _C, flash
from helpers import make_qkv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,H,Hk,M,N,D,causal", [
    (2, 8, 8, 512, 512, 64, False), (1, 8, 2, 300, 333, 128, True), (2, 4, 4, 129, 65, 64, True),
    (1, 16, 4, 700, 1000, 32, True), (1, 8, 8, 1000, 4096, 128, False), (1, 8, 8, 200, 2048, 64, True)])
def test_kept_bits_are_the_drawn_ones(B, H, Hk, M, N, D, causal, dtype):
    q, k, v, do = make_qkv(B, H, Hk, M, N, D, dtype, "cuda", seed=M + N)
    p, seed, offset = 0.3, 77, 2 ** 32 - 1000   # counters cross 2^32
    junk = torch.full((8 << 20,), 255, dtype=torch.uint8, device="cuda")   # the buffer may come from this memory
    del junk
    o, lse, bits = flash._forward(q, k, v, causal, D ** -0.5, p, seed, offset, True)
    assert bits is not None
    o2, lse2 = flash._forward(q, k, v, causal, D ** -0.5, p, seed, offset)
    assert torch.equal(o, o2) and torch.equal(lse, lse2)
    got = flash._backward(q, k, v, o, lse, do, causal, D ** -0.5, None, p, seed, offset, bits)
    want = flash._backward(q, k, v, o, lse, do, causal, D ** -0.5, None, p, seed, offset)
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    # dq is summed in any order: a rounding to 16 bits apart at most
    ulp = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7
    assert (got[0].float() - want[0].float()).abs().max() <= ulp * want[0].float().abs().max()


def test_where_none_are_kept():
    q, k, v, _ = make_qkv(1, 8, 8, 200, 2112, 64, torch.float16, "cuda")
    assert flash._forward(q, k, v, False, 0.1, 0.1, 1, 0, True)[2] is None      # more than 32 D keys
    x = q[:, :, :160]
    assert flash._forward(x, x, x, False, 0.1, 0.0, 1, 0, True)[2] is None      # no dropout
    with _C.kernel_family("generic"):
        assert flash._forward(x, x, x, False, 0.1, 0.1, 1, 0, True)[2] is None
    y = x[:, :1].expand(1, 8, 160, 64)                                          # broadcast over the heads
    o, _, bits = flash._forward(x, y, y, False, 0.1, 0.1, 1, 0, True)
    want = flash._forward(x, y.contiguous(), y.contiguous(), False, 0.1, 0.1, 1, 0)[0]
    assert bits is None and (o.float() - want.float()).abs().max() <= 4 * 2 ** -11 * want.float().abs().max()


def test_backward_kernels_chosen_later():
    """The mode in force when the gradients are asked for decides, whatever the forward kept."""
    q, k, v, do = make_qkv(4, 16, 16, 768, 768, 64, torch.float16, "cuda", seed=9)   # 38 M elements: kept
    for x in (q, k, v):
        x.requires_grad_()
    saved = []
    torch.cuda.manual_seed(5)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: saved.append(t) or t, lambda t: t):
        o = fa.flash_attention(q, k, v, True, dropout_p=0.2)
        fa.flash_attention(q[:, :, :256], k[:, :, :256], v[:, :, :256], True, dropout_p=0.2)   # 4 M: drawn again
    assert len(saved) == 6 + 5
    one = torch.autograd.grad(o, (q, k, v), do, retain_graph=True)
    with flash.backward_mode("two_kernel"):
        two = torch.autograd.grad(o, (q, k, v), do, retain_graph=True)
    for a, b in zip(one, two):
        assert (a.float() - b.float()).abs().max() <= 8 * 2 ** -11 * b.float().abs().max()
