"""The forward at head_dim 16 and 32 and with dropout against 64 bits.  P goes into P V as a 16-bit value and a 16-bit
remainder there, so what is left is the rounding of the output."""
import math

import pytest
import torch

import flagattention_b200 as fa

pytestmark = pytest.mark.gpu


def _exact(q, k, v, causal, keep=None, far=None, w=0):
    M, N, g = q.shape[2], k.shape[2], q.shape[1] // k.shape[1]
    q, k, v = q.double(), k.double().repeat_interleave(g, 1), v.double().repeat_interleave(g, 1)
    s = q @ k.transpose(2, 3)
    distance = torch.arange(M, device=q.device)[:, None] + N - M - torch.arange(N, device=q.device)
    if far is not None:
        s = torch.where(distance >= w, far[0].double() @ far[1].double().transpose(2, 3), s)
    s = s * q.shape[3] ** -0.5
    if causal:
        s = s.masked_fill(distance < 0, -math.inf)
    p = torch.softmax(s, -1)
    return (p if keep is None else p * keep) @ v, torch.logsumexp(s, -1)


def _check(o, want):
    relative = lambda x: ((x.double() - want).norm() / want.norm()).item()
    # the output's own rounding; the remainder leaves 2^-16 (bf16) or 2^-22 of a weight, sums are fp32: a hundredth
    assert relative(o) <= 1.01 * relative(want.to(o.dtype))


def _inputs(dtype, scale, *shapes):
    gen = torch.Generator(device="cuda").manual_seed(sum(shapes[0]))
    return [(torch.randn(s, generator=gen, device="cuda") * (scale if i < len(shapes) - 1 else 1)).to(dtype)
            for i, s in enumerate(shapes)]


# scores of deviation 1 and 4: with the second a few weights carry a row
@pytest.mark.parametrize("scale", [1.0, 2.0])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,H,Hk,M,N,D,causal", [
    (2, 4, 2, 300, 2100, 16, True), (1, 4, 4, 1100, 1100, 32, False), (8, 8, 8, 640, 2056, 16, True),
    (8, 8, 2, 640, 1025, 32, False)])
def test_padded_head_dim(B, H, Hk, M, N, D, causal, dtype, scale):
    q, k, v = _inputs(dtype, scale, (B, H, M, D), (B, Hk, N, D), (B, Hk, N, D))
    o, lse = fa.flash_attention(q, k, v, causal, return_log_normalizer=True)[:2]
    want, want_lse = _exact(q, k, v, causal)
    _check(o, want)
    # lse = shift + log(sum): two roundings of a number below 32, the logarithm's and those of the sum's 2^11 terms
    assert (lse - want_lse).abs().max() <= 4 * 2 ** -20


@pytest.mark.parametrize("scale", [1.0, 2.0])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,D,w", [(1300, 1300, 16, 300), (200, 1030, 32, 128)])
def test_padded_piecewise(M, N, D, w, dtype, scale):
    q1, k1, q2, k2, v = _inputs(dtype, scale, (2, 4, M, D), (2, 4, N, D), (2, 4, M, D), (2, 4, N, D), (2, 4, N, D))
    _check(fa.piecewise_attention(q1, k1, q2, k2, v, w, causal=True), _exact(q1, k1, v, True, None, (q2, k2), w)[0])


@pytest.mark.parametrize("scale", [1.0, 2.0])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,H,Hk,M,N,D,causal", [
    (2, 8, 8, 512, 512, 64, False), (1, 8, 2, 700, 901, 128, True), (2, 8, 8, 333, 1031, 32, True),
    (2, 8, 4, 333, 1031, 16, False)])
def test_dropout(B, H, Hk, M, N, D, causal, dtype, scale):
    p = 0.1
    q, k, v = _inputs(dtype, scale, (B, H, M, D), (B, Hk, N, D), (B, Hk, N, D))
    o, _, _, seed, offset = fa.flash_attention(q, k, v, causal, dropout_p=p, return_seed_offset=True)
    keep = fa.testing.recompute_mask(B, H, M, N, p, seed, offset, "cuda").double() / (1 - p)
    _check(o, _exact(q, k, v, causal, keep)[0])


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,M,N,D", [(2, 300, 2100, 16), (2, 300, 1100, 32), (40, 300, 1100, 32)])
def test_infinite_values(B, M, N, D, dtype):
    """An infinite value that every query sees gives its column that infinity."""
    q, k, v = _inputs(dtype, 1.0, (B, 4, M, D), (B, 4, N, D), (B, 4, N, D))
    v[:, :, 100, 3], v[:, :, 5, 9] = float("inf"), -float("inf")
    o = fa.flash_attention(q, k, v)
    assert (o[..., 3] == float("inf")).all() and (o[..., 9] == -float("inf")).all()
    assert o.isfinite().sum() == o.numel() // D * (D - 2)
