"""The keep bits the tcgen05 kernels compute for themselves, element by element against the mask the library
regenerates: counters that cross 2^32 inside a tile (and inside a thread's run of 32), ragged sizes, grouped heads,
both memory layouts; the shortest cases at head_dim 16 and 32 run on the shape-generic kernels.  With q = k = 0 every
weight is 1 / N, so the outputs of one-hot values are the mask itself."""
import pytest
import torch

import flagattention_b200 as fa
from flagattention_b200 import flash

pytestmark = pytest.mark.gpu

STREAMS = [(0, 0), (2 ** 63 + 12345, 2 ** 32 - 4000), (2 ** 40 + 17, 2 ** 34 - 100), (7, 2 ** 33 + 3)]


@pytest.mark.parametrize("seed,offset", STREAMS)
@pytest.mark.parametrize("p", [0.1, 0.5, 0.9999])
@pytest.mark.parametrize("H,M,N,D", [(3, 300, 64, 64), (2, 129, 128, 128), (5, 70, 31, 32), (2, 500, 16, 16)])
def test_forward_mask(H, M, N, D, p, seed, offset):
    q, k = (torch.zeros(2, H, n, D, device="cuda", dtype=torch.float16) for n in (M, N))
    v = torch.eye(N, D, device="cuda", dtype=torch.float16).expand(2, H, N, D).contiguous()
    o, _ = flash._forward(q, k, v, False, 1.0, p, seed, offset)
    mask = fa.testing.recompute_mask(2, H, M, N, p, seed, offset, "cuda")
    assert torch.equal(o[..., :N] > 0.5 / (N * (1 - p)), mask)


@pytest.mark.parametrize("seed,offset", STREAMS)
@pytest.mark.parametrize("p", [0.1, 0.5])
@pytest.mark.parametrize("M,N,D", [(64, 300, 64), (128, 257, 128), (31, 100, 32), (32, 320, 32)])
def test_backward_mask(M, N, D, p, seed, offset):
    H, Hk = 4, 2
    q = torch.zeros(2, H, M, D, device="cuda", dtype=torch.float16)
    k, v = (torch.zeros(2, Hk, N, D, device="cuda", dtype=torch.float16) for _ in range(2))
    # dV[n, m] = (keep of the group's first head + 2 * keep of its second) / (N (1 - p))
    do = torch.eye(M, D, device="cuda", dtype=torch.float16) * torch.tensor([1., 2.] * 2, device="cuda").half()[:, None, None]
    do = do.expand(2, H, M, D).contiguous()
    o, lse = flash._forward(q, k, v, False, 1.0, p, seed, offset)
    dq, dk, dv = flash._backward(q, k, v, o, lse, do, False, 1.0, None, p, seed, offset)
    mask = fa.testing.recompute_mask(2, H, M, N, p, seed, offset, "cuda").to(torch.int64)
    got = (dv.float() * (N * (1 - p))).round().to(torch.int64)[..., :M].transpose(2, 3)
    assert torch.equal(got, mask[:, 0::2] + 2 * mask[:, 1::2])
    assert not dq.any() and not dk.any()   # k = 0 and q = 0


@pytest.mark.parametrize("seed,offset", STREAMS)
@pytest.mark.parametrize("D", [16, 32])
def test_forward_mask_of_long_rows(D, seed, offset):
    """head_dim 16 and 32 padded: the values are one-hot over a window of D keys."""
    H, M, N, p = 3, 130, 1100, 0.1
    q, k = (torch.zeros(2, H, n, D, device="cuda", dtype=torch.float16) for n in (M, N))
    mask = fa.testing.recompute_mask(2, H, M, N, p, seed, offset, "cuda")
    for first in (0, 56, 1024, N - D):
        v = torch.zeros(2, H, N, D, device="cuda", dtype=torch.float16)
        v[:, :, first:first + D] = torch.eye(D, device="cuda", dtype=torch.float16)
        o, _ = flash._forward(q, k, v, False, 1.0, p, seed, offset)
        assert torch.equal(o > 0.5 / (N * (1 - p)), mask[..., first:first + D])


@pytest.mark.parametrize("H,Hk,M,N,D,causal", [(4, 2, 300, 300, 64, True), (4, 4, 129, 200, 128, False), (8, 2, 150, 1030, 32, True)])
def test_layouts(H, Hk, M, N, D, causal):
    """(batch, length, heads, head_dim) in memory gives the bits of the contiguous call; dq is a sum of fp32 reductions
    in any order, rounded once: a unit of bf16 at most."""
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    make = lambda h, n: torch.randn(2, n, h, D, generator=gen, device="cuda", dtype=torch.bfloat16).transpose(1, 2)
    q, k, v, do = make(H, M), make(Hk, N), make(Hk, N), make(H, M)
    got = []
    for ready in (lambda x: x, lambda x: x.contiguous()):
        a, b, c, d = map(ready, (q, k, v, do))
        o, lse = flash._forward(a, b, c, causal, D ** -0.5, 0.2, 11, 2 ** 32 - 999)
        got.append((o, lse) + flash._backward(a, b, c, o, lse, d, causal, D ** -0.5, None, 0.2, 11, 2 ** 32 - 999))
    for name, x, y in zip(("o", "lse", "dq", "dk", "dv"), *got):
        if name == "dq":
            torch.testing.assert_close(x, y, atol=2 ** -8 * y.abs().max().item() * 2 ** -6, rtol=2 ** -7)
        else:
            assert torch.equal(x, y), name
