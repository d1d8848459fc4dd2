"""Decoding kernels against 64 bits: what is left is the rounding of the output, whatever the partitions are."""
import pytest
import torch

import flagattention_b200 as fa

pytestmark = pytest.mark.gpu


def _relative(x, want):
    return ((x.double() - want).norm() / want.norm()).item()


def _limit(want, dtype):
    # The output's own rounding.  On top: P as value and remainder is good to 2^-22 (fp16) or 2^-16 (bf16) of itself
    # (a remainder below fp16's smallest number, 2^-24 of the run's maximum, is lost: weights that small do not count),
    # and fp32 sums of up to 2^15 / 64 groups a warp.  A hundredth of the rounding covers both.
    return 1.01 * _relative(want.to(dtype), want)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("seqs,Hk,group,D,hi,splits", [
    (12, 8, 4, 128, 32768, 0), (12, 8, 4, 128, 32768, 16), (2, 2, 8, 64, 9000, 0), (3, 2, 20, 256, 700, 1), (1, 1, 1, 16, 33, 0)])
def test_paged(seqs, Hk, group, D, hi, splits, dtype):
    gen = torch.Generator(device="cuda").manual_seed(hi + D)
    lens = torch.randint(1, hi + 1, (seqs,), generator=torch.Generator().manual_seed(hi))
    lens[0] = hi
    blocks = -(-hi // 16)
    cache = [torch.randn((blocks + 5, Hk, 16, D), generator=gen, device="cuda", dtype=dtype) for _ in range(2)]
    q = torch.randn((seqs, Hk * group, D), generator=gen, device="cuda", dtype=dtype)
    table = torch.randint(0, blocks + 5, (seqs, blocks), generator=gen, device="cuda", dtype=torch.int32)
    out = fa.paged_attention(q, *cache, lens.int().cuda(), table, D ** -0.5, hi, splits)
    want = torch.empty(q.shape, dtype=torch.float64, device="cuda")
    for i, n in enumerate(lens.tolist()):
        k, v = (x[table[i, :-(-n // 16)].long()].double().transpose(0, 1).flatten(1, 2)[:, :n] for x in cache)
        s = q[i].double().unflatten(0, (Hk, group)) @ k.transpose(1, 2) * D ** -0.5
        want[i] = (torch.softmax(s, -1) @ v).flatten(0, 1)
    assert _relative(out, want) <= _limit(want, dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,H,Hk,M,N,D", [(1, 8, 8, 1, 65536, 128), (2, 8, 2, 3, 4096, 64)])
def test_dense(B, H, Hk, M, N, D, dtype):
    gen = torch.Generator(device="cuda").manual_seed(N)
    q, k, v = (torch.randn((B, h, n, D), generator=gen, device="cuda", dtype=dtype) for h, n in ((H, M), (Hk, N), (Hk, N)))
    kk, vv = (x.double().repeat_interleave(H // Hk, 1) for x in (k, v))
    want = torch.softmax(q.double() @ kk.transpose(2, 3) * D ** -0.5, -1) @ vv
    assert _relative(fa.flash_attention(q, k, v), want) <= _limit(want, dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("group", [1, 8, 16])
def test_infinite_values(group, dtype):
    """An infinite value gives its column that infinity, with the remainder in rows of its own (up to 8) and without."""
    gen = torch.Generator(device="cuda").manual_seed(group)
    q, k, v = (torch.randn((2, h, n, 64), generator=gen, device="cuda", dtype=dtype) for h, n in ((2 * group, 1), (2, 1040), (2, 1040)))
    v[:, :, 700, 3], v[:, :, 5, 60] = float("inf"), -float("inf")
    o = fa.flash_attention(q, k, v)
    assert (o[..., 3] == float("inf")).all() and (o[..., 60] == -float("inf")).all()
    assert o.isfinite().sum() == o.numel() // 64 * 62
