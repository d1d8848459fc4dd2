"""The partition sizes paged and dense decoding choose for themselves, and the results they give at the edges of
the rule against one pass over the keys."""
import pytest
import torch

import flagattention_b200 as fa
from flagattention_b200 import paged


@pytest.mark.parametrize("start", [256, 512])
@pytest.mark.parametrize("pairs", [1, 4, 8, 32, 118, 119, 512, 2048])
@pytest.mark.parametrize("context", [1025, 4096, 32767, 131072])
def test_partitions_double_while_the_gpu_is_busy(start, pairs, context):
    for most in (2048, 4096):
        size = paged.coarsen_partition(start, pairs, context, 148, most)
        assert size % start == 0 and start <= size <= most and size & (size - 1) == 0
        ctas = pairs * -(-context // size)
        assert size == start or ctas >= 0.8 * 148
        assert size == most or pairs * -(-context // (2 * size)) < 0.8 * 148


@pytest.mark.gpu
@pytest.mark.parametrize("seqs,Hk,group,hi,block", [(1, 1, 4, 40000, 16), (3, 4, 8, 32769, 32), (30, 8, 1, 4097, 16),
                                                    (80, 4, 4, 4096, 16), (2, 2, 1, 1025, 16)])
def test_paged_against_one_pass(seqs, Hk, group, hi, block):
    D, gen = 64, torch.Generator().manual_seed(hi)
    blocks = -(-hi // block)
    lens = torch.randint(1, hi + 1, (seqs,), generator=gen)
    lens[0] = hi
    cache = [torch.randn((blocks + 3, Hk, block, D), generator=gen).half().cuda() for _ in range(2)]
    q = torch.randn((seqs, Hk * group, D), generator=gen).half().cuda()
    table = torch.randint(0, blocks + 3, (seqs, blocks), generator=gen).to(torch.int32).cuda()
    args = (q, *cache, lens.to(torch.int32).cuda(), table, D ** -0.5, hi)
    # both accumulate in fp32 and round once to fp16: half a unit each, outputs below 1
    torch.testing.assert_close(fa.paged_attention(*args), fa.paged_attention(*args, 1), atol=2 ** -11, rtol=2 ** -10)


@pytest.mark.gpu
@pytest.mark.parametrize("B,H,Hk,N", [(1, 16, 16, 262144), (1, 8, 2, 65536), (2, 8, 8, 2048), (16, 8, 8, 2064)])
def test_dense_decode_against_64_bits(B, H, Hk, N):
    gen = torch.Generator(device="cuda").manual_seed(N)
    q, k, v = (torch.randn((B, h, n, 128), generator=gen, device="cuda", dtype=torch.float16)
               for h, n in ((H, 1), (Hk, N), (Hk, N)))
    o = fa.flash_attention(q, k, v)
    for b in range(B):
        for h in range(0, H, 5):
            s = torch.softmax(k[b, h * Hk // H].double() @ q[b, h, 0].double() * 128 ** -0.5, 0)
            want = s @ v[b, h * Hk // H].double()
            # P is rounded to 16 bits: an error of 2^-12 of |p v| a key, adding up like noise; and o once
            bound = 6 * 2 ** -12 * (s[:, None] * v[b, h * Hk // H].double()).norm(dim=0).max() + 2 ** -11 * want.abs().max()
            assert (o[b, h, 0] - want).abs().max() <= bound
