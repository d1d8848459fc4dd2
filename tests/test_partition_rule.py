"""The partition sizes paged and dense decoding choose for themselves, and the results they give at the edges of
the rule against one pass over the keys or against 64 bits."""
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
@pytest.mark.parametrize("seqs,Hk,group,hi,block", [(60, 1, 16, 1100, 16), (37, 2, 8, 1100, 16), (38, 2, 8, 1100, 16),
                                                    (290, 1, 16, 1100, 16), (290, 1, 8, 1100, 16)])
def test_rows_of_the_reduction(seqs, Hk, group, hi, block):
    """Few and many rows: 256, 128, 64 and 32 threads reduce one."""
    test_paged_against_one_pass(seqs, Hk, group, hi, block)


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
    # Both take P as a value and a remainder, add up in fp32 and round once to fp16, so that a result falls to the
    # next number at most.  In the fp32 sums of 40000 / 64 groups a warp, of numbers that add up to at most the
    # largest |v| (5), 2^-24 a step adds up like noise: sqrt(625) * 5 * 2^-24 < 2^-17, where the outputs are small.
    torch.testing.assert_close(fa.paged_attention(*args), fa.paged_attention(*args, 1), atol=2 ** -17, rtol=2 ** -10)


@pytest.mark.parametrize("base", [256, 512])
@pytest.mark.parametrize("seqs", [1, 4, 16, 64, 511, 3000])
@pytest.mark.parametrize("ctas", [1, 2, 8, 32, 128, 300])
@pytest.mark.parametrize("context", [1025, 2048, 4097, 32768, 131072])
def test_workspace_partitions(base, seqs, ctas, context):
    size, finest, coarsest, busy, parts = paged.size_partitions(base, seqs, ctas, context, 148)
    cdiv = lambda a, b: -(-a // b)
    largest = size or next(base << i for i in range(9) if base << i >= context)
    assert largest in [base << i for i in range(4)] and coarsest == 2048 and finest in (base, size)
    # growing to this size left one sequence enough CTAs of its own, or took away launches worth more
    assert (largest == base or ctas * cdiv(context, largest) >= 0.8 * 148
            or seqs * ctas * cdiv(context, largest // 2) > 35 * 148)
    if size:
        assert context > size and (busy > 0) != (parts > 0) and (busy == 0 or seqs <= 2048)
        # shorter sequences than the bound are cut finer where there are few of them
        assert finest == base or seqs * ctas >= 2 * 148


def test_a_split_count_that_changes_in_place_makes_another_plan():
    plan = lambda n: paged._plan(2, 8, 8, 16, 5000, n, 148)
    n = torch.tensor(4)
    assert plan(n) == plan(4) == (2048, 3, None)
    n.fill_(8)
    assert plan(n) == plan(8) == (1024, 5, None)


def _partitions(monkeypatch, lens, most, Hk, group, D=64, block=16):
    """Partitions each sequence was cut into: the slots of the NaN-filled workspace that the kernel wrote."""
    kept = []
    real = paged.partition_workspace

    def filled(rows, P, D, device):
        ws = real(rows, P, D, device)
        ws[0].fill_(float("nan"))
        kept.append((ws[0], rows, P))
        return ws

    monkeypatch.setattr(paged, "partition_workspace", filled)
    q = torch.zeros((len(lens), Hk * group, D), device="cuda", dtype=torch.float16)
    cache = torch.zeros((8, Hk, block, D), device="cuda", dtype=torch.float16)
    table = torch.zeros((len(lens), -(-most // block)), device="cuda", dtype=torch.int32)
    fa.paged_attention(q, cache, cache, torch.tensor(lens, dtype=torch.int32, device="cuda"), table, 1.0, most)
    (ws, rows, P), = kept
    written = ws[rows * P * D:][:rows * P].view(len(lens), Hk * group, P).isfinite().sum(2)
    assert (written == written[:, :1]).all()
    return written[:, 0].tolist(), P


@pytest.mark.gpu
@pytest.mark.parametrize("lens,most,Hk,group", [
    ([1500] * 4, 32768, 8, 4), ([1500] * 8, 131072, 2, 8), ([1500] * 20, 32768, 2, 8), ([4096] + [200] * 63, 4096, 2, 8),
    ([4096] + [200] * 63, 4096, 8, 4), ([2048] * 16, 2048, 8, 4), ([3000, 1, 0, 17], 3000, 8, 1), ([1500] * 3, 20000, 4, 40)])
def test_lengths_below_the_bound_keep_the_gpu_busy(monkeypatch, lens, most, Hk, group):
    """max_context_len is an upper bound, and lengths differ: there are as many CTAs as keep the GPU busy, or as many as
    partitions of 256 tokens give."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    parts, P = _partitions(monkeypatch, lens, most, Hk, group)
    assert all((n > 0) == (length > 0) and n <= P for n, length in zip(parts, lens))
    finest = [-(-length // 256) for length in lens]
    rows = Hk * -(-group // 16)
    assert sum(parts) * rows >= min(int(0.8 * sms), sum(finest) * rows)
    assert all(n <= f for n, f in zip(parts, finest))


@pytest.mark.gpu
@pytest.mark.parametrize("lens,most", [([32768] + [200] * 63, 32768), ([5000, 4095, 4097, 1], 5000), ([1025, 1, 256, 257], 60000)])
@pytest.mark.parametrize("index", [torch.int32, torch.int64])
def test_uneven_lengths_against_one_pass(lens, most, index):
    D, Hk, gen = 64, 2, torch.Generator(device="cuda").manual_seed(most)
    q = torch.randn((len(lens), Hk * 4, D), generator=gen, device="cuda", dtype=torch.float16)
    cache = [torch.randn((500, Hk, 32, D), generator=gen, device="cuda", dtype=torch.float16) for _ in range(2)]
    table = torch.randint(0, 500, (len(lens), -(-most // 32)), generator=gen, device="cuda").to(index)
    args = (q, *cache, torch.tensor(lens, dtype=torch.int32, device="cuda"), table, D ** -0.5, most)
    torch.testing.assert_close(fa.paged_attention(*args), fa.paged_attention(*args, 1), atol=2 ** -17, rtol=2 ** -10)


def test_sizes_that_do_not_nest_are_refused(built_lib):
    """Before any CUDA call."""
    from flagattention_b200 import _C
    args = _C.PagedArgs()
    for name, _ in args._fields_:
        if name in ("query", "key_cache", "value_cache", "out", "context_lens", "block_tables", "part_out", "part_max", "part_sum"):
            setattr(args, name, 0x1000)
    args.num_seqs, args.num_q_heads, args.num_kv_heads, args.head_size, args.block_size = 1, 1, 1, 64, 16
    args.max_context_len, args.partition_size = 5000, 1024
    call = lambda *a: _C.call("fa_paged_attention")(bytes(args), *a, 0)
    for bad in ((0, 2048, 100, 0), (24, 2048, 100, 0), (2048, 2048, 100, 0), (256, 128, 100, 0), (256, 768, 100, 0),
                (768, 1536, 100, 0), (256, 2048, 0, 0), (256, 2048, -1, 1), (256, 1 << 25, 100, 0)):
        assert call(*bad) == -1
    args.partition_size = 0
    assert call(256, 2048, 100, 0) == -1
    args.partition_size, args.num_seqs = 1024, 2049
    assert call(256, 2048, 100, 0) == -1


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
