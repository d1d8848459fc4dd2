"""paged_attention: single-token decode over a block-table KV cache.

Mirrors src/flag_attn/paged.py:6-163: same arguments, same split rule
(num_splits == 0 picks it automatically, 1 disables it, > 1 fixes the count),
returns a new tensor shaped like `query`.
"""
import functools

import torch

from . import _C, _native

__all__ = ["attention", "reshape_and_cache"]


def _next_power_of_2(n):
    return 1 << (max(int(n), 1) - 1).bit_length()


def _cdiv(a, b):
    return (a + b - 1) // b


def plan_partitions(num_seqs, num_kv_heads, kv_block_size, max_context_len, num_splits, num_sms):
    """Returns (num_splits, partition_size) by the reference's rule
    (src/flag_attn/paged.py:40-53); partition_size is 0 when there is one pass."""
    partition_size = 0
    if num_splits == 0:
        if num_seqs * num_kv_heads > 2 * num_sms:
            num_splits = 1
            if max_context_len >= 4096:
                partition_size = max(256, kv_block_size)
                num_splits = _cdiv(max_context_len, partition_size)
        else:
            partition_size = max(256, kv_block_size)
            num_splits = _cdiv(max_context_len, partition_size)
            if max_context_len <= 1024 or kv_block_size >= 256:
                num_splits = 1
    elif num_splits > 1:
        partition_size = _next_power_of_2(_cdiv(max_context_len, num_splits))
    if num_splits == 1:
        partition_size = 0
    return num_splits, partition_size


def coarsen_partition(partition_size, pairs, context_len, num_sms, most=2048):
    """Partitions of `partition_size` tokens, doubled up to `most` while `pairs` contexts of `context_len` tokens, one
    CTA a partition, keep the GPU busy with them.

    A CTA's four warps fill a ring of loads and merge their results once per partition, and every partition writes and
    re-reads a row of fp32 partial output, so short ones cost bandwidth; fewer CTAs than SMs cost more (fp16, one
    context of 32768 over 4 kv heads: 256: 54 us, 512: 37, 1024: 33, 2048: 40)."""
    while partition_size < most and pairs * _cdiv(int(context_len), 2 * partition_size) >= 0.8 * num_sms:
        partition_size *= 2
    return partition_size


@functools.lru_cache(maxsize=1024)
def size_partitions(base, num_seqs, ctas, max_context_len, num_sms):
    """(workspace partition, finest, coarsest, ctas, parts) of a fa_paged_attention call: how far partitions of `base`
    tokens may grow when max_context_len is an upper bound and lengths differ.  `ctas`: CTAs that a partition of one
    sequence takes; workspace partition 0: one pass does it.

    The workspace partition is the largest at which one sequence still has CTAs enough for the GPU, or until the grid is
    down to 35 CTAs an SM: doubling lengthens the longest partition (1 us per 100 tokens of a CTA by itself) and spares
    half the launches (1 ns each).  Shorter sequences are cut finer on the GPU: into two waves' worth each where there
    are fewer sequences than that; or, where the workspace partition had to stay small but many sequences might fill
    larger ones, by the sum of all lengths (both kernels then read every length: below 1 us).  fp16, head_size 128, us;
    256 tokens each / sized by the bound as if every context had it / this:
      8 kv heads   4 x 1500 under 32768 15 / 20 / 10, 16 x 2048 at most 22 / 27 / 20, 4096 and 63 x 200 35 / 36 / 31,
                   64 x 32768 at most 852 / 642 / 647, 64 x 8192 at most 233 / 189 / 192, 4 x 32768 at most 103 / 74 / 75
      2 kv heads   4 x 1500 under 32768 9.5 / 21 / 10.3, 4096 and 63 x 200 16.5 / 26 / 17.5, 16 x 32768 at most
                   96 / 52 / 55, 32768 and 15 x 1000 44 / 33 / 32, 64 x 32768 at most 253 / 159 / 174"""
    coarsest = base
    while coarsest < 2048:
        coarsest *= 2
    size = base
    while size < coarsest and (ctas * _cdiv(max_context_len, 2 * size) >= 0.8 * num_sms
                               or num_seqs * ctas * _cdiv(max_context_len, size) > 35 * num_sms):
        size *= 2
    if max_context_len <= size:
        return 0, base, coarsest, 0, 1
    pairs = num_seqs * ctas
    by_length = (size < min(coarsest, 4 * base) and num_seqs <= 2048
                 and pairs * _cdiv(max_context_len, 2 * size) >= 0.8 * num_sms)
    if by_length:
        return size, base, coarsest, int(0.8 * num_sms), 0
    return size, base if pairs < 2 * num_sms else size, coarsest, 0, max(1, _cdiv(2 * num_sms, pairs))


def partition_workspace(rows, P, D, device):
    """One allocation for the partial results of `rows` (sequence, query head) rows over P partitions:
    (tensor, address of the outputs (rows, P, D), of the maxima (rows, P), of the sums (rows, P)), all fp32."""
    stats = (rows * P + 63) // 64 * 64
    ws = torch.empty(rows * P * D + 2 * stats, dtype=torch.float32, device=device)
    base = ws.data_ptr()
    part_max = base + rows * P * D * 4
    return ws, base, part_max, part_max + stats * 4


def _plan(num_seqs, num_q_heads, num_kv_heads, kv_block_size, max_context_len, num_splits, num_sms):
    """(partition size, partitions of the workspace, sizing or None) of a call; partition size 0: one pass."""
    # kept for plain numbers only: a tensor hashes by identity, and its value may change
    plan = _kept_plan if type(num_splits) is int else _kept_plan.__wrapped__
    return plan(num_seqs, num_q_heads, num_kv_heads, kv_block_size, max_context_len, num_splits, num_sms)


@functools.lru_cache(maxsize=1024)
def _kept_plan(num_seqs, num_q_heads, num_kv_heads, kv_block_size, max_context_len, num_splits, num_sms):
    free_choice = num_splits == 0
    num_splits, partition_size = plan_partitions(num_seqs, num_kv_heads, kv_block_size, max_context_len, num_splits,
                                                 num_sms)
    sizing = None
    if free_choice and partition_size:
        partition_size, *sizing = size_partitions(
            partition_size, num_seqs, num_kv_heads * _cdiv(num_q_heads // num_kv_heads, 16), max_context_len, num_sms)
    if not partition_size:
        return 0, 0, None
    return partition_size, _cdiv(max_context_len, partition_size), sizing


def attention(query, key_cache, value_cache, context_lens, block_tables, attn_scale,
              max_context_len, num_splits=0):
    """query [num_seqs, kv_heads * group, head]; caches [num_blocks, kv_heads, block, head]
    with identical strides; context_lens [num_seqs] int32; block_tables
    [num_seqs, max_blocks] int32 or int64."""
    if type(max_context_len) is int and max_context_len > 0 and num_splits == 0 and _native.usable(query):
        out = _native_attention(query, key_cache, value_cache, context_lens, block_tables, attn_scale, max_context_len)
        if out is not None:
            return out
    num_seqs, num_q_heads, head_size = query.shape
    num_kv_heads, kv_block_size = key_cache.shape[1], key_cache.shape[2]
    assert key_cache.shape[3] == head_size
    assert num_q_heads % num_kv_heads == 0
    query_group_size = num_q_heads // num_kv_heads
    assert head_size in (16, 32, 64, 128, 256, 512), f"head_size={head_size}"
    assert head_size <= 256, "head_size 512 is not built for B200 yet"
    assert query_group_size == 1 or kv_block_size >= 16, f"kv_block_size={kv_block_size}"
    assert key_cache.stride() == value_cache.stride(), "key and value cache must share strides"
    assert query.is_cuda and query.dtype == key_cache.dtype == value_cache.dtype
    assert block_tables.dtype in (torch.int32, torch.int64)
    for name, t in (("key_cache", key_cache), ("value_cache", value_cache),
                    ("context_lens", context_lens), ("block_tables", block_tables)):
        assert t.device == query.device, f"{name} is on {t.device}, query on {query.device}"

    if context_lens.dtype != torch.int32:
        context_lens = context_lens.to(torch.int32)
    context_lens = context_lens.contiguous()
    if block_tables.stride(-1) != 1:
        block_tables = block_tables.contiguous()
    if query.stride(-1) != 1 or query.data_ptr() % 16 or query.stride(0) % 8 or query.stride(1) % 8:
        query = query.contiguous()
    if key_cache.stride(-1) != 1 or any(s % 8 for s in key_cache.stride()[:-1]):
        key_cache, value_cache = key_cache.contiguous(), value_cache.contiguous()

    with _C.device_guard(query.device):
        partition_size, P, sizing = _plan(num_seqs, num_q_heads, num_kv_heads, kv_block_size, int(max_context_len),
                                          num_splits, _C.sm_count(query.device))
        part_out = part_max = part_sum = 0
        if partition_size:
            assert partition_size >= kv_block_size and partition_size % kv_block_size == 0, \
                f"partition_size={partition_size}, kv_block_size={kv_block_size}"
            assert partition_size % 16 == 0, f"partition_size={partition_size}"
            ws, part_out, part_max, part_sum = partition_workspace(
                num_seqs * num_q_heads, P, head_size, query.device)

        out = torch.empty(query.shape, dtype=query.dtype, device=query.device)
        kb, kh, kt = key_cache.stride()[:3]
        args = _C.PAGED_ARGS.pack(
            _C.dtype_code(query.dtype), num_seqs, num_q_heads, num_kv_heads, head_size, kv_block_size,
            int(max_context_len), 1 if block_tables.dtype == torch.int64 else 0, partition_size, attn_scale,
            query.data_ptr(), query.stride(0), query.stride(1), key_cache.data_ptr(), value_cache.data_ptr(), kb, kh, kt,
            context_lens.data_ptr(), block_tables.data_ptr(), block_tables.stride(0),
            out.data_ptr(), out.stride(0), out.stride(1), part_out, part_max, part_sum, 0)
        stream = _C.raw_stream(query.device)
        if sizing and partition_size:
            _C.check(_C.call("fa_paged_attention")(args, *sizing, stream), "fa_paged_attention")
            return out
        _C.check(_C.call("fa_paged_decode")(args, stream), "fa_paged_decode")
        if partition_size:
            _C.check(_C.call("fa_paged_reduce")(args, stream), "fa_paged_reduce")
    return out


def _native_attention(query, key_cache, value_cache, context_lens, block_tables, attn_scale, max_context_len):
    """The call through native code, or None: partitions and their workspace chosen here, the rest there."""
    if query.dim() != 3 or key_cache.dim() != 4:
        return None
    num_seqs, num_q_heads, head_size = query.shape
    num_kv_heads, kv_block_size = key_cache.shape[1:3]
    if not num_seqs or not num_kv_heads or num_q_heads % num_kv_heads or not kv_block_size or head_size > 256:
        return None
    partition_size, P, sizing = _plan(num_seqs, num_q_heads, num_kv_heads, kv_block_size, max_context_len, 0,
                                      _C.sm_count(query.device))
    part_out = part_max = part_sum = 0
    if partition_size:
        ws, part_out, part_max, part_sum = partition_workspace(num_seqs * num_q_heads, P, head_size, query.device)
    return _native.load().paged(query, key_cache, value_cache, context_lens, block_tables, attn_scale, max_context_len,
                                partition_size, part_out, part_max, part_sum, *(sizing or (0, 0, 0, 0)))


def reshape_and_cache(key, value, key_cache, value_cache, slot_mapping):
    """Writes new tokens into the paged caches `attention` reads.

    key, value: [num_tokens, kv_heads, head]; caches [num_blocks, kv_heads, block, head];
    slot_mapping [num_tokens] integer: token i goes to block slot // block, position slot % block;
    negative slots are skipped.  The reference has no writer (its tests fill the caches with random
    numbers); a serving loop runs this step right before the decode kernel."""
    if _native.usable(key) and _native.load().append(key, value, key_cache, value_cache, slot_mapping):
        return
    num_tokens, num_kv_heads, head_size = key.shape
    assert value.shape == key.shape and key_cache.shape == value_cache.shape
    assert key_cache.shape[1] == num_kv_heads and key_cache.shape[3] == head_size
    assert key.dtype == value.dtype == key_cache.dtype == value_cache.dtype
    assert key_cache.stride() == value_cache.stride(), "key and value cache must share strides"
    assert key_cache.stride(-1) == 1 and all(s % 8 == 0 for s in key_cache.stride()[:-1]), \
        "caches need unit inner stride and 16-byte aligned rows"
    assert slot_mapping.numel() == num_tokens
    assert key.is_cuda, "inputs must be CUDA tensors"
    for name, t in (("value", value), ("key_cache", key_cache), ("value_cache", value_cache),
                    ("slot_mapping", slot_mapping)):
        assert t.device == key.device, f"{name} is on {t.device}, key on {key.device}"
    if key.stride() != value.stride() or key.stride(-1) != 1 or any(s % 8 for s in key.stride()[:-1]) \
            or key.data_ptr() % 16 or value.data_ptr() % 16:
        key, value = key.contiguous(), value.contiguous()
    slots = slot_mapping.to(torch.int64).contiguous()
    kb, kh, kt = key_cache.stride()[:3]
    with _C.device_guard(key.device):
        st = _C.call("fa_paged_cache_append")(
            _C.dtype_code(key.dtype), num_tokens, num_kv_heads, head_size, key_cache.shape[2], key.data_ptr(),
            value.data_ptr(), key.stride(0), key.stride(1), key_cache.data_ptr(), value_cache.data_ptr(), kb, kh, kt,
            slots.data_ptr(), _C.raw_stream(key.device))
    _C.check(st, "fa_paged_cache_append")
