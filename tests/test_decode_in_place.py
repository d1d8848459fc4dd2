"""Dense decoding reads a (batch, kv heads, length, head_dim) tensor as a paged cache without a block table in device
memory: nothing is kept between calls, filled on another call's stream or referred to by a captured graph."""
import ctypes

import pytest
import torch

import flagattention_b200 as fa
from flagattention_b200 import _C, flash


def test_no_device_state_behind_the_call(monkeypatch):
    seen = []
    monkeypatch.setattr(_C, "sm_count", lambda device: 148)
    monkeypatch.setattr(_C, "raw_stream", lambda device: 0)
    monkeypatch.setattr(_C, "call", lambda name: lambda args, stream: seen.append((name, args)) or 0)
    for N in (1024, 65536):
        k = torch.zeros(2, 4, N, 64, dtype=torch.float16)
        flash._decode_forward(torch.zeros(2, 8, 1, 64, dtype=torch.float16), k, k, 1.0)
    assert {name for name, _ in seen} == {"fa_paged_decode", "fa_paged_reduce"}
    for _, packed in seen:
        args = _C.PagedArgs.from_buffer_copy(packed)
        assert args.block_table_is_i64 == _C.FA_BLOCK_TABLE_IN_PLACE
        assert not args.block_tables and not args.context_lens
        assert args.bt_stride_s * 16 == 4 * args.max_context_len   # blocks of 16 keys from one batch element to the next
    held = [n for n, x in vars(flash).items() if isinstance(x, torch.Tensor) or (isinstance(x, dict) and not n.startswith("__"))]
    assert not held


@pytest.mark.parametrize("B,Hk,N,size", [(32, 32, 8192, 4096), (8, 32, 32768, 4096), (2, 16, 131072, 4096), (32, 32, 4096, 0)])
def test_partitions_of_long_contexts(monkeypatch, B, Hk, N, size):
    """At most 4096 keys: longer ones are slower for most shapes that would have three waves of them."""
    seen = []
    monkeypatch.setattr(_C, "sm_count", lambda device: 148)
    monkeypatch.setattr(_C, "raw_stream", lambda device: 0)
    monkeypatch.setattr(_C, "call", lambda name: lambda args, stream: seen.append(args) or 0)
    k = torch.empty(B, Hk, N, 128, dtype=torch.float16, device="meta")
    flash._decode_forward(torch.empty(B, Hk, 1, 128, dtype=torch.float16, device="meta"), k, k, 1.0)
    assert _C.PagedArgs.from_buffer_copy(seen[0]).partition_size == size


def test_a_missing_table_is_refused(built_lib):
    """Before any CUDA call: null tables stay an error unless the caller says that there are none."""
    args = _C.PagedArgs()
    for name in ("query", "key_cache", "value_cache", "out", "context_lens", "block_tables"):
        setattr(args, name, 0x1000)
    for name in ("num_seqs", "num_q_heads", "num_kv_heads", "max_context_len"):
        setattr(args, name, 1)
    args.head_size, args.block_size, args.partition_size = 64, 16, 24      # 24: refused by a later check (-1 too)
    lib = _C.load()
    for kind, table, lens in ((0, 0, 0x1000), (1, 0, 0x1000), (0, 0x1000, 0), (2, 0x1000, 0), (2, 0, 0x1000), (0, 0, 0)):
        args.block_table_is_i64, args.block_tables, args.context_lens, args.head_size = kind, table, lens, 48
        assert lib.fa_paged_decode(ctypes.byref(args), None) == -1
    args.block_table_is_i64, args.block_tables, args.context_lens, args.partition_size = 2, 0, 0, 0
    assert lib.fa_paged_decode(ctypes.byref(args), None) == -2             # accepted; head_size 48 is not built
    args.head_size = 64
    visited = ctypes.c_int64(0)
    assert lib.fa_paged_trace_blocks(ctypes.byref(args), ctypes.byref(visited), 1, None) == -1   # no table to trace


def _through_a_table(q, k, v, causal=False):
    """The same call through paged_attention and the table that the kernel stands in for (M = 1)."""
    B, H, _, D = q.shape
    N = k.shape[2]
    sb, sh, sl, _ = k.stride()
    table, lens = flash._identity_block_table(B, N // 16, sb // (16 * sl), k.device)
    blocks = (B - 1) * (sb // (16 * sl)) + N // 16
    cache = [x.as_strided((blocks, k.shape[1], 16, D), (16 * sl, sh, sl, 1)) for x in (k, v)]
    return fa.paged_attention(q[:, :, 0], *cache, lens, table, D ** -0.5, N, 1).unsqueeze(2)


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["bhld", "blhd", "padded"])
@pytest.mark.parametrize("B,H,Hk,N,D", [(3, 8, 2, 208, 64), (1, 4, 4, 16, 128), (40, 8, 4, 240, 32)])
def test_same_as_through_a_table(B, H, Hk, N, D, layout):
    gen = torch.Generator(device="cuda").manual_seed(N)
    make = lambda *s: torch.randn(s, generator=gen, device="cuda", dtype=torch.bfloat16)
    q = make(B, H, 1, D)
    if layout == "bhld":
        k, v = make(B, Hk, N, D), make(B, Hk, N, D)
    elif layout == "blhd":
        k, v = (make(B, N, Hk, D).transpose(1, 2) for _ in range(2))
    else:   # the filled part of a longer cache
        k, v = (make(B, Hk, N + 64, D)[:, :, :N] for _ in range(2))
    assert torch.equal(fa.flash_attention(q, k, v), _through_a_table(q, k, v))


@pytest.mark.gpu
def test_streams_and_captured_graphs():
    """A first call on a side stream right after another length's, and a replay after many other lengths."""
    make = lambda *s: torch.randn(s, device="cuda", dtype=torch.float16)
    q, k, v = make(2, 8, 1, 64), make(2, 8, 4096, 64), make(2, 8, 4096, 64)
    want = fa.flash_attention(q, k, v)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        out = fa.flash_attention(q, k, v)
    for n in range(16, 16 * 12, 16):
        fa.flash_attention(q, k[:, :, :n], v[:, :, :n])
        junk = torch.full((4096,), -1, dtype=torch.int32, device="cuda")   # memory a freed table would have left
        del junk
    out.zero_()
    graph.replay()
    assert torch.equal(out, want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = fa.flash_attention(q, k[:, :, :2048], v[:, :, :2048])
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(got, fa.flash_attention(q, k[:, :, :2048], v[:, :, :2048]))
