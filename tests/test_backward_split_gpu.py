"""Backward calls of a few kv heads with many query heads each: several CTAs share the walk of a key block and leave their
shares of dK and dV in fp32.  Shares that begin inside a query head, empty ones, partial last blocks, dropout and padded
head_dims, against the oracle and the pair of kernels; dk and dv stay bitwise reproducible."""
import pytest
import torch

import flagattention_b200 as fa
import oracle
from flagattention_b200 import _C, _native, flash
from helpers import assert_within_2x, make_qkv

pytestmark = pytest.mark.gpu

SHARED = [
    (1, 8, 1, 1000, 1000, 128, True), (2, 16, 2, 700, 700, 64, True), (1, 24, 1, 300, 420, 128, True),
    (1, 16, 1, 500, 333, 64, False), (1, 32, 2, 257, 129, 128, True), (1, 32, 1, 400, 400, 32, True)]


def _workspace(B, H, Hk, M, N, D, causal):
    """(bytes of the backward's workspace, CTAs that share a walk)"""
    total = _C.call("fa_flash_bwd_workspace_bytes")(_C.pack_shape(torch.float16, B, H, Hk, M, N, D, causal, 0.1))
    up, width = (lambda n: -(-n // 128) * 128), max(D, 64)
    plain = B * H * up(M) * width * 4 + 16 + B * H * M * 4
    return total, max(1, (total - plain) // (2 * B * Hk * up(N) * width * 4))


@pytest.mark.parametrize("B,H,Hk,M,N,D,causal", SHARED)
def test_these_walks_are_shared(B, H, Hk, M, N, D, causal):
    assert _workspace(B, H, Hk, M, N, D, causal)[1] in (2, 4, 8)


@pytest.mark.parametrize("B,H,Hk,M,N,D,split", [
    (1, 4, 2, 4096, 4096, 128, 4),    # the last key block has 2 tiles: 2 of its 4 shares are empty
    (1, 4, 1, 2100, 2100, 64, 8),
    (1, 2, 1, 3000, 3333, 128, 4)])
def test_shares_without_a_tile(B, H, Hk, M, N, D, split):
    """They leave nothing behind, and what is in their memory reaches neither dk nor dv."""
    bytes_, shares = _workspace(B, H, Hk, M, N, D, True)
    blocks = [(-(-M // 128) - max(0, n0 - (N - M)) // 128) * (H // Hk) for n0 in range(0, N, 128)]
    assert shares == split > min(blocks) > 0
    q, k, v, do = make_qkv(B, H, Hk, M, N, D, torch.bfloat16, "cuda", seed=M)
    for x in (q, k, v):
        x.requires_grad_()
    with flash.backward_mode("one_pass"):
        o = fa.flash_attention(q, k, v, True)
        torch.cuda.empty_cache()
        junk = torch.full((bytes_,), 255, dtype=torch.uint8, device="cuda")   # NaN; the workspace comes from this memory
        del junk
        got = torch.autograd.grad(o, (q, k, v), do)
    ref = torch.autograd.grad(oracle.flash_attention(q, k, v, True, upcast=True), (q, k, v), do)
    tor = torch.autograd.grad(oracle.flash_attention(q, k, v, True, upcast=False), (q, k, v), do)
    for name, x, r, t in zip(("dq", "dk", "dv"), got, ref, tor):
        assert_within_2x(x, r, t, name)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,H,Hk,M,N,D,causal", SHARED)
def test_shared_walks(B, H, Hk, M, N, D, causal, dtype):
    q, k, v, do = make_qkv(B, H, Hk, M, N, D, dtype, "cuda", seed=M + N)
    for x in (q, k, v):
        x.requires_grad_()
    run = lambda: torch.autograd.grad(fa.flash_attention(q, k, v, causal), (q, k, v), do)
    with flash.backward_mode("one_pass"):
        got, again = run(), run()
    assert torch.equal(got[1], again[1]) and torch.equal(got[2], again[2])
    ref = torch.autograd.grad(oracle.flash_attention(q, k, v, causal, upcast=True), (q, k, v), do)
    tor = torch.autograd.grad(oracle.flash_attention(q, k, v, causal, upcast=False), (q, k, v), do)
    for name, x, r, t in zip(("dq", "dk", "dv"), got, ref, tor):
        assert_within_2x(x, r, t, name)


def test_shares_use_their_own_workspace_and_their_dropout():
    need = lambda Hk: _C.call("fa_flash_bwd_workspace_bytes")(_C.pack_shape(torch.float16, 1, 16, Hk, 1000, 1000, 64, True, 0.1))
    plain = 16 * 1024 * 64 * 4 + 16 + 16 * 1000 * 4
    assert need(16) == plain and (need(1) - plain) % (2 * 1024 * 64 * 4) == 0 and need(1) > plain
    q, k, v, do = make_qkv(1, 16, 1, 1000, 1000, 64, torch.float16, "cuda", seed=3)
    o, lse = flash._forward(q, k, v, True, 0.125, 0.25, 11, 7)
    got = flash._backward(q, k, v, o, lse, do, True, 0.125, None, 0.25, 11, 7)
    with flash.backward_mode("two_kernel"):
        want = flash._backward(q, k, v, o, lse, do, True, 0.125, None, 0.25, 11, 7)
    for a, b in zip(got, want):   # both round P, dS and the result to 16 bits
        assert (a.float() - b.float()).norm() <= 4 * 2 ** -11 * b.float().norm()


class _memory_left:
    """`with _memory_left(n)`: at most n bytes beside what is allocated."""

    def __init__(self, n):
        self.n = n

    def __enter__(self):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + self.n) / total)

    def __exit__(self, *exc):
        torch.cuda.set_per_process_memory_fraction(1.0)
        return False


@pytest.mark.parametrize("native", [True, False])
def test_walks_are_not_shared_where_memory_is_short(monkeypatch, native):
    B, H, Hk, L, D = 1, 16, 2, 8192, 128
    bytes_, shares = _workspace(B, H, Hk, L, L, D, True)
    least = _C.call("fa_flash_bwd_least_workspace_bytes")(_C.pack_shape(torch.float16, B, H, Hk, L, L, D, True, 0.1))
    assert shares > 1 and bytes_ - least >= 64 << 20
    if not native:
        monkeypatch.setattr(_native, "usable", lambda x: False)
    q, k, v, do = make_qkv(B, H, Hk, L, L, D, torch.bfloat16, "cuda", seed=1)
    for x in (q, k, v):
        x.requires_grad_()
    run = lambda o: torch.autograd.grad(o, (q, k, v), do)
    with flash.backward_mode("one_pass"):
        want = run(fa.flash_attention(q, k, v, True))
        o = fa.flash_attention(q, k, v, True)
        grads = 2 * q.numel() + 4 * k.numel()
        with _memory_left(least + grads + (40 << 20)):   # (the allocator's segments: 20 MB)
            got = run(o)
    for a, b in zip(got, want):   # other sums in fp32, each rounded to 16 bits once
        assert (a.float() - b.float()).norm() <= 2 * 2 ** -8 * b.float().norm()


def test_decisions_are_drawn_again_where_memory_is_short():
    B, H, L, D = 1, 32, 4096, 128
    q, k, v, do = make_qkv(B, H, H, L, L, D, torch.bfloat16, "cuda", seed=2)
    for x in (q, k, v):
        x.requires_grad_()
    kept = _C.call("fa_flash_keep_bits_bytes")(_C.pack_shape(torch.bfloat16, B, H, H, L, L, D, True, 0.1, 0.2))
    assert kept >= 64 << 20
    saved = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: saved.append(t.shape) or t, lambda t: t):
        torch.cuda.manual_seed(4)
        want = torch.autograd.grad(fa.flash_attention(q, k, v, True, dropout_p=0.2), (q, k, v), do)
        with _memory_left(2 * q.numel() + (30 << 20)):
            torch.cuda.manual_seed(4)
            o = fa.flash_attention(q, k, v, True, dropout_p=0.2)
    assert len(saved) == 6 + 5
    got = torch.autograd.grad(o, (q, k, v), do)
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
