"""The rules that the native host code restates, against the Python ones; no GPU needed."""
import itertools

import pytest
import torch

import flagattention_b200 as fa
from flagattention_b200 import _C, _native, flash, paged


def test_partition_growth_is_the_same_rule(built_lib):
    n = _native.load()
    for pairs in (1, 3, 16, 32, 100, 1024):
        for context in (1, 255, 256, 1000, 8192, 131072, 1 << 20):
            for sms in (108, 148):
                assert n.coarsen_partition(256, pairs, context, sms, 4096) == \
                    paged.coarsen_partition(256, pairs, context, sms, 4096)


def test_tensors_elsewhere_are_not_taken(built_lib):
    n, x = _native.load(), torch.zeros(1, 2, 16, 64, dtype=torch.float16)
    assert n.flash(x, x, x, True, None) is None and n.piecewise(x, x, x, x, x, 1, True, None) is None
    assert n.rotary_pair(x, x[0, 0].float(), x, x, x, False) is None and n.append(x, x, x, x, x) is False
    assert n.paged(x, x, x, x, x, 1.0, 1, 0, 0, 0, 0, 0, 0, 0, 0) is None
    assert not _native.usable(x)


def _views(B, H, L, D):
    """The forms a (B, H, L, D) operand comes in: orders, gaps, offsets, broadcasts, inner strides."""
    new = lambda *s: torch.zeros(s, dtype=torch.float16)
    yield new(B, H, L, D)
    yield new(B, L, H, D).transpose(1, 2)
    yield new(H, B, L, D).transpose(0, 1)
    yield new(L, B, H, D).permute(1, 2, 0, 3)
    yield new(B, H, D, L).transpose(2, 3)
    yield new(B, H, L, 2 * D)[..., ::2]
    for pad in (1, 4, 8):
        yield new(B, H, L, D + pad)[..., :D]
        yield new(B, H, L + pad, D)[:, :, pad:]
    yield new(B * H * L * D + 4)[4:].view(B, H, L, D)     # not 16-byte aligned
    yield new(B * H * L * D + 8)[8:].view(B, H, L, D)
    yield new(1, 1, 1, D).expand(B, H, L, D)
    yield new(B, 1, L, D).expand(B, H, L, D)
    yield new(B, H, L, 3 * D).chunk(3, -1)[1]


@pytest.mark.parametrize("B,H,L,D", [(2, 4, 32, 64), (1, 4, 32, 16), (2, 1, 48, 32), (1, 1, 1, 128), (3, 2, 17, 64)])
def test_layouts_are_told_apart_alike(built_lib, B, H, L, D):
    n = _native.load()
    for x in _views(B, H, L, D):
        # (a contiguous tensor off the alignment: neither form can help it by a copy, the library refuses it)
        ready = _C.kernel_ready(x) is x and x.data_ptr() % 16 == 0
        assert n.kernel_ready(x) == ready, (x.shape, x.stride(), x.storage_offset())


@pytest.mark.parametrize("B,Hk,N,D", [(2, 2, 32, 64), (1, 1, 48, 32), (2, 4, 16, 128), (1, 2, 17, 64), (3, 1, 16, 16)])
def test_decode_rule_is_the_same(built_lib, B, Hk, N, D):
    n = _native.load()
    for k, v in itertools.product(_views(B, Hk, N, D), repeat=2):
        if k.stride() != v.stride() and k.is_contiguous():
            continue
        for group, M, causal in itertools.product((1, 4, 64), (1, 2, 16, 20), (False, True)):
            q = torch.zeros(B, Hk * group, M, D, dtype=torch.float16)
            assert n.decode_covered(q, k, v, causal) == flash._decode_covered(q, k, v, causal)
