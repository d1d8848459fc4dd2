"""The rules that have a cluster of CTAs share the walk of a query tile, at calls whose forms were
measured; no GPU needed."""
import pytest
import torch

from flagattention_b200 import _C, flash


def _split(B, H, M, N, D, causal, dropout=0.0):
    return _C.call("fa_flash_key_split")(_C.pack_shape(torch.float16, B, H, H, M, N, D, causal, 0.1, dropout), 148)


@pytest.mark.parametrize("B,H,M,N,D,causal,best", [
    # more clusters than run at once, or two CTAs of them an SM: slower than fewer CTAs a tile, or than one
    (1, 8, 1152, 1152, 128, True, 2), (1, 12, 672, 672, 64, True, 2), (2, 3, 1536, 1536, 64, False, 2),
    (1, 3, 1536, 1536, 64, False, 4), (2, 3, 668, 1729, 64, False, 4), (2, 8, 1115, 1115, 128, False, 1),
    (1, 8, 1159, 1159, 128, False, 1), (1, 8, 1195, 1195, 128, True, 2), (1, 24, 254, 549, 128, True, 1),
    # what the rule gained from
    (1, 32, 512, 7300, 128, True, 2), (1, 32, 64, 7300, 128, True, 8), (1, 8, 1024, 16384, 128, True, 4),
    (1, 4, 1024, 1024, 128, True, 4), (1, 4, 512, 512, 64, True, 4), (2, 4, 256, 256, 64, True, 1),
    (1, 32, 1024, 4096, 128, True, 1), (1, 4, 8192, 8192, 128, True, 2), (1, 12, 4096, 4096, 128, True, 1),
    (1, 3, 3072, 3170, 128, True, 4), (1, 16, 1052, 1052, 64, True, 2)])
def test_walks_are_shared_where_it_was_faster(built_lib, B, H, M, N, D, causal, best):
    assert _split(B, H, M, N, D, causal) == best


@pytest.mark.parametrize("B,H,M,N,D,causal,pays", [
    # split-KV kernels against clusters, us
    (1, 3, 37, 424, 64, False, 0),      # 6.9, 9.0
    (1, 1, 41, 8859, 64, True, 0),      # 14.8, 19.0
    (8, 2, 91, 424, 64, True, 0),       # 7.4, 9.4
    (1, 32, 33, 389, 64, True, 0),      # 7.4, 9.0
    (1, 1, 222, 921, 64, True, 0),      # 8.1, 9.7
    (2, 16, 44, 497, 32, True, 0),      # 6.7, 7.9
    (1, 4, 46, 9570, 32, True, 0),      # 16.7, 19.2
    (8, 4, 37, 346, 64, True, 0), (1, 4, 32, 1000, 128, True, 0),
    (1, 4, 300, 300, 32, True, 0),      # fewer keys than the tcgen05 kernels take at head_dim 32
    (1, 8, 31, 16384, 128, True, 0),
    (1, 8, 32, 16384, 128, True, 1),    # 43.7, 30.2
    (1, 4, 128, 16384, 128, True, 1),   # 79.8, 31.4
    (1, 16, 64, 4096, 128, True, 1),    # 43.6, 17.4
    (1, 12, 88, 11400, 128, True, 1),   # 109, 24.4
    (1, 16, 57, 3500, 64, True, 1),     # 27.9, 14.1
    (1, 1, 45, 180, 128, True, 1)])     # 8.2, 6.9
def test_few_rows_go_to_the_faster_form(built_lib, B, H, M, N, D, causal, pays):
    assert flash._few_rows_pay(B, H, M, N, D, causal, 148) == bool(pays)
