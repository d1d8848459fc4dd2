"""The partition rule that the native host code restates, against the Python one; no GPU needed."""
import torch

import flagattention_b200 as fa
from flagattention_b200 import _native, paged


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
