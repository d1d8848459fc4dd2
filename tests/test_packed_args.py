"""The packed argument structs of flagattention_b200/_C.py against the ctypes declarations (which tests/test_cabi.py
holds to the header), and the typed calls against the header's parameter lists."""
import os
import re

import pytest
import torch

from flagattention_b200 import _C

HEADER = os.path.join(os.path.dirname(_C.__file__), "..", "include", "flagattn_b200.h")


def test_structs():
    s = _C.FlashShape.from_buffer_copy(_C.pack_shape(torch.bfloat16, 1, 2, 3, 4, 5, 6, True, 0.5, 0.25, 2 ** 63 + 1, 7))
    want = _C.flash_shape(torch.bfloat16, 1, 2, 3, 4, 5, 6, True, 0.5, 0.25, 2 ** 63 + 1, 7)
    assert all(getattr(s, n) == getattr(want, n) for n, _ in s._fields_)
    x = torch.empty(2, 1, 5, 16).transpose(1, 2)
    for t in (x, x[:1], torch.empty(2, 3, 4, 8)[..., ::2]):
        got, want = _C.Tensor4.from_buffer_copy(_C.pack4(t)), _C.tensor4(t)
        assert all(getattr(got, n) == getattr(want, n) for n, _ in got._fields_)
    values = list(range(1, 10)) + [0.5] + list(range(10, 28))
    args = _C.PagedArgs.from_buffer_copy(_C.PAGED_ARGS.pack(*values))
    assert [getattr(args, n) for n, _ in args._fields_] == values


@pytest.mark.parametrize("name", sorted(_C._SIGNATURES))
def test_signatures(name):
    text = re.search(r"\b%s\(([^)]*)\)" % name, open(HEADER).read()).group(1)
    kinds = "".join("p" if "*" in a else "l" if "int64_t" in a else "i" for a in text.split(","))
    assert _C._SIGNATURES[name] == kinds
