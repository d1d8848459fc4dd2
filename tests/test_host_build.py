"""The host extension is as good as the torch and Python it was compiled for: an older one is built anew and never loaded;
no GPU needed."""
import os

import pytest
import torch

import flagattention_b200 as fa  # noqa: F401
from flagattention_b200 import _native, build


def test_the_extension_names_what_it_was_built_for(built_lib):
    assert _native.load().built_for == build.host_tag() and torch.__version__ in build.host_tag()


def test_another_release_makes_it_stale(built_lib, monkeypatch):
    header = os.path.join(build.INCLUDE, "flagattn_b200.h")
    assert build._host_current(header)
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "2.99.0")
        assert not build._host_current(header)
    with monkeypatch.context() as m:
        m.setattr(build, "HOST_FLAGS", build.HOST_FLAGS + ["-g"])
        assert not build._host_current(header)
    assert build._host_current(header)


def test_another_release_is_not_loaded(built_lib, monkeypatch):
    _native.load()
    monkeypatch.setattr(_native, "_module", None)
    monkeypatch.setattr(torch, "__version__", "2.99.0")
    with pytest.raises(RuntimeError, match="was built for"):
        _native.load()
    assert _native._module is None
