"""The operators' usual calls in one step of native code (csrc/host/ops.cpp): checks, allocations, launches and the
autograd nodes.  Its functions return None for a call that they do not take, which then goes through the Python form of
the operator."""
import importlib.machinery
import importlib.util
import os
import threading

import torch  # noqa: F401  (the extension's libraries are torch's, loaded by this import)

PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "lib", "flagattn_host.so")
_lock = threading.Lock()
_module = None
_backward_mode = 0


def _check_release(module):
    """Raises for an extension built against another torch or Python: its inlined layouts would be silently wrong."""
    from . import build
    if module.built_for != build.host_tag():
        raise RuntimeError("flagattn_host.so was built for %s, this is %s. Run `python -m flagattention_b200.build`."
                           % (module.built_for, build.host_tag()))


def load():
    """The extension module, raising if it has not been built."""
    global _module
    if _module is None:
        with _lock:
            if _module is None:
                if not os.path.exists(PATH):
                    raise RuntimeError("flagattn_host.so is not built (%s). Run `python -m flagattention_b200.build`; "
                                       "there is no fallback path." % PATH)
                loader = importlib.machinery.ExtensionFileLoader("flagattn_host", PATH)
                module = importlib.util.module_from_spec(importlib.util.spec_from_loader("flagattn_host", loader))
                loader.exec_module(module)
                _check_release(module)
                module.set_backward_mode(_backward_mode)
                _module = module
    return _module


def set_backward_mode(code):
    """0 auto, 1 one_pass, 2 two_kernel, as flash.set_backward_mode() selected."""
    global _backward_mode
    with _lock:
        _backward_mode = code
        if _module is not None:
            _module.set_backward_mode(code)


def usable(x):
    """Whether the native form may be asked: a CUDA tensor, outside of a graph that torch.compile traces."""
    return x.is_cuda and not torch.compiler.is_compiling()
