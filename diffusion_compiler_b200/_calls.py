"""The native binding for calls on torch tensors (binding/torch_calls.cpp). There is no fallback: a missing one is an error."""
from __future__ import annotations

import os

from . import _lib

_module = None


def calls():
    global _module
    if _module is None:
        _lib.lib()  # the binding links against it; a missing library says so here
        if not os.path.exists(os.path.join(_lib.HERE, "_torch_calls.so")):
            raise RuntimeError("_torch_calls.so is not built (%s). Run `python -m diffusion_compiler_b200.build`." % _lib.HERE)
        import torch  # noqa: F401  (its libraries first)

        from . import _torch_calls
        _module = _torch_calls
    return _module
