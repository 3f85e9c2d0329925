"""Loads the torch extension lib/dk_torch.so (csrc/dk_torch.cpp: argument checks, allocation and the autograd nodes of the
operators in C++) and hands it the entry points of the loaded libdk_b200.so.  No fallback: a missing extension raises."""
import ctypes
import importlib.machinery
import importlib.util
import os

from . import _cabi

_PATH = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lib", "dk_torch.so")

if not os.path.exists(_PATH):
    raise ImportError("dk_torch.so not found at %s: build it with `python deformable-kernels_b200/build.py`" % _PATH)

_loader = importlib.machinery.ExtensionFileLoader("dk_torch", _PATH)
native = importlib.util.module_from_spec(importlib.util.spec_from_loader("dk_torch", _loader))
_loader.exec_module(native)
native.bind({name: ctypes.cast(getattr(_cabi.lib, name), ctypes.c_void_p).value for name in native.entry_points()},
            _cabi.DkError)
