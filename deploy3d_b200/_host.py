"""Loads ``libs/_d3d_host.so`` (csrc/host/dispatch.cpp), the native path of a plugin's ``enqueue``.

The module gets the addresses of the C-ABI entry points from the library that ``_lib`` has loaded, so that the checked
and the tuning builds go through the same path.  There is no interpreted fallback: a missing module is an error.
"""
import ctypes
import importlib.machinery
import importlib.util
import os

from . import _lib

PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "libs", "_d3d_host.so")
_MODULE = None


def module():
    global _MODULE
    if _MODULE is None:
        import torch  # noqa: F401  (its libraries must be in the process before the module is)
        if not os.path.exists(PATH):
            raise RuntimeError("%s is missing: build it with `python -m deploy3d_b200.build`" % PATH)
        loader = importlib.machinery.ExtensionFileLoader("_d3d_host", PATH)
        mod = importlib.util.module_from_spec(importlib.util.spec_from_loader("_d3d_host", loader))
        loader.exec_module(mod)
        mod.set_check(_lib.check)
        _MODULE = mod
    return _MODULE


def _address(name):
    fn = getattr(_lib.lib(), name) if name in _lib.SIGNATURES else None
    return ctypes.cast(fn, ctypes.c_void_p).value if fn is not None else 0


def call(name, prefix):
    """Native enqueue of the plugin `name` whose C-ABI functions start with `prefix`."""
    return module().Call(name, prefix, _address(prefix + "_output_desc"), _address(prefix + "_workspace"),
                         _address(prefix + "_enqueue"))
