"""Loader of the native host path (torch_shim/kda_host.cpp, part of lib/libkda_b200_torch.so).

One pybind call per operator: checks, allocations, launches and the autograd node are made in C++.  Every function
returns None, with nothing done, when its inputs are not the plain valid case; the callers then run their Python checks,
which raise with the reason.
"""

from __future__ import annotations

import importlib.machinery
import importlib.util

from . import _lib, build

_mod = None


def load():
    global _mod
    if _mod is None:
        _lib.load()
        name = "libkda_b200_torch"
        loader = importlib.machinery.ExtensionFileLoader(name, build.build_torch_ops())
        spec = importlib.util.spec_from_file_location(name, loader.path, loader=loader)
        mod = importlib.util.module_from_spec(spec)
        loader.exec_module(mod)
        _mod = mod
    return _mod
