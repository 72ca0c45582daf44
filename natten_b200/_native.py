"""The native front of the operators (csrc/torch_binding.cpp): eager calls on plain CUDA tensors go
from here straight to the kernels. Every function returns None for a call it does not take - wrong
arguments included, so that the Python checks report them - and the caller continues in Python.

Like the C library itself it is required: importing this module raises when it is not built."""
import importlib.util
import os

import torch  # noqa: F401  (its libraries have to be loaded first)

from . import _lib

_PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "lib", "torch_binding.so")


def _load():
    if not os.path.exists(_PATH):
        raise ImportError(f"{_PATH} is missing. Build it with `python natten_b200/build.py`.")
    spec = importlib.util.spec_from_file_location("torch_binding", _PATH)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    module.init(_lib.LIB_PATH)
    _lib.native_launches = module.launches
    return module


_module = _load()
na, attention, layer, tiles = _module.na, _module.attention, _module.layer, _module.tiles
