"""The native host path (csrc/py/native.cpp): argument checks, allocation and the C ABI call of one
operator in one function.  Built in-tree like the kernel library; there is no Python fallback."""
from __future__ import annotations

import importlib.util
from pathlib import Path

import torch  # noqa: F401  (its libraries must be loaded before the extension)

from . import _lib as L

LIB_PATH = Path(__file__).resolve().parent / "csrc" / "py" / "_native.so"


def _load():
    if not LIB_PATH.exists():
        raise ImportError(
            f"{LIB_PATH} is missing: build it with `python -m flashlight_b200.csrc.build` "
            "(there is no fallback path)")
    spec = importlib.util.spec_from_file_location("_native", LIB_PATH)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    mod.set_check(L.check)
    return mod


native = _load()
