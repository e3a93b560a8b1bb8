"""The torch binding ``_C.so`` (csrc/torch_bind.cpp), loaded on first use.  As with the library itself there is no
fallback: where it has not been built, the calls that need it raise."""
from __future__ import annotations

import importlib
import os

_EXT_PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "_C.so")
_ext = None


def ext():
    global _ext
    if _ext is None:
        if not os.path.exists(_EXT_PATH):
            raise RuntimeError(f"{_EXT_PATH} not found: build the CUDA library first (python -m daisy_b200.build); "
                               "daisy_b200 has no CPU or PyTorch fallback")
        _ext = importlib.import_module("daisy_b200._C")
    return _ext
