"""Builds and loads checks.cu: device functions of the library, called on chosen values."""

import ctypes
import subprocess
from pathlib import Path

from cfm_b200 import _native

SOURCE = Path(__file__).resolve().parent / "checks.cu"
LIBRARY = SOURCE.with_name("libdevice_checks.so")

_library = None


def load() -> ctypes.CDLL:
    """The checks, compiled with the library's flags where the sources are newer."""
    global _library
    if _library is None:
        newest = max(p.stat().st_mtime for p in [SOURCE, *_native.HEADERS])
        if not LIBRARY.exists() or LIBRARY.stat().st_mtime < newest:
            subprocess.run([_native.nvcc(), *_native.NVCC_FLAGS, f"-I{_native.PACKAGE / 'csrc'}",
                            "-o", str(LIBRARY), str(SOURCE)], check=True, capture_output=True)
        _library = ctypes.CDLL(str(LIBRARY))
    return _library


def call(name: str, *arguments) -> None:
    """Runs a check to its end; tensors go as their addresses."""
    code = getattr(load(), name)(*(
        ctypes.c_void_p(a.data_ptr()) if hasattr(a, "data_ptr") else ctypes.c_int(a)
        for a in arguments))
    assert code == 0, f"{name}: CUDA error {code}"
