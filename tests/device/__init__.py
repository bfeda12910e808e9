"""Builds and loads checks.cu, rules.cpp and impatient.cu: parts of the library, called on chosen values."""

import ctypes
import subprocess
from functools import cache
from pathlib import Path

from cfm_b200 import _native

HERE = Path(__file__).resolve().parent
INCLUDES = [f"-I{_native.PACKAGE / 'csrc'}", f"-I{_native.PACKAGE.parent / 'include'}"]


@cache
def _load(source: str, *compiler: str) -> ctypes.CDLL:
    """The source as a library, compiled again where it or a header is newer."""
    path = HERE / source
    library = path.with_name(f"lib{path.stem}.so")
    newest = max(p.stat().st_mtime for p in [path, *_native.HEADERS, *_native.SOURCES])
    if not library.exists() or library.stat().st_mtime < newest:
        subprocess.run([*compiler, *INCLUDES, "-o", str(library), str(path)], check=True, capture_output=True)
    return ctypes.CDLL(str(library))


def call(name: str, *arguments) -> None:
    """Runs a check of checks.cu to its end; tensors go as their addresses."""
    library = _load("checks.cu", _native.nvcc(), *_native.NVCC_FLAGS)
    code = getattr(library, name)(*(
        ctypes.c_void_p(a.data_ptr()) if hasattr(a, "data_ptr") else ctypes.c_int(a)
        for a in arguments))
    assert code == 0, f"{name}: CUDA error {code}"


def impatient_screen():
    """`cfm_screen` of a library whose waits run out within microseconds."""
    function = _load("impatient.cu", _native.nvcc(), *_native.NVCC_FLAGS).cfm_screen
    function.restype, function.argtypes = _native.load().cfm_screen.restype, _native.load().cfm_screen.argtypes
    return function


def dispatch(tokens: int, **sizes: int) -> dict[str, int]:
    """What the library takes for a call: `sizes` are fields of cfm_layer."""
    layer = _native.Layer(**sizes)
    out = (ctypes.c_int32 * 5)()
    _load("rules.cpp", "g++", "-O1", "-std=c++17", "-shared", "-fPIC").dispatch(
        ctypes.byref(layer), ctypes.c_int(tokens), out)
    return dict(zip(("tcgen05", "pass_pairs", "by_pair", "shares_encoder", "by_union"), out))
