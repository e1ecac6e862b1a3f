"""ctypes bindings of the C ABI declared in `include/dscuda_c_api.h`.

Mirrors the helpers of the reference's `benchmarks/common.py:19-40`
(`library`, `bind`, `checked`): a non-zero status becomes a RuntimeError
carrying `dscuda_<prefix>_last_error()`.
"""

from __future__ import annotations

import ctypes
import functools
import importlib.machinery
import importlib.util
import os
import pathlib
import re
import sys

ROOT = pathlib.Path(__file__).resolve().parents[1]
P, I, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_float

# name -> (argument types, result type); the order is the C declaration order.
MLA_SYMBOLS = {
    "dscuda_mla_last_error": ([], ctypes.c_char_p),
    "dscuda_mla_forward": ([P] * 6 + [I] * 5 + [F, P], I),
    "dscuda_mla_backward": ([P] * 11 + [I] * 5 + [F, P], I),
    "dscuda_mla_workspace_elements": ([I] * 4, ctypes.c_size_t),
    "dscuda_mla_decode": ([P] * 7 + [I] * 7 + [F, P], I),
    "dscuda_mla_decode_checked": ([P] * 7 + [I] * 8 + [F, P], I),
    "dscuda_mla_decode_static_capacity": ([], ctypes.c_size_t),
    "dscuda_mla_decode_static": ([P] * 6 + [I] * 7 + [F, P], I),
    "dscuda_mla_cache_append": ([P] * 6 + [I] * 7 + [P], I),
    "dscuda_mla_cache_append_fp8": ([P] * 6 + [I] * 7 + [P], I),
    "dscuda_mla_cache_dequantize_fp8": ([P] * 2 + [ctypes.c_longlong] * 2 + [P], I),
    "dscuda_mla_rope_apply": ([P] * 3 + [ctypes.c_longlong] + [I] * 3 + [F, P], I),
    "dscuda_mla_prefill_forward": ([P] * 8 + [I] * 7 + [F, P], I),
    "dscuda_mla_prefill_backward_workspace_bytes": ([I] * 4, ctypes.c_size_t),
    "dscuda_mla_prefill_backward_scratch_limit": ([ctypes.c_longlong], ctypes.c_size_t),
    "dscuda_mla_prefill_backward_launches": ([I] * 5, I),
    "dscuda_mla_prefill_backward": ([P] * 14 + [I] * 7 + [F, P], I),
    "dscuda_mla_prefill_backward_sized": ([P] * 14 + [ctypes.c_size_t] + [I] * 7 + [F, P], I),
    "dscuda_mla_up_project": ([P] * 5 + [ctypes.c_longlong, I, P], I),
    "dscuda_mla_absorb_query": ([P] * 3 + [ctypes.c_longlong, I, P], I),
    "dscuda_mla_unabsorb_output": ([P] * 3 + [ctypes.c_longlong, I, P], I),
    "dscuda_mla_device_status": ([I], I),
}
FLASH_SYMBOLS = {
    "dscuda_flash_last_error": ([], ctypes.c_char_p),
    "dscuda_flash_forward": ([P] * 5 + [I] * 5 + [F, P], I),
    "dscuda_flash_device_status": ([I], I),
}


def build_directory() -> pathlib.Path:
    """`build/` at the repository root, or the directory named by DSCUDA_BUILD_DIR."""
    return pathlib.Path(os.environ["DSCUDA_BUILD_DIR"]) if os.environ.get("DSCUDA_BUILD_DIR") else ROOT / "build"


def library_path(name: str) -> pathlib.Path:
    return build_directory() / f"libdscuda_{name}_bench.so"


def _built(path: pathlib.Path) -> pathlib.Path:
    if not path.exists():
        raise RuntimeError(f"{path} is missing: run `python -m dscuda_b200.build` (there is no fallback path)")
    return path


@functools.lru_cache(maxsize=None)
def library(name: str) -> ctypes.CDLL:
    """Load `build/libdscuda_<name>_bench.so` and set every prototype."""
    lib = ctypes.CDLL(str(_built(library_path(name))))
    for symbol, (arguments, result) in (MLA_SYMBOLS if name == "mla" else FLASH_SYMBOLS).items():
        function = getattr(lib, symbol)
        function.argtypes, function.restype = arguments, result
    return lib


@functools.lru_cache(maxsize=None)
def extension():
    """The Python extension over both libraries (`csrc/bindings/torch_bridge.cpp`): torch tensors in, C-ABI calls out.
    It belongs to one torch and one Python; the libraries themselves need neither."""
    import torch  # its shared libraries must be loaded first

    library("mla"), library("flash_attention")
    name = "_dscuda_torch"
    path = str(_built(build_directory() / f"{name}.so"))
    loader = importlib.machinery.ExtensionFileLoader(name, path)
    again = f"run `python -m dscuda_b200.build` with the interpreter that uses it ({sys.executable})"
    try:
        module = importlib.util.module_from_spec(importlib.util.spec_from_file_location(name, path, loader=loader))
        loader.exec_module(module)
    except ImportError as error:
        raise RuntimeError(f"{path} does not load into torch {torch.__version__}: {error}; {again}") from error
    if re.match(r"\d+\.\d+\.\d+", torch.__version__)[0] != module.torch_version:        # pre-release and build suffixes aside
        raise RuntimeError(f"{path} was built for torch {module.torch_version}, this is {torch.__version__}; {again}")
    return module


def checked(lib: ctypes.CDLL, prefix: str, status: int) -> None:
    if status:
        raise RuntimeError(getattr(lib, f"dscuda_{prefix}_last_error")().decode())
