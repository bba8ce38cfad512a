"""Loader of the in-tree native library.

The library is looked for next to the package (``mojodiffusion_b200/_C.so``). On a machine with a GPU a
missing library is an error on first use: the CUDA path is the product, and a silent fall-back to eager
PyTorch there would hide that it is not running. Without a GPU (unit tests on CPU) the pure-torch
references in ``ops.reference`` serve instead.
"""
from __future__ import annotations

import os
import threading
from pathlib import Path

import torch
from torch.autograd import forward_ad

# None where the standard mapping keeps its names in another way: then its ``get`` answers
_Environ = type(os.environ) if isinstance(getattr(os.environ, "_data", None), dict) and hasattr(os.environ, "encodekey") else None
if _Environ is not None:
    _FORCE_REFERENCE, _ONE = os.environ.encodekey("MDB200_FORCE_REFERENCE"), os.environ.encodevalue("1")

_LIB = Path(__file__).resolve().parent.parent / "_C.so"
_lock = threading.Lock()
_loaded = False
_error: str | None = None


def lib_path() -> Path:
    return _LIB


def load(required: bool = False) -> bool:
    """Load ``_C.so`` once. Returns True when ``torch.ops.mdb200`` is usable."""
    global _loaded, _error
    if _loaded:
        return True
    with _lock:
        if _loaded:
            return True
        if not _LIB.exists():
            _error = f"{_LIB} not found: run `python -m mojodiffusion_b200._build`"
        else:
            try:
                torch.ops.load_library(str(_LIB))
                _loaded = True
                _error = None
            except Exception as e:  # pragma: no cover - depends on the machine
                _error = f"loading {_LIB} failed: {e}"
    if not _loaded and required:
        raise RuntimeError(f"mojodiffusion_b200 native kernels unavailable: {_error}")
    return _loaded


def available() -> bool:
    return load(False)


def ops():
    """``torch.ops.mdb200`` (raises if the library cannot be loaded)."""
    if not _loaded:
        load(True)
    return torch.ops.mdb200


def _forced_reference() -> bool:
    """Whether MDB200_FORCE_REFERENCE is 1 in the os.environ of this moment. Every operation asks, so the usual mapping is looked up by
    encoded name: its ``get`` raises and catches an error for an absent name, 2 us (a small SDXL step 23.8 ms, with it 26.2)."""
    env = os.environ
    if type(env) is _Environ:
        return env._data.get(_FORCE_REFERENCE) == _ONE
    return env.get("MDB200_FORCE_REFERENCE") == "1"


def use_native(t: torch.Tensor) -> bool:
    """True when `t` lives on a GPU; the native library is then mandatory."""
    if not t.is_cuda:
        return False
    if _forced_reference():
        return False
    return _loaded or load(True)


def direct(*tensors: torch.Tensor) -> bool:
    """Whether nothing but the kernels looks at an operation on these tensors: plain tensors outside every functorch transform
    (vmap, grad, jvp), forward-mode AD level, dispatch mode and trace. Ops that also have a form in torch operations keep to it
    otherwise."""
    return (all(type(t) is torch.Tensor or type(t) is torch.nn.Parameter for t in tensors)
            and torch._C._functorch.peek_interpreter_stack() is None and forward_ad._current_level < 0
            and torch._C._len_torch_dispatch_stack() == 0 and not torch.jit.is_tracing() and not torch.compiler.is_compiling())


def check_status(like: torch.Tensor | None = None, reset: bool = True) -> None:
    """Raise if any kernel since the last check abandoned a bounded wait (synchronises the device)."""
    if like is None:
        if not torch.cuda.is_available():
            return
        like = torch.empty(0, device="cuda")
    if not like.is_cuda or not available():
        return
    code, where, block, extra = ops().read_status(like, reset)
    if code != 0:
        names = {1: "TIMEOUT", 2: "BAD_ARG", 3: "BOUNDS"}
        raise RuntimeError(
            f"mdb200 kernel reported {names.get(code, code)} (where={where}, block={block}, extra={extra})")
