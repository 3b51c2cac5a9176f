"""Host-side mirror of the reference's PackedFunc surface for the dequantize-matmul path.

``get_global_func(name)`` plays the role of ``tvm.get_global_func`` (used by the reference's
tests, e.g. tests/python/contrib/test_cutlass.py:1113,1146): it returns a callable bound to the
library's global registry.  Arguments are torch tensors (passed as DLTensor views, no copy),
ints, floats, strings or None; the call launches on torch's current CUDA stream.
"""
from __future__ import annotations

import ctypes
from typing import Any, Callable, List

import torch

from . import _lib
from ._host import native

_call, _call_like = native.call, native.call_like

class BoundCall:
    """A PackedFunc call with its arguments fixed (``PackedFunc.bind``): for serving loops that pass the
    same buffers on every step.  Calling it launches on torch's current stream of the device the
    tensors are on; the binding keeps the tensors alive."""

    __slots__ = ("_handle", "_args")

    def __init__(self, handle, args):
        self._handle, self._args = handle, args

    def __call__(self):
        _call(self._handle, *self._args)


class PackedFunc:
    """One global function of the registry (what ``TVMFuncGetGlobal`` hands back)."""

    def __init__(self, name: str, handle: int):
        self.name = name
        self.handle = handle

    def bind(self, *args: Any) -> BoundCall:
        """The call with these tensors and scalars, to be repeated."""
        native.check(*args)
        return BoundCall(self.handle, args)

    def __call__(self, *args: Any):
        return _call(self.handle, *args)


def list_global_func_names() -> List[str]:
    lib = _lib.load()
    n = ctypes.c_int()
    arr = ctypes.POINTER(ctypes.c_char_p)()
    _lib.check(lib.RB200FuncListGlobalNames(ctypes.byref(n), ctypes.byref(arr)))
    return [arr[i].decode() for i in range(n.value)]


def _wrap_preprocess(pf: PackedFunc) -> Callable:
    """The reference's ft_preprocess_weight returns a freshly allocated array of the input's
    shape, dtype and device (weight_preprocess.cc:55-57); allocate it here and pass it as the
    destination."""

    def call(packed_weight: torch.Tensor, *rest):
        return _call_like(pf.handle, packed_weight, *rest)

    call.__name__ = pf.name
    return call


_ALLOCATING = {"cutlass.ft_preprocess_weight", "relax_b200.preprocess_weight_q4f16",
               "relax_b200.preprocess_weight_autogptq", "relax_b200.preprocess_weight_gate_up"}
_CACHE = {}


def adopt_managed_tensor(handle: int) -> torch.Tensor:
    """Turns a ``DLManagedTensor*`` returned by a PackedFunc (the allocating form of
    ``cutlass.ft_preprocess_weight``) into a torch tensor without a copy; torch calls the
    tensor's deleter when the last reference goes away."""
    new_capsule = ctypes.pythonapi.PyCapsule_New
    new_capsule.restype = ctypes.py_object
    new_capsule.argtypes = [ctypes.c_void_p, ctypes.c_char_p, ctypes.c_void_p]
    return torch.utils.dlpack.from_dlpack(new_capsule(handle, b"dltensor", None))


def get_global_func(name: str, allow_missing: bool = False, raw: bool = False):
    """``tvm.get_global_func`` counterpart.  Destination-passing operators are returned as is;
    the preprocess functions are wrapped so that they allocate and return their result, like the
    reference's.  ``raw=True`` returns the registered function itself (what a C host gets from
    ``RB200FuncGetGlobal``), without that wrapper."""
    if raw:
        lib = _lib.load()
        h = ctypes.c_void_p()
        _lib.check(lib.RB200FuncGetGlobal(name.encode(), ctypes.byref(h)))
        if not h.value:
            raise ValueError("Cannot find global function %s" % name)
        return PackedFunc(name, h.value)
    hit = _CACHE.get(name)
    if hit is not None:
        return hit
    lib = _lib.load()
    h = ctypes.c_void_p()
    _lib.check(lib.RB200FuncGetGlobal(name.encode(), ctypes.byref(h)))
    if not h.value:
        if allow_missing:
            return None
        raise ValueError("Cannot find global function %s" % name)
    pf = PackedFunc(name, h.value)
    fn = _wrap_preprocess(pf) if name in _ALLOCATING else pf
    _CACHE[name] = fn
    return fn
