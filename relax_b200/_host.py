"""Loads ``_torch_host.so`` (csrc_host/torch_host.cc): the package's entry points in native code, bound to
the addresses of the library that :mod:`relax_b200._lib` loaded.  There is no fallback."""
from __future__ import annotations

import ctypes
import importlib.util
import os

import torch  # noqa: F401  (its libraries have to be in the process first)

from . import _lib, build

_PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "_torch_host.so")
_SYMBOLS = ("rb200_last_error", "rb200_set_stream", "RB200FuncCall", "RB200FuncGetGlobal", "rb200_encode_ft",
            "rb200_moe_route", "rb200_moe_route_workspace_bytes", "rb200_moe_gather", "rb200_moe_combine")


def check_abi(built_for, here):
    if built_for != here:
        raise RuntimeError("relax_b200: _torch_host.so was built for %s, this is %s - rebuild it with "
                           "`python relax_b200/build.py`" % (built_for, here))


def _load():
    if not os.path.exists(_PATH):
        raise RuntimeError("relax_b200: %s is missing - build it with `python relax_b200/build.py`; there is no "
                           "fallback path" % _PATH)
    spec = importlib.util.spec_from_file_location("_torch_host", _PATH)
    mod = importlib.util.module_from_spec(spec)
    try:
        spec.loader.exec_module(mod)
    except ImportError as e:
        raise RuntimeError("relax_b200: %s does not load beside %s - rebuild it with `python relax_b200/build.py`"
                           % (_PATH, build.host_abi())) from e
    check_abi(mod.built_for, build.host_abi())
    lib = _lib.load()
    mod.init(_lib.RB200Error, {s: ctypes.cast(getattr(lib, s), ctypes.c_void_p).value for s in _SYMBOLS})
    return mod


native = _load()
