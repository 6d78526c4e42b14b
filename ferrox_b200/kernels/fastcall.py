"""Builds and loads ``csrc/py/fastcall.c``, a small extension module that calls the kernel library's entry points without
ctypes (3 us a call of two dozen arguments there, half a microsecond here; a step that is not a replayed graph makes some
sixty).  It needs a C compiler and Python's headers once; without them, or where the module does not load, :func:`bind` returns
None and ctypes takes the calls.
"""
from __future__ import annotations

import hashlib
import importlib.machinery
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
import threading
from ctypes import c_double, c_float, c_int, c_long, c_ulonglong, c_void_p

from .lib import _log, build_dir

_HERE = os.path.dirname(os.path.abspath(__file__))
SOURCE = os.path.normpath(os.path.join(_HERE, "..", "csrc", "py", "fastcall.c"))
NAME = "_fx_fastcall"
FLAGS = ["-O2", "-fPIC", "-shared", "-Wall"]
CODES = {c_void_p: "P", c_int: "I", c_long: "L", c_ulonglong: "U", c_float: "F", c_double: "D"}

_lock = threading.Lock()
_module = None       # None: not looked for yet; False: there is none


def build():
    """The module's path, compiled if need be; None without a compiler or Python's headers."""
    include = sysconfig.get_paths()["include"]
    if not os.path.exists(os.path.join(include, "Python.h")):
        return None
    cc = next((c for c in (os.environ.get("CC"), shutil.which("gcc"), shutil.which("cc"), shutil.which("clang"))
               if c and (os.path.exists(c) or shutil.which(c))), None)
    if cc is None:
        return None
    h = hashlib.sha256(" ".join([*FLAGS, sysconfig.get_config_var("EXT_SUFFIX") or sys.implementation.cache_tag or "",
                                 sysconfig.get_platform()]).encode())
    with open(SOURCE, "rb") as f:
        h.update(f.read())
    path = os.path.join(build_dir(), f"{NAME}.{h.hexdigest()[:16]}.so")
    if not os.path.exists(path):
        tmp = f"{path}.{os.getpid()}.tmp"
        r = subprocess.run([cc, *FLAGS, "-I", include, "-o", tmp, SOURCE], capture_output=True, text=True)
        if r.returncode != 0:
            _log(f"{SOURCE} does not compile, entry points are called by ctypes:\n{r.stderr}")
            return None
        os.replace(tmp, path)
    return path


def module():
    """The extension module, or None where it cannot be built or loaded (a compiler that does not run, a folder that code is not
    loaded from, a file of another system); built and loaded by the first call."""
    global _module
    with _lock:
        if _module is None:
            _module = False
            try:
                path = build()
                if path is not None:
                    loader = importlib.machinery.ExtensionFileLoader(NAME, path)
                    m = importlib.util.module_from_spec(importlib.util.spec_from_file_location(NAME, path, loader=loader))
                    loader.exec_module(m)
                    _module = m
            except (OSError, ImportError) as e:
                _log(f"no extension module, entry points are called by ctypes: {e}")
    return _module or None


def bind(function, argtypes):
    """The ctypes function ``function`` of ``argtypes`` as a callable of the extension module, or None."""
    m = module()
    if m is None or any(t not in CODES for t in argtypes):
        return None
    return m.bind(_address(function), "".join(CODES[t] for t in argtypes))


def _address(function) -> int:
    from ctypes import cast

    return cast(function, c_void_p).value
