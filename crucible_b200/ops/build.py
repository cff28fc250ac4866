"""Builds the CUDA sources of `csrc/` into shared libraries, one per source file,
each at its first use.

`nvcc -gencode arch=compute_100a,code=sm_100a -shared` straight to a `.so` that
is loaded with ctypes, whose functions a small extension module then calls (`csrc/host_call.cpp`; ctypes itself
where that module cannot be had); there is no framework header in the kernels, so a file
compiles in seconds.  The library is kept beside the package (`lib/`) under a
name that carries a hash of its sources and flags, so a changed source is
rebuilt and a fresh checkout compiles only what the model at hand needs.  If
the package folder cannot be written, a per-user folder under the system's
temporary directory is used instead.  While a file compiles, a line is printed
to stderr at the start and every few seconds.
"""
from __future__ import annotations

import ctypes
import hashlib
import importlib.machinery
import importlib.util
import os
import platform
import re
import shutil
import subprocess
import sys
import sysconfig
import tempfile
import threading
import time
from typing import Dict, List

_HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(_HERE), "csrc")
_LIB_DIR = os.path.join(os.path.dirname(_HERE), "lib")

UNSUPPORTED = 100001       # `csrc/common.cuh`: an entry does not take this call

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
              "-shared", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]

# Host-only sources (C++, no device code): compiled by the same nvcc call, which hands them
# to the host compiler.
HOST_SOURCES = {"host_step": "host_step.cpp", "host_cache": "host_cache.cpp", "host_call": "host_call.cpp"}
# `host_call` is an extension of the interpreter: without its headers, where it cannot be built or loaded, or on
# another machine than x86-64 Linux, the kernels' entry points are called through ctypes alone.  Its file carries the
# interpreter's own tag (a debug or free-threaded one lays its objects out differently).
PYTHON_INCLUDE = sysconfig.get_paths()["include"]
PYTHON_TAG = sysconfig.get_config_var("SOABI") or sys.implementation.cache_tag or "python"
NATIVE_CALLS = (platform.machine() == "x86_64" and sys.platform.startswith("linux") and sys.implementation.name == "cpython"
                and os.path.exists(os.path.join(PYTHON_INCLUDE, "Python.h")))

# source file -> extra headers whose change must trigger a rebuild
MODULES: Dict[str, List[str]] = {
    "host_step": [],
    "host_cache": [],
    **({"host_call": []} if NATIVE_CALLS else {}),
    "elementwise": ["common.cuh"],
    "gemm_simt": ["common.cuh"],
    "attention_generic": ["common.cuh"],
    "attention_f32": ["common.cuh"],
    "sampling": ["common.cuh", "no_alloc_argmax.h"],
    "streams": ["common.cuh"],
    "sink_attention": ["common.cuh"],
    "recurrent": ["common.cuh"],
    "recurrent_chunks": ["common.cuh", "tc_common.cuh"],
    "polynorm": ["common.cuh"],
    "hashed_embedding": ["common.cuh"],
    "activations": ["common.cuh"],
    "latent_attention": ["common.cuh"],
    "moe": ["common.cuh"],
    "input_conv": ["common.cuh"],
    "differential": ["common.cuh"],
    "layer_close": ["common.cuh"],
}

_loaded: Dict[str, ctypes.CDLL] = {}
_lock = threading.Lock()


class BuildError(RuntimeError):
    pass


def register_module(name: str, headers: List[str]) -> None:
    MODULES[name] = list(headers)


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise BuildError("nvcc was not found (looked at $NVCC, PATH and /usr/local/cuda/bin); "
                     "the CUDA kernels of crucible_b200 cannot be built")


def _digest(name: str) -> str:
    h = hashlib.sha256()
    h.update(" ".join(NVCC_FLAGS).encode())
    if name == "host_call":
        h.update(PYTHON_TAG.encode())
    for fn in [_source(name)] + MODULES[name]:
        with open(os.path.join(CSRC, fn), "rb") as f:
            h.update(fn.encode())
            h.update(f.read())
    return h.hexdigest()[:16]


def _source(name: str) -> str:
    return HOST_SOURCES.get(name, name + ".cu")


def _writable_dir() -> str:
    try:
        os.makedirs(_LIB_DIR, exist_ok=True)
        probe = os.path.join(_LIB_DIR, f".probe-{os.getpid()}")
        with open(probe, "w"):
            pass
        os.remove(probe)
        return _LIB_DIR
    except OSError:
        d = os.path.join(tempfile.gettempdir(), f"crucible_b200-lib-{os.getuid()}")
        os.makedirs(d, exist_ok=True)
        return d


def library_path(name: str) -> str:
    """Path of the built library of module `name`, building it if needed."""
    if name not in MODULES:
        raise BuildError(f"no CUDA module named {name!r}; known: {sorted(MODULES)}")
    stem = f"cb_{name}.{PYTHON_TAG}-" if name == "host_call" else f"cb_{name}-"
    fname = f"{stem}{_digest(name)}.so"
    in_tree = os.path.join(_LIB_DIR, fname)
    if os.path.exists(in_tree):
        return in_tree
    out_dir = _writable_dir()
    target = os.path.join(out_dir, fname)
    if os.path.exists(target):
        return target
    for old in os.listdir(out_dir):
        if old.startswith(stem) and old.endswith(".so"):
            try:
                os.remove(os.path.join(out_dir, old))
            except OSError:
                pass
    tmp = os.path.join(out_dir, f".{fname}.{os.getpid()}.tmp")
    cmd = [_nvcc()] + NVCC_FLAGS + ["-I", CSRC, "-o", tmp, os.path.join(CSRC, _source(name))]
    if name == "host_call":
        cmd += ["-I", PYTHON_INCLUDE]
    print(f"[crucible_b200] compiling {_source(name)} for sm_100a (first use) ...",
          file=sys.stderr, flush=True)
    t0 = time.time()
    env = dict(os.environ)
    env.setdefault("TMPDIR", tempfile.gettempdir())
    proc = subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, env=env)
    out_chunks: List[bytes] = []
    reader = threading.Thread(target=lambda: out_chunks.append(proc.stdout.read()), daemon=True)
    reader.start()
    while True:
        try:
            proc.wait(timeout=5)
            break
        except subprocess.TimeoutExpired:
            print(f"[crucible_b200] ... still compiling {_source(name)} ({time.time() - t0:.0f} s)",
                  file=sys.stderr, flush=True)
    reader.join()
    log = b"".join(out_chunks).decode(errors="replace")
    if proc.returncode != 0:
        try:
            os.remove(tmp)
        except OSError:
            pass
        raise BuildError(f"nvcc failed on {_source(name)}:\n{log}")
    os.replace(tmp, target)
    print(f"[crucible_b200] built {name} in {time.time() - t0:.1f} s", file=sys.stderr, flush=True)
    return target


_C_TYPES = {"int": ctypes.c_int, "long": ctypes.c_long, "long long": ctypes.c_longlong, "float": ctypes.c_float}


def signatures(text: str) -> Dict[str, tuple]:
    """name -> (result, [parameters]) as ctypes, of every entry point that a kernel source exports."""
    out = {}
    text = re.sub(r"//[^\n]*", "", text)
    for result, name, params in re.findall(r"^CB_EXPORT\s+([^(]*?)(\w+)\s*\(([^)]*)\)", text, re.M):
        kinds = []
        for p in params.replace("\n", " ").split(","):
            p = re.sub(r"\bconst\b|\b__restrict__\b", "", p).strip()
            if not p or p == "void":
                continue
            kind = ctypes.c_void_p if "*" in p else _C_TYPES.get(" ".join(p.split()[:-1]))
            if kind is None:
                raise BuildError(f"{name}: parameter {p!r} is of no type that the wrappers pass")
            kinds.append(kind)
        result = result.strip()
        kind = ctypes.c_char_p if "char" in result else None if result == "void" else _C_TYPES.get(result)
        if kind is None and result != "void":
            raise BuildError(f"{name}: result {result!r} is of no type that the wrappers take")
        out[name] = kind, kinds
    return out


_KINDS = {ctypes.c_void_p: "p", ctypes.c_int: "i", ctypes.c_long: "i", ctypes.c_longlong: "i", ctypes.c_float: "f"}


_calls: List[object] = []       # the extension module, or None where it cannot be had; empty: not asked for yet


def _native_calls():
    """The extension module that calls entry points (`csrc/host_call.cpp`), or None."""
    if not NATIVE_CALLS:
        return None
    if not _calls:
        try:
            loader = importlib.machinery.ExtensionFileLoader("cb_host_call", library_path("host_call"))
            module = importlib.util.module_from_spec(importlib.util.spec_from_loader("cb_host_call", loader))
            loader.exec_module(module)
        except (BuildError, ImportError, OSError) as e:
            print(f"[crucible_b200] host_call is not to be had, entry points go through ctypes: {e}",
                  file=sys.stderr, flush=True)
            module = None
        _calls.append(module)
    return _calls[0]


def load(name: str) -> ctypes.CDLL:
    """The library of module `name`.  A kernel source's entry points know their parameters' types, read off
    the source's own declarations, so that the wrappers pass plain numbers and addresses, and those that
    return a status are called without ctypes (`_native_calls`)."""
    lib = _loaded.get(name)
    if lib is not None:
        return lib
    with _lock:
        lib = _loaded.get(name)
        if lib is None:
            lib = ctypes.CDLL(library_path(name))
            if name not in HOST_SOURCES:
                native = _native_calls()
                with open(os.path.join(CSRC, _source(name))) as f:
                    for entry, (result, kinds) in signatures(f.read()).items():
                        fn = getattr(lib, entry)
                        fn.restype, fn.argtypes = result, kinds
                        if native is not None and result is ctypes.c_int:
                            direct = native.wrap(ctypes.cast(fn, ctypes.c_void_p).value, "".join(_KINDS[k] for k in kinds), fn)
                            if direct is not None:
                                setattr(lib, entry, direct)
            _loaded[name] = lib
        return lib


def build_all() -> List[str]:
    """Builds every module; `host_call`, which the others do without, where it can be had."""
    return [library_path(name) for name in sorted(MODULES) if name != "host_call" or _native_calls() is not None]
