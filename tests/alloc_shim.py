"""Runs a function of a test module in a process whose device allocations pass
through tests/cpp/alloc_shim.cpp, and returns what it returns (JSON)."""
from __future__ import annotations

import json
import os
import subprocess
import sys
from pathlib import Path

HERE = Path(__file__).resolve().parent
ROOT = HERE.parent
PKG = ROOT / "spgemm-hpc-thesis_gb300"


class Shim:
    """The shim as loaded in the child process."""

    def __init__(self, path: str):
        import ctypes
        self._c = ctypes
        self.lib = ctypes.CDLL(path, mode=ctypes.RTLD_GLOBAL)
        self.lib.shim_size.restype = ctypes.c_longlong
        self.lib.shim_size.argtypes = [ctypes.c_void_p]
        self.lib.shim_start.argtypes = [ctypes.c_longlong, ctypes.c_longlong]

    def start(self, fail_from: int = 0, fail_count: int = 0) -> None:
        self.lib.shim_start(fail_from, fail_count)

    def limit(self, more: int = -1) -> None:
        self.lib.shim_limit(self._c.c_longlong(more))

    def slow(self, from_bytes: int, ms: int) -> None:
        self.lib.shim_slow(self._c.c_longlong(from_bytes), self._c.c_longlong(ms))

    def stats(self) -> dict:
        out = (self._c.c_longlong * 5)()
        self.lib.shim_stats(out)
        return dict(zip(("calls", "failed", "held", "peak", "total"), out))

    def size(self, pointer: int) -> int:
        return self.lib.shim_size(pointer)


def build(folder) -> str:
    so = Path(folder) / "alloc_shim.so"
    cuda = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{cuda / 'include'}",
                    str(HERE / "cpp" / "alloc_shim.cpp"), "-o", str(so), "-Wl,--no-as-needed", f"-L{cuda / 'lib64'}", "-lcudart", "-ldl"],
                   check=True)
    return str(so)


def run(folder, module: str, function: str, *args, timeout: float = 300):
    """module.function(shim, *args) in a child process."""
    code = (f"import sys, json; sys.path[:0] = {[str(ROOT), str(PKG), str(HERE)]!r}; import alloc_shim; "
            f"shim = alloc_shim.Shim({build(folder)!r}); import importlib; "
            f"out = getattr(importlib.import_module({module!r}), {function!r})(shim, *json.loads(sys.argv[1])); "
            "print('\\n' + json.dumps(out))")
    r = subprocess.run([sys.executable, "-c", code, json.dumps(args)], capture_output=True, text=True, timeout=timeout)
    assert r.returncode == 0, r.stderr[-4000:]
    return json.loads(r.stdout.strip().splitlines()[-1])
