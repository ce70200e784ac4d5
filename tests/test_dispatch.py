"""Rules of the dispatch that depend on sizes alone (csrc/dispatch.h), compiled for
the host."""
from __future__ import annotations

import os
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_rules(tmp_path):
    cuda = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
    exe = tmp_path / "dispatch_test"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{cuda / 'include'}", f"-I{ROOT / 'spgemm-hpc-thesis_gb300' / 'csrc'}",
                    str(ROOT / "tests" / "cpp" / "dispatch_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
