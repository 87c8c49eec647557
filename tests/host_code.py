"""Compile the library's plain C++ headers (iane_gb300/csrc/*.h) for the host, so that a CPU test
runs the kernels' and launchers' own rules rather than a copy of them."""
from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def compile_host(tmp_path, source: str) -> ctypes.CDLL:
    cxx = shutil.which("g++") or shutil.which("c++")
    assert cxx, "no host C++ compiler"
    src, out = tmp_path / "host.cpp", tmp_path / "libhost.so"
    src.write_text(source)
    cmd = [cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", str(ROOT / "iane_gb300" / "csrc"),
           str(src), "-o", str(out)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    return ctypes.CDLL(str(out))
