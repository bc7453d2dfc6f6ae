"""Runs host code of the library in a child process on the stand-in runtime (fake_cudart.cpp)."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

_PRELUDE = """
import ctypes as C
import sys
sys.path.insert(0, {root!r})
import numpy as np
from rtc8_gb300 import _lib, nrc
from rtc8_gb300._lib import VptError
from rtc8_gb300.configs import C1, VolumeSpec
from rtc8_gb300.renderer import Renderer, frame_params
fake = C.CDLL(None)
fake.fake_bytes.restype = C.c_size_t
fake.fake_limit.argtypes = [C.c_size_t]
MALLOC, COPY, MEMINFO, LAUNCH, MEMSET = range(5)
def failed(f):
    try:
        f()
    except (VptError, nrc.NrcError) as e:
        return str(e)
    return None
"""


def run(code: str, tmp_path: Path) -> str:
    """Output of `code` (after the prelude above) in a child process on the stand-in runtime."""
    from rtc8_gb300 import build

    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    build.build()
    shim = tmp_path / "libfake_cudart.so"
    include = Path(build.nvcc()).resolve().parent.parent / "include"
    subprocess.run([cxx, "-std=c++17", "-shared", "-fPIC", "-w", "-I", str(include), str(ROOT / "tests" / "fake_cudart.cpp"),
                    "-o", str(shim)], check=True)
    res = subprocess.run([sys.executable, "-c", _PRELUDE.format(root=str(ROOT)) + code], capture_output=True, text=True,
                         env=dict(os.environ, LD_PRELOAD=str(shim)))
    assert res.returncode == 0, res.stdout + res.stderr
    return res.stdout
