"""Runs a piece of Python with the library on the stand-in CUDA runtime of
fake_cudart.cpp (compiled here, preloaded in a process of its own)."""
import os
import shutil
import subprocess
import sys

from conftest import ROOT

PRELUDE = """
import ctypes
import numpy as np
from cuco_gb300 import Box, BoxConfig, _native, ics
from cuco_gb300.engine import MODE_FIXED, MODE_PLAIN
from cuco_gb300.ensemble import Ensemble
lib = _native.load()
fake = ctypes.CDLL(None)
fake.fake_log.restype = ctypes.c_char_p
fake.fake_live.restype = fake.fake_peak.restype = ctypes.c_ulonglong
fake.fake_alloc.restype = ctypes.c_void_p
fake.fake_alloc.argtypes = [ctypes.c_size_t, ctypes.c_int]
def config(n, M, G=None, **more):
    return BoxConfig(n=n, pm_grid=M, cell_grid=G or max(16, M // 4), boxsize=1000.0, mass=1.0, G=ics.G_INTERNAL,
                     softening=300.0 / M, **more)
def log():
    return [l.rsplit(" ", 1) for l in fake.fake_log().decode().splitlines()]
"""


def run(tmp_path, script):
    so = os.path.join(str(tmp_path), "fake_cudart.so")
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I" + include, "-o", so,
                    os.path.join(ROOT, "tests", "fake_cudart.cpp")], check=True)
    from cuco_gb300 import build
    build.build()
    r = subprocess.run([sys.executable, "-c", PRELUDE + script], cwd=ROOT, env={**os.environ, "LD_PRELOAD": so},
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    return r.stdout
