"""Runs a piece of Python with the CUDA runtime replaced by fake_cudart.c, so
that failing allocations and the device memory in use can be tested without a
GPU.  The code runs in a process of its own, with the package and the fake's
functions at hand as ``lib`` (libgame_gb300.so) and ``fake``."""
import os
import subprocess
import sys
import tempfile

import pytest

from game_archived_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))

PRELUDE = """
import ctypes, sys
sys.path[:0] = [{root!r}, {tests!r}]
from game_archived_gb300 import abi, native
from helpers import make_model
fake = ctypes.CDLL({so!r})
fake.fake_fail_malloc.argtypes = [ctypes.c_long, ctypes.c_int]
for f in ("fake_mallocs", "fake_launches", "fake_unordered_clears"):
    getattr(fake, f).restype = ctypes.c_long
fake.fake_live_bytes.restype = ctypes.c_size_t
lib = native.gpu()
error = lambda: lib.game_gpu_last_error().decode()
"""


def run(code):
    if not os.path.exists(build.GPU_LIB):
        pytest.skip("libgame_gb300.so is not built")
    with tempfile.TemporaryDirectory() as d:
        so = os.path.join(d, "fake_cudart.so")
        subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", so, os.path.join(HERE, "fake_cudart.c")], check=True)
        r = subprocess.run([sys.executable, "-c", PRELUDE.format(root=os.path.dirname(HERE), tests=HERE, so=so) + code],
                           env=dict(os.environ, LD_PRELOAD=so), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return r.stdout
