"""A program that resets the device between two deblending calls (after
agd_gpu_release_cache, which gives back the library's blocks): the second call
sets up its kernels and constant tables again and returns what the first did,
in float and in double.  In a process of its own, as the reset ends the
process's context."""
import os
import subprocess
import sys

import pytest

from agdeblend_b200 import build
from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, sys
import numpy as np
import agdeblend_b200 as A
from agdeblend_b200 import synthetic as S

surveys = [S.gather_2d(seed=11, n_shots=64, nt=300, window=(16, 128), n_its=30),
           S.two_volume_3d(seed=43, n_ch=32, n_shots=32, nt=300, window=(16, 16, 128))]

def calls():
    return [np.concatenate([o.ravel() for o in A.deblend(
        sv.volumes, sv.window_shapes, sv.coords, sv.shottimes, sv.channels, sv.trace_types, 1.0,
        10, 0, [d.astype(t) for d in sv.data])]) for sv in surveys for t in (np.float32, np.float64)]

first = calls()
for t in (np.float32, np.float64):
    A.load_library(t).agd_gpu_release_cache()
assert ctypes.CDLL(sys.argv[1]).cudaDeviceReset() == 0
for a, b in zip(first, calls()):
    tol = 1e-5 if a.dtype == np.float32 else 1e-11
    assert np.linalg.norm(a - b) <= tol * np.linalg.norm(a)
"""


def test_deblend_after_a_device_reset():
    rt = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "lib64",
                      "libcudart.so")
    if not os.path.exists(rt):
        pytest.skip("no shared CUDA runtime")
    env = dict(os.environ, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD, rt], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
