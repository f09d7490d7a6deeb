"""Distances and phases of the FP64 integrands (csrc/phase.cuh): the square root
by Newton's step against CUDA's sqrt, the series of sine and cosine against
extended precision."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
N = 1 << 20


@pytest.fixture(scope="module")
def phase(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("phase") / "phase_check.so")
    csrc = os.path.join(ROOT, "3d_bem_gb300", "csrc")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    nvcc = os.path.join(cuda, "bin", "nvcc")
    cmd = [nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared",
           "-Xcompiler", "-fPIC", "-I", csrc, os.path.join(ROOT, "tests", "cpp", "phase_check.cu"),
           "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ct.CDLL(out)


def _call(f, x, *more):
    a, b = np.full_like(x, np.nan), np.full_like(x, np.nan)
    ptr = [v.ctypes.data_as(ct.c_void_p) for v in (x, a, b)]
    assert f(*ptr, x.size, *more) == 0
    return a, b


def test_newton_square_root(phase):
    """The step leaves 1e-31 beside its rounding, so it is the rounded root (as
    CUDA's sqrt is) unless that lies within 1e-31 of a tie: 1e-15 of all values."""
    rng = np.random.default_rng(1)
    x = np.exp(rng.uniform(np.log(1e-24), np.log(1e24), N))
    x[:1000] = np.arange(1, 1001) ** 2.0  # squares, and their neighbours
    x[1000:2000] = np.nextafter(x[:1000], 0.0)
    x[2000:3000] = np.nextafter(x[:1000], np.inf)
    root, ref = _call(phase.phase_roots, x)
    assert np.array_equal(root, ref)
    assert np.array_equal(root[:1000], np.arange(1, 1001.0))


@pytest.mark.parametrize("most,wide", [(0.35, 0), (1.0, 1)])
def test_series_of_small_phases(phase, most, wide):
    """Within the declared range: half an ulp of the result (1.1e-16), as much again
    for the rounding of the series behind the first term, and the terms left out
    (1e-17)."""
    rng = np.random.default_rng(2)
    x = rng.uniform(-most, most, N)
    x[:3] = (-most, 0.0, most)
    s, c = _call(phase.phase_sincos, x, wide)
    w = x.astype(np.longdouble)
    assert np.abs(s - np.sin(w)).max() < 2.4e-16
    assert np.abs(c - np.cos(w)).max() < 2.4e-16
    assert s[1] == 0.0 and c[1] == 1.0
