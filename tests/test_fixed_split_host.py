"""The histograms' fixed-point split (csrc/wbgpu_fixed.cuh), compiled for the host: floor(v 2^60) exactly in two words for
|v| < 2^67, and the nearest end of the range beyond it."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), '..', 'wannier-berri_gb300', 'csrc')
SOURCE = r"""
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>
using std::isfinite;
static struct { int x; } threadIdx, blockDim;
static long long __double_as_longlong(double v) { long long r; memcpy(&r, &v, 8); return r; }
static unsigned long long atomicAdd(unsigned long long* p, unsigned long long v) { const unsigned long long o = *p; *p += v; return o; }
#include "wbgpu_fixed.cuh"
extern "C" void split(const double* v, long long n, unsigned long long* out) {
  for (long long i = 0; i < n; ++i) fx_split(v[i], out[2 * i], out[2 * i + 1]);
}
"""


def test_split(tmp_path):
    cxx = shutil.which('g++')
    nvcc = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), 'include')
    if cxx is None or not os.path.exists(os.path.join(inc, 'cuda_runtime.h')):
        pytest.skip("needs g++ and the CUDA headers")
    src, so = str(tmp_path / 's.cpp'), str(tmp_path / 's.so')
    with open(src, 'w') as f:
        f.write(SOURCE)
    r = subprocess.run([cxx, '-std=c++17', '-O1', '-w', '-shared', '-fPIC', '-I', inc, '-I', CSRC, src, '-o', so],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rng = np.random.default_rng(0)
    mag = rng.uniform(1.0, 2.0, 4000) * 2.0 ** rng.integers(-140, 120, 4000)
    v = np.r_[mag, -mag, 0.0, -0.0, 5e-324, -5e-324, 2.0 ** -60, -2.0 ** -60, np.nextafter(2.0 ** 67, 0), 2.0 ** 67,
              -2.0 ** 67, np.nextafter(-2.0 ** 67, -np.inf), 1e300, -1e300]
    out = np.zeros((len(v), 2), dtype=np.uint64)
    ctypes.CDLL(so).split(ctypes.c_void_p(v.ctypes.data), ctypes.c_longlong(len(v)), ctypes.c_void_p(out.ctypes.data))
    for x, (lo, hi) in zip(v.tolist(), out.tolist()):
        num, den = x.as_integer_ratio()
        exact = num * 2 ** 60 // den  # floor
        got = (hi - (hi >> 63 << 64)) * 2 ** 64 + lo
        if abs(x) < 2.0 ** 67:
            assert got == exact, x
        else:  # the last word's range, not a wrapped value
            assert got == (2 ** 63 - 1 << 64 if x > 0 else -2 ** 127), x
