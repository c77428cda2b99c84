"""The QL sweep with a warp per matrix (csrc/wbgpu_eigh_ql.cuh), compiled for the host with its 32 lanes as
coroutines: between two warp barriers or votes any of them may be ahead of the others, as on a GPU, and the result must
not depend on which."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), '..', 'wannier-berri_gb300', 'csrc')

HARNESS = r"""
#include <cuda_runtime.h>
#include <math.h>
#include <type_traits>
#include <ucontext.h>
#include <string.h>
#include <vector>
// what the kernel takes from the device: index variables, warp barrier and votes, named roundings
static struct { int x; } threadIdx, blockIdx, blockDim;
static int lane_now;
static ucontext_t host_ctx, lane_ctx[32];
static bool done[32], waiting[32];
static unsigned votes, rnd;
static unsigned next_rnd() { return (rnd = rnd * 1664525u + 1013904223u) >> 8; }
static void yield_lane() {
  const int me = lane_now;
  swapcontext(&lane_ctx[me], &host_ctx);
  lane_now = me;
  threadIdx.x = me;
}
static void warp_barrier() {
  waiting[lane_now] = true;
  yield_lane();
}
static void preempt() {  // between any two operations another lane may go on
  if (next_rnd() % 16 == 0) yield_lane();
}
static void __syncwarp() { warp_barrier(); }
static unsigned __ballot_sync(unsigned, int p) {
  warp_barrier();  // every lane has read the previous vote
  votes &= ~(1u << lane_now);
  if (p) votes |= 1u << lane_now;
  warp_barrier();
  return votes;
}
static int __any_sync(unsigned m, int p) { return __ballot_sync(m, p) != 0; }
template <typename T> T __shfl_xor_sync(unsigned, T v, int) { return v; }  // named by a helper the sweep does not call
static int __ffs(unsigned v) { return __builtin_ffs((int)v); }
static int atomicOr(int* p, int v) { const int o = *p; *p |= v; return o; }
static double __dmul_rn(double a, double b) { preempt(); return a * b; }
static double __fma_rn(double a, double b, double c) { preempt(); return fma(a, b, c); }
static float lane_fmaf(float a, float b, float c) { preempt(); return fmaf(a, b, c); }
#define fmaf lane_fmaf
static double rsqrt(double q) { return 1.0 / sqrt(q); }
#include "wbgpu_common.cuh"
#include "wbgpu_df64.cuh"
static unsigned char smq[1 << 16] __attribute__((aligned(16)));
#undef __shared__
#define __shared__
#undef __launch_bounds__
#define __launch_bounds__(...)
#include "wbgpu_eigh_ql.cuh"

static const double *g_d, *g_e;
static int g_n, g_flag, g_serial;
static double* g_out;
template <typename R> void body() {
  std::vector<R>* v = new std::vector<R>[2];
  for (int i = 0; i < g_n; ++i) { v[0].push_back(Arith<R>::from(g_d[i])); v[1].push_back(Arith<R>::from(g_e[i])); }
  if (g_serial) eigh_ql<R>(v[0].data(), v[1].data(), g_n, 1, g_out, &g_flag);
  else eigh_ql_warp<R>(v[0].data(), v[1].data(), g_n, 1, g_out, &g_flag);
  delete[] v;
}
static int g_df;
static void entry() {
  const int me = lane_now;
  threadIdx.x = me;
  if (g_df) body<df64>(); else body<double>();
  done[me] = true;
  swapcontext(&lane_ctx[me], &host_ctx);
}
extern "C" int sweep(const double* d, const double* e, int n, int df, unsigned seed, double* out) {
  // seed 0: eigh_ql, one thread
  static char stacks[32][1 << 16];
  g_d = d; g_e = e; g_n = n; g_df = df; g_out = out; g_flag = 0; g_serial = seed == 0;
  blockDim.x = 1;
  memset(smq, 0x7f, sizeof smq);
  rnd = seed;
  for (int l = 0; l < 32; ++l) {
    waiting[l] = false;
    done[l] = g_serial && l > 0;
    getcontext(&lane_ctx[l]);
    lane_ctx[l].uc_stack.ss_sp = stacks[l];
    lane_ctx[l].uc_stack.ss_size = sizeof stacks[l];
    lane_ctx[l].uc_link = 0;
    makecontext(&lane_ctx[l], entry, 0);
  }
  while (true) {
    int run[32], n_run = 0;
    bool live = false;
    for (int l = 0; l < 32; ++l) {
      live |= !done[l];
      if (!done[l] && !waiting[l]) run[n_run++] = l;
    }
    if (!live) break;
    if (n_run == 0) {  // every lane has come to the barrier
      for (int l = 0; l < 32; ++l) waiting[l] = false;
      continue;
    }
    lane_now = run[next_rnd() % n_run];
    threadIdx.x = lane_now;
    swapcontext(&host_ctx, &lane_ctx[lane_now]);
  }
  return g_flag;
}
"""


@pytest.fixture(scope='module')
def lib(tmp_path_factory):
    cxx = shutil.which('g++')
    nvcc = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), 'include')
    if cxx is None or not os.path.exists(os.path.join(inc, 'cuda_runtime.h')):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp('ql')
    src, so = str(d / 'ql.cpp'), str(d / 'ql.so')
    with open(src, 'w') as f:
        f.write(HARNESS)
    r = subprocess.run([cxx, '-std=c++17', '-O1', '-w', '-ffp-contract=off', '-shared', '-fPIC', '-I', inc, '-I', CSRC, src, '-o',
                        so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(so)
    lib.sweep.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_uint, ctypes.c_void_p]
    return lib


def _matrices():
    rng = np.random.default_rng(5)
    for n in (1, 2, 3, 8, 31, 32, 33, 47, 96):
        yield f'random {n}', rng.standard_normal(n), rng.standard_normal(n)
    yield 'diagonal', np.arange(40.0) % 7 - 3.0, np.zeros(40)
    e = rng.standard_normal(40)
    e[[4, 5, 20, 33]] = 0.0
    yield 'decoupled', rng.standard_normal(40), e
    # rotations whose f^2 + g^2 underflows to zero (a zero pivot)
    yield 'zero pivot', np.zeros(6), np.full(6, 1e-170)
    yield 'zero pivots and others', np.r_[rng.standard_normal(5), np.zeros(6)], np.r_[rng.standard_normal(5), np.full(6, 1e-25)]


@pytest.mark.parametrize("df", [0, 1])
def test_result_does_not_depend_on_the_order_of_the_lanes(lib, df):
    """The same bits and convergence flag in every order, and as the sweep with a thread per matrix; eigenvalues
    within 4 n eps |T| of LAPACK's (eps 2^-53 / 2^-46)."""
    for name, d, e in _matrices():
        n = len(d)
        run = lambda seed, out: lib.sweep(d.ctypes.data, e.ctypes.data, n, df, seed, out.ctypes.data)
        one, out = np.empty(n), np.empty(n)
        flag = run(0, one)
        for s in range(1, 5):
            out[:] = np.nan
            assert run(977 * s + n, out) == flag, name
            assert np.array_equal(out, one), name
        if 'zero' not in name:
            assert flag == 0, name
            ref = np.linalg.eigvalsh(np.diag(d) + np.diag(e[:n - 1], 1) + np.diag(e[:n - 1], -1))
            assert np.abs(one - ref).max() <= 4 * n * (2.0 ** -46 if df else 2.0 ** -53) * np.abs(ref).max(), name
