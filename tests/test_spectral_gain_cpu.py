"""How far the short DFTs' constants, rounded to float32, are off on average
(spectral_dft.cuh with its data in float64, compiled for the host; CPU).

A rounded constant is the same in every butterfly of every transform: its error
is a gain, which a dose passes six times and S^ three, where the roundings of the
data average out.  The 16-point stage, on every axis of every pass, has none; the
N2-point stages stay below 2.2e-8.
"""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "conehead_gb300", "csrc")
LIST = re.search(r"#define SPEC_N2\(X\)(.*)", open(os.path.join(CSRC, "spectral_16n.cuh")).read()).group(1)
N2S = [int(n) for n in re.findall(r"X\((\d+)\)", LIST)]

SOURCE = r"""
#include <cuda_runtime.h>
#include <math.h>
#define float2 double2
#define make_float2 make_double2
#define __builtin_fmaf(k, a, b) fma((double)(k), a, b)
#include "spectral_dft.cuh"
using namespace ch;
template <int N>
static int run(double2* x, int inv) {
  double2(&a)[N] = *reinterpret_cast<double2(*)[N]>(x);
  if (inv) Dft<true, N>::run(a); else Dft<false, N>::run(a);
  return 0;
}
extern "C" int dft(int n, int inv, double2* x) {
  switch (n) {
%s
  }
  return 1;
}
extern "C" void dft16_all(int inv, int half, double2* x) {
  double2(&a)[16] = *reinterpret_cast<double2(*)[16]>(x);
  if (half) { if (inv) dft16_half_in<true>(a); else dft16_half_in<false>(a); }
  else { if (inv) dft16<true>(a); else dft16<false>(a); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    d = tmp_path_factory.mktemp("gain")
    src, so = d / "gain.cpp", d / "gain.so"
    src.write_text(SOURCE % "\n".join(f"    case {n}: return run<{n}>(x, inv);" for n in N2S))
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(cuda, "include"), "-I", CSRC,
                           str(src), "-o", str(so)])
    L = ctypes.CDLL(str(so))
    for f in (L.dft, L.dft16_all):
        f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    return L


def _matrix(n, run):
    A = np.empty((n, n), complex)
    for j in range(n):
        x = np.zeros(n, complex)
        x[j] = 1
        A[:, j] = run(x)
    return A


def _gain(A, inv):
    n = A.shape[1]
    E = np.exp((2j if inv else -2j) * np.pi * np.outer(np.arange(A.shape[0]), np.arange(n)) / A.shape[0])
    assert np.abs(A - E).max() < 1e-7
    return (A * E.conj()).real.mean() - 1


@pytest.mark.parametrize("inv", [0, 1])
def test_sixteen_points_have_no_gain(lib, inv):
    m = np.arange(16)

    def run(x, half=0):
        lib.dft16_all(inv, half, x.ctypes.data)
        return x[4 * (m % 4) + m // 4]
    A = _matrix(16, run)
    H = np.stack([run(np.eye(16, dtype=complex)[j].copy(), 1) for j in range(8)], axis=1)
    assert np.array_equal(H, A[:, :8])
    assert abs(_gain(A, inv)) < 1e-9


@pytest.mark.parametrize("n", N2S)
@pytest.mark.parametrize("inv", [0, 1])
def test_gain_of_the_other_lengths(lib, n, inv):
    def run(x):
        assert lib.dft(n, inv, x.ctypes.data) == 0
        return x
    # a constant's rounding is at most 2^-24 / cos 45 = 8e-8 of it; a length's mean of them
    assert abs(_gain(_matrix(n, run), inv)) < 2.2e-8
