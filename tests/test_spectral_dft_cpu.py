"""The short DFTs of the cone stage's FFT passes (spectral_dft.cuh), compiled for
the host from the header itself, against numpy's float64 FFT (CPU): every N2 of
SPEC_N2 and the 16-point forms, both directions.
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
BASES = [1, 2]

SOURCE = r"""
#include "spectral_dft.cuh"
using namespace ch;
template <int N>
static int run(float2* x, int inv) {
  float2(&a)[N] = *reinterpret_cast<float2(*)[N]>(x);
  if (inv) Dft<true, N>::run(a); else Dft<false, N>::run(a);
  return 0;
}
extern "C" int dft(int n, int inv, float2* x) {
  switch (n) {
%s
  }
  return 1;
}
extern "C" void dft16_all(int inv, int half, float2* x) {
  float2(&a)[16] = *reinterpret_cast<float2(*)[16]>(x);
  if (half) { if (inv) dft16_half_in<true>(a); else dft16_half_in<false>(a); }
  else { if (inv) dft16<true>(a); else dft16<false>(a); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    d = tmp_path_factory.mktemp("dft")
    src, so = d / "dft.cpp", d / "dft.so"
    src.write_text(SOURCE % "\n".join(f"    case {n}: return run<{n}>(x, inv);" for n in sorted(set(N2S + BASES))))
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(cuda, "include"), "-I", CSRC,
                           str(src), "-o", str(so)])
    L = ctypes.CDLL(str(so))
    for f in (L.dft, L.dft16_all):
        f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    return L


def _input(n, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)


def _expect(x, inv):
    return (np.fft.ifft(x.astype(complex)) * x.size) if inv else np.fft.fft(x.astype(complex))


def _close(got, ref, x):
    # at most four roundings of 2^-24 of the running sums per factor of two, and one of each constant
    bound = 4 * (np.log2(max(x.size, 2)) + 1) * 2.0 ** -24 * np.linalg.norm(x)
    assert np.abs(got - ref).max() <= bound


@pytest.mark.parametrize("n", sorted(set(N2S + BASES)))
@pytest.mark.parametrize("inv", [0, 1])
def test_short_dft(lib, n, inv):
    units = [np.eye(n, dtype=np.complex64)[k] * w for k in range(n) for w in (1, 1j)]
    for x in [_input(n, s) for s in range(20)] + units:
        y = x.copy()
        assert lib.dft(n, inv, y.ctypes.data) == 0
        _close(y, _expect(x, inv), x)


@pytest.mark.parametrize("inv", [0, 1])
@pytest.mark.parametrize("half", [0, 1])
def test_dft16(lib, inv, half):
    m = np.arange(16)
    for x in [_input(16, s) for s in range(50)] + [np.eye(16, dtype=np.complex64)[k] for k in range(16)]:
        if half:
            x[8:] = 0
        y = x.copy()
        lib.dft16_all(inv, half, y.ctypes.data)
        _close(y[4 * (m % 4) + m // 4], _expect(x, inv), x)     # X[m] sits there


def test_lengths():
    """15 lengths from 48 to 512, every one a product of 2, 3 and 5."""
    assert len(N2S) == 15 and N2S == sorted(N2S) and (N2S[0], N2S[-1]) == (3, 32)
    for n in N2S:
        for p in (2, 3, 5):
            while n % p == 0:
                n //= p
        assert n == 1
