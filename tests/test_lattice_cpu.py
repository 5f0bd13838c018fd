"""Facts the sub-sample lattice and the radiological scatter rest on (CPU).

* v / S^3 by a rounded reciprocal and one residual step equals the quotient
  for every float32 significand and S = 1..16 (``div_count``).
* floor(100 t - 5) from the float32 product and its residual equals the
  float64 form (``kernel_index_f32``), also one ulp beside every index's edge.
* The float32 difference of two table entries held as float32 pairs is the
  float64 difference rounded once (``pair_diff``), up to one ulp.
"""
import subprocess

import numpy as np

F = np.float32

DIV = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
int main() {
  for (int S = 1; S <= 16; ++S) {
    const double n = (double)(S * S * S), inv = 1.0 / n;
    for (unsigned m = 0; m < (1u << 23); ++m) {
      const unsigned bits = 0x3f800000u | m;
      float v;
      std::memcpy(&v, &bits, 4);
      const double q = (double)v * inv, r = std::fma(std::fma(-n, q, (double)v), inv, q);
      if (r != (double)v / n) { std::printf("S %d m %u\n", S, m); return 1; }
    }
  }
  return 0;
}
"""


def test_division_by_the_sample_count(tmp_path):
    src, exe = tmp_path / "div.cpp", tmp_path / "div"
    src.write_text(DIV)
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _index_f32(t):
    with np.errstate(invalid="ignore", over="ignore"):
        p = t * F(100)
        e = (t.astype(np.float64) * 100.0 - p.astype(np.float64)).astype(F)     # what the fused product leaves
        f = np.floor(p + F(2.0 ** -51))
        f = np.where((f == p) & (e < 0), f - F(1), f)
        i = np.fmin(np.abs(f - F(5)), F(5995))
    return np.where(p > F(-9.223372036854775808e18), i, F(0)).astype(np.int64)


def test_kernel_index():
    rng = np.random.default_rng(1)
    edges = (np.arange(0, 6200, dtype=np.float64) / 100.0).astype(F)
    t = np.concatenate([rng.uniform(0, 70, 400000).astype(F), edges, np.nextafter(edges, F(np.inf)),
                        np.nextafter(edges, F(-np.inf)), rng.uniform(-3, 3, 1000).astype(F),
                        np.array([0, -0.0, 1e-30, 1e20, -1e10], dtype=F)])
    ref = np.abs(np.floor(t.astype(np.float64) * 100.0 - 5.0))
    assert np.array_equal(_index_f32(t), np.minimum(ref, 5995).astype(np.int64))
    assert np.array_equal(_index_f32(np.array([np.inf, -np.inf, np.nan], dtype=F)), [5995, 0, 0])


def test_difference_of_pairs(settings):
    from conehead_gb300.kernel import poly_kernel_tables
    K = poly_kernel_tables(settings["energy_weights"])[0]
    rng = np.random.default_rng(2)
    row, a = rng.integers(0, K.shape[0], 200000), rng.integers(0, 5995, 200000)
    b = np.minimum(a + rng.integers(0, 60, a.size), 5995)
    hi = K.astype(F)
    lo = (K - hi.astype(np.float64)).astype(F)
    k1, k0, l1, l0 = hi[row, b], hi[row, a], lo[row, b], lo[row, a]
    d = k1 - k0
    bb = d - k1
    err = (k1 - (d - bb)) - (k0 + bb)
    got = d + (err + (l1 - l0))
    ref = K[row, b] - K[row, a]
    assert np.all(np.abs(got.astype(np.float64) - ref) <= np.spacing(np.abs(ref).astype(F)))
