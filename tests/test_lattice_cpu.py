"""Facts the sub-sample lattice rests on (CPU).

* v / S^3 by a rounded reciprocal and one residual step equals the quotient
  for every float32 significand and S = 1..16 (``div_count``).
"""
import subprocess

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
