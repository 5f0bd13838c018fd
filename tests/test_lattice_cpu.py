"""Facts the sub-sample lattice and the radiological scatter rest on (CPU).

* v / S^3 by a rounded reciprocal and one residual step equals the quotient
  for every float32 significand and S = 1..16 (``div_count``).
* floor(100 t - 5) from the float32 product rounded down equals the float64
  form for t >= 0 (``kernel_index_f32``), also one ulp beside every index's edge.
* The float32 difference of two table entries held as float32 pairs is the
  float64 difference rounded once (``pair_diff``), up to one ulp.
* A sub-sample's float32 cell coordinates, stepped along the lattice, stay
  within ``lattice_centre``'s bound of the reference's (a float32 sample point,
  ray and plane point, float64 in between).
"""
import subprocess

import numpy as np
import pytest

from conehead_gb300.source import Source

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
    """The float32 form, t >= 0: the product rounded down, floored."""
    v = t.astype(np.float64) * 100.0                     # exact
    p = v.astype(F)
    p = np.where(p.astype(np.float64) > v, np.nextafter(p, F(-np.inf)), p)
    return np.minimum(np.abs(np.floor(np.fmin(p, F(6100))).astype(np.int64) - 5), 5995)


def test_kernel_index():
    rng = np.random.default_rng(1)
    edges = (np.arange(0, 6200, dtype=np.float64) / 100.0).astype(F)
    t = np.concatenate([rng.uniform(0, 70, 400000).astype(F), edges, np.nextafter(edges, F(np.inf)),
                        np.nextafter(edges[1:], F(-np.inf)), rng.uniform(0, 3, 1000).astype(F),
                        np.array([0, 1e-45, 1e-30, 1e20, np.inf], dtype=F)])
    ref = np.abs(np.floor(t.astype(np.float64) * 100.0 - 5.0))
    assert np.array_equal(_index_f32(t), np.minimum(ref, 5995).astype(np.int64))


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


@pytest.mark.parametrize("seed", range(12))
def test_projection_bound(seed):
    rng = np.random.default_rng(seed)
    src = Source()
    src.gantry, src.collimator = float(rng.uniform(0, 360)), float(rng.uniform(0, 90))
    n = rng.integers(24, 260, 3)
    sp = rng.choice([0.1, 0.2, 0.25, 0.3, 0.5], 3).astype(F)
    org = (-(n - 1) * sp / 2 + rng.uniform(-8, 8, 3)).astype(F)
    S = int(rng.integers(1, 6))
    pos, vy, m = np.asarray(src.position, float), np.asarray(src.v_y, float), np.asarray(src.transform, float)
    srcf = pos.astype(F).astype(float)
    vyw = (vy[0] * srcf[0] + vy[1] * srcf[1]) + vy[2] * srcf[2]
    # constants of the beam
    corners = np.array([[org[k] + (n[k] - 0.5 if c >> k & 1 else -0.5) * float(sp[k]) for k in range(3)]
                        for c in range(8)])
    P, P1 = np.abs(corners).max(), np.abs(corners).sum(1).max()
    D = np.sqrt(((pos - corners) ** 2).sum(1)).max()
    ray = np.sqrt(3) * P + D + 8 * P1
    err_x = 2.0 ** -24 * (ray + 5 * max(abs(m[0] @ pos), abs(m[2] @ pos)))
    err_n = 2.0 ** -24 * (ray + 5 * abs(vy @ pos))
    h = 1.0001 * sp.astype(float) * (S - 1) / (2 * S)
    lat_n = float(h @ np.abs(vy))
    vyf, m0f, m2f = vy.astype(F), m[0].astype(F), m[2].astype(F)
    K, c0, c2 = F(-vyw) * F(100), F(m[0] @ srcf) * F(100), F(m[2] @ srcf) * F(100)
    vox = np.stack([rng.integers(0, k, 20000) for k in n], axis=1)
    p = (org.astype(float) + sp.astype(float) * vox).astype(F)
    nd = F(vy @ pos) - (vyf[0] * p[:, 0] + vyf[1] * p[:, 1] + vyf[2] * p[:, 2])
    x0 = F(m[0] @ pos) - (m0f[0] * p[:, 0] + m0f[1] * p[:, 1] + m0f[2] * p[:, 2])
    x2 = F(m[2] @ pos) - (m2f[0] * p[:, 0] + m2f[1] * p[:, 1] + m2f[2] * p[:, 2])
    near = np.abs(nd) - F(lat_n)
    ok = near > F(0.2) * abs(F(-vyw))
    mag = np.abs(K) / near
    lat = np.maximum(np.abs(x0 / nd), np.abs(x2 / nd))
    delta = mag * (F(err_x) + (lat + F(0.01)) * F(err_n)) + F(0.002)
    off = sp / F(S)
    i = rng.integers(0, S, (len(p), 3))
    mid = F(0.5) * F(S - 1)
    a, b, c = nd, x0, x2
    for k in range(3):
        r = off[k] * (i[:, k].astype(F) - mid)
        a, b, c = a - vyf[k] * r, b - m0f[k] * r, c - m2f[k] * r
    si = K / a
    u, w = si * b + c0, si * c + c2
    # the reference's arithmetic
    ps = np.stack([(((p[:, k].astype(float) - float(sp[k]) * 0.5) + float(off[k]) * 0.5) + float(off[k]) * i[:, k])
                   .astype(F) for k in range(3)], axis=1)
    rd = (pos - ps.astype(float)).astype(F).astype(float)
    t = -vyw / ((vy[0] * rd[:, 0] + vy[1] * rd[:, 1]) + vy[2] * rd[:, 2])
    pp = (srcf + t[:, None] * rd).astype(F).astype(float)
    ref = [(((m[q][0] * pp[:, 0] + m[q][1] * pp[:, 1]) + m[q][2] * pp[:, 2]).astype(F) * F(100)) for q in (0, 2)]
    on = ok & (np.abs(ref[0]) < 2200) & (np.abs(ref[1]) < 2200)
    assert on.any()
    worst = np.maximum(np.abs(u - ref[0]), np.abs(w - ref[1]))[on] / delta[on]
    assert worst.max() < 0.8, worst.max()        # two more ulp of the fast division stay inside the rest
