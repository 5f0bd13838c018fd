"""Pairs of float32 in the place of float64 sums and differences, against 80-bit
values (CPU): no further off than the float64 form they stand for.

* pair_diff (stencil.cu): differences of kernel table entries, rounded to float32.
* blocked_fraction (prologue.cu): a voxel's map samples, added in pairs and divided
  once, against the reference's sum of quotients.
* blocked_adjoint_kernel (prologue.cu): shares times counts, added along runs, in
  float32 as the gradient is stored.
"""
import numpy as np
import pytest

from test_adjoint_runs_cpu import _adds

F, L = np.float32, np.longdouble


def _rms(got, ref):
    return float(np.sqrt(np.mean(((got - ref) / np.where(ref == 0, 1, ref)) ** 2)))


@pytest.mark.parametrize("span", [1, 3, 10, 60, 1000])
def test_table_differences(settings, span):
    from conehead_gb300.kernel import poly_kernel_tables
    K = poly_kernel_tables(settings["energy_weights"])[0]
    rng = np.random.default_rng(span)
    row, a = rng.integers(0, K.shape[0], 200000), rng.integers(0, 5990, 200000)
    b = np.minimum(a + rng.integers(1, span + 1, a.size), 5995)
    hi = K.astype(F)
    lo = (K - hi.astype(float)).astype(F)
    k1, k0 = hi[row, b], hi[row, a]
    d = k1 - k0
    bb = d - k1
    got = d + (((k1 - (d - bb)) - (k0 + bb)) + (lo[row, b] - lo[row, a]))
    ref = K[row, b].astype(L) - K[row, a]
    f64 = (K[row, b] - K[row, a]).astype(F)
    # a pair holds 48 bits: a tie of the difference, up to 2^-16 of the entries, is straddled once in 2^8 or less
    assert (got != f64).mean() <= 2.0 ** -8
    assert _rms(got, ref) <= _rms(f64, ref) * (1 + 1e-4)


@pytest.mark.parametrize("S", [2, 3, 5])
def test_map_sums(S):
    rng = np.random.default_rng(S)
    v = rng.random((S ** 3, 100000)).astype(F)
    v[rng.random(v.shape) < 0.3] = 1
    v[rng.random(v.shape) < 0.2] = 0
    n = float(S ** 3)
    hi, lo, ones = (np.zeros(v.shape[1], t) for t in (F, F, np.float64))
    acc, ref = np.zeros(v.shape[1]), np.zeros(v.shape[1], L)
    for x in v:
        acc = acc + x.astype(float) / n
        ref = ref + x
        graded = (x != 0) & (x != 1)
        ones += x == 1
        t = hi + x
        bb = t - hi
        low = lo + ((hi - (t - bb)) + (x - bb))
        hi, lo = np.where(graded, t, hi), np.where(graded, low, lo)
    got = ((hi.astype(float) + lo.astype(float)) + ones) / n
    assert _rms(got, ref / n) <= _rms(acc, ref / n)


def test_adjoint_runs():
    rng = np.random.default_rng(4)
    cols, rows = 6, 5
    same, off = 0, []
    for _ in range(400):
        a, k = np.full(32, rng.integers(0, rows - 1)), np.sort(rng.integers(0, cols - 1, 32))
        cnt = rng.integers(0, 14, (32, 4))
        g = rng.random(32) * 10.0 ** rng.uniform(-3, 0, 32)
        got, f64, ref = np.zeros(rows * cols), np.zeros(rows * cols), np.zeros(rows * cols, L)
        for j, x in _adds(a, k, cnt, g, cols):
            got[j] += x
        for i in range(32):
            for f in range(4):
                j = (a[i] + (f >> 1)) * cols + k[i] + (f & 1)
                f64[j] += g[i] * cnt[i, f]
                ref[j] += L(g[i]) * int(cnt[i, f])
        same += int((got.astype(F) == f64.astype(F)).sum())
        off.append((_rms(got.astype(F), ref), _rms(f64.astype(F), ref)))
    # sums of 32 shares of 47 bits straddle a float32 tie once in 2^18
    assert same >= 400 * rows * cols - 2
    assert np.mean([o[0] for o in off]) <= np.mean([o[1] for o in off]) * (1 + 1e-4)
