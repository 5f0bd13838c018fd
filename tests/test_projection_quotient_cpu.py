"""The projection in pairs of float32 with an approximate quotient, at right
angles too (prologue.cu, project_pairs; CPU).

The kernel divides by __fdividef, off by up to two units in the last place; the
correction q2 takes that back.  Entries of 6e-17 and 4e-33, the sines of right
angles and their products, are part of the transform as they are.
"""
import numpy as np
import pytest

from test_projection_pairs_cpu import D, L, _dot, _fma, _mirror, _split, _two_sum, f


def _pairs(src, vy, m0, m2, rd, ulps):
    vyw = D(f(src[0])) * vy[0] + D(f(src[1])) * vy[1] + D(f(src[2])) * vy[2]
    wh, wl = _split(vyw)
    dh, dl = _dot(vy, rd)
    h = dh + dl
    lo = (dh - h) + dl
    q1 = (-wh / h) * (f(1) + f(ulps) * f(2.0 ** -23))
    q2 = ((_fma(-q1, lo, _fma(-q1, h, np.broadcast_to(-wh, h.shape))) - wl) / h) * (f(1) - f(ulps) * f(2.0 ** -23))
    pp = []
    for k in range(3):
        m = q1 * rd[k]
        e = _fma(q2, rd[k], _fma(q1, rd[k], -m))
        s, se = _two_sum(np.broadcast_to(f(src[k]), m.shape), m)
        pp.append(s + (se + e))
    return [a + b for a, b in (_dot(m0, pp), _dot(m2, pp))]


@pytest.mark.parametrize("gantry,collimator", [(g, c) for g in (0.0, 90.0, 180.0, 270.0) for c in (0.0, 90.0, 180.0)] +
                         [(1e-3, 0.0), (44.9, 12.0), (301.7, 270.0)])
def test_pairs_at_any_angle(gantry, collimator):
    from conehead_gb300 import Source
    s = Source()
    s.gantry, s.collimator = gantry, collimator
    src, vy = np.asarray(s.position, float), np.asarray(s.v_y, float)
    m0, m2 = np.asarray(s.transform, float)[[0, 2]]
    rng = np.random.default_rng(int(gantry + collimator))
    p = rng.uniform(-25, 25, (3, 100000)).astype(f)
    p[:, :2000] = np.round(p[:, :2000])            # voxel planes through the axes
    rd = [f(src[k] - D(p[k])) for k in range(3)]
    ref, true = _mirror(src, vy, m0, m2, rd), _mirror(src, vy, m0, m2, rd, L)
    for ulps in (-2, 0, 2):
        got = _pairs(src, vy, m0, m2, rd, ulps)
        # what the dose reads is the off-axis distance.  The pair is off by about 2^-46 of terms up to
        # 64, 1e-12: it straddles a tie of a coordinate uniform in +-25 with probability 5e-7 per octave,
        # 20 octaves, and of three plane coordinates and the result
        oad = [np.sqrt(a * a + b * b) for a, b in (got, ref)]
        assert (oad[0] != oad[1]).mean() <= 2e-4
        for a, b, t in zip(got, ref, true):
            assert np.abs(D(a) - D(b)).max() <= 3 * 2.0 ** -18
            ea, eb = (np.sqrt(np.mean((L(x) - t) ** 2)) for x in (a, b))
            assert ea <= eb * (1 + 1e-6)
