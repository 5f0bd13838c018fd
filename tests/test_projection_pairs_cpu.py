"""The projection in pairs of float32 (prologue.cu, project_pairs) against the
float64 projection it stands for, both written out in numpy (CPU)."""
import numpy as np
import pytest

f, D, L = np.float32, np.float64, np.longdouble


def _fma(a, b, c):
    return (L(a) * L(b) + L(c)).astype(f)


def _two_sum(a, b):
    s = a + b
    bb = s - a
    return s, (a - (s - bb)) + (b - bb)


def _split(v):
    h = f(v)
    return h, f(D(v) - D(h))


def _dot(v, r):
    p, e = [], []
    for k in range(3):
        h, lo = _split(v[k])
        m = h * r[k]
        p.append(m)
        e.append(_fma(lo, r[k], _fma(h, r[k], -m)))
    a, ae = _two_sum(p[0], p[1])
    t, te = _two_sum(a, p[2])
    return t, ((e[0] + e[1]) + ae) + (e[2] + te)


def _pairs(src, vy, m0, m2, rd):
    vyw = D(f(src[0])) * vy[0] + D(f(src[1])) * vy[1] + D(f(src[2])) * vy[2]
    wh, wl = _split(vyw)
    dh, dl = _dot(vy, rd)
    h = dh + dl
    lo = (dh - h) + dl
    q1 = -wh / h
    q2 = (_fma(-q1, lo, _fma(-q1, h, np.broadcast_to(-wh, h.shape))) - wl) / h
    pp = []
    for k in range(3):
        m = q1 * rd[k]
        e = _fma(q2, rd[k], _fma(q1, rd[k], -m))
        s, se = _two_sum(np.broadcast_to(f(src[k]), m.shape), m)
        pp.append(s + (se + e))
    return [a + b for a, b in (_dot(m0, pp), _dot(m2, pp))]


def _mirror(src, vy, m0, m2, rd, T=D):
    """T = D: project_exact_mixed; T = L: the same formula with no rounding but the ray's."""
    r = [T(x) for x in rd]
    w = [T(f(s)) for s in src]
    vyw = w[0] * vy[0] + w[1] * vy[1] + w[2] * vy[2]
    si = -vyw / (vy[0] * r[0] + vy[1] * r[1] + vy[2] * r[2])
    pp = [w[k] + si * r[k] for k in range(3)]
    if T is D:
        pp = [D(f(x)) for x in pp]
    out = [m[0] * pp[0] + m[1] * pp[1] + m[2] * pp[2] for m in (m0, m2)]
    return [f(x) for x in out] if T is D else out


@pytest.mark.parametrize("gantry,collimator,sad", [(0.0, 0.0, 100.0), (30.0, 0.0, 100.0), (90.0, 45.0, 100.0),
                                                   (213.7, 12.3, 100.0), (300.0, 90.0, 80.0), (61.0, 179.0, 150.0)])
def test_pairs_equal_float64(gantry, collimator, sad):
    g, c = np.deg2rad(gantry), np.deg2rad(collimator)
    rot_g = np.array([[np.cos(g), -np.sin(g), 0], [np.sin(g), np.cos(g), 0], [0, 0, 1]])
    rot_c = np.array([[np.cos(c), 0, np.sin(c)], [0, 1, 0], [-np.sin(c), 0, np.cos(c)]])
    xf = rot_c @ rot_g
    vy, m0, m2 = xf[1], xf[0], xf[2]
    src = -sad * vy
    rng = np.random.default_rng(int(gantry))
    p = rng.uniform(-25, 25, (3, 200000)).astype(f)
    rd = [f(src[k] - D(p[k])) for k in range(3)]
    got, ref, true = _pairs(src, vy, m0, m2, rd), _mirror(src, vy, m0, m2, rd), _mirror(src, vy, m0, m2, rd, L)
    for a, b, t in zip(got, ref, true):
        # a plane point one step of float32 off (|pp| < 64: 2^-18) where the pair
        # and the float64 value straddle a tie, three of them at most
        assert np.abs(D(a) - D(b)).max() <= 3 * 2.0 ** -18
        assert (a != b).mean() <= 1e-3
        ea, eb = (np.sqrt(np.mean((L(x) - t) ** 2)) for x in (a, b))
        assert ea <= eb * (1 + 1e-4)
