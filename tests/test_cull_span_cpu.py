"""The span of voxels that the prologue lists on an (x, y) line holds every voxel
that the per-voxel frustum test keeps (CPU).

``line_span`` of conehead_gb300/csrc/prologue.cu, restated in float32 numpy, against
``voxel_candidates`` of test_cull_lines_cpu.py, on seeded grids, openings and beams,
grids that reach the source plane, single-voxel lines and coarse voxels."""
import numpy as np
import pytest

from conehead_gb300.source import Source
from test_cull_lines_cpu import F, beam_consts, voxel_candidates


def line_span(c, px, py, cz):
    nz = len(cz)
    whole = np.stack([np.zeros(px.shape, int), np.full(px.shape, nz)])
    if not c["enable"]:
        return whole
    kk = np.abs(c["a_K"])
    n_xy = c["vyf"][0] * px + c["vyf"][1] * py
    xs = [c["a_m0S"] - (c["m0f"][0] * px + c["m0f"][1] * py), c["a_m2S"] - (c["m2f"][0] * px + c["m2f"][1] * py)]
    ends = [cz[0], cz[-1]]
    depth = [(n_xy + c["vyf"][2] * z) - c["a_nS"] for z in ends]
    lin = [[xs[0] - c["m0f"][2] * z for z in ends], [xs[1] - c["m2f"][2] * z for z in ends]]
    ok = (depth[0] > F(0.2) * kk) & (depth[1] > F(0.2) * kk)
    with np.errstate(all="ignore"):
        inv = [F(1) / d for d in depth]
        lat = np.maximum(*[np.maximum(np.abs(lin[0][e]), np.abs(lin[1][e])) * inv[e] for e in (0, 1)])
        M = c["k"] * kk * np.maximum(*inv) * (F(1) + lat) + F(0.02)
        lo, hi = np.zeros(px.shape, F), np.full(px.shape, F(nz - 1))
        none = np.zeros(px.shape, bool)
        for k in range(4):
            v, cc = lin[k // 2], (c["a_c0"], c["a_c2"])[k // 2]
            edge = (c["cx_lo"], c["cx_hi"], c["cz_lo"], c["cz_hi"])[k]
            w, K = ((edge - cc) + M, c["a_K"]) if k & 1 else ((cc - edge) + M, -c["a_K"])
            g0, g1 = w * depth[0] + K * v[0], w * depth[1] + K * v[1]
            none |= (g0 < 0) & (g1 < 0)
            t = g0 / (g0 - g1) * F(nz - 1)
            lo = np.where((g0 < 0) & (g1 >= 0), np.fmax(lo, t - F(0.01)), lo)
            hi = np.where((g1 < 0) & (g0 >= 0), np.fmin(hi, t + F(0.01)), hi)
    z0, z1 = np.maximum(np.ceil(lo), 0).astype(int), np.minimum(np.floor(hi), nz - 1).astype(int) + 1
    empty = none | (z1 <= z0)
    z0, z1 = np.where(empty, 0, z0), np.where(empty, 0, z1)
    return np.where(ok, np.stack([z0, z1]), whole)


@pytest.mark.parametrize("seed", range(6))
def test_span_holds_every_candidate(seed):
    rng = np.random.default_rng(100 + seed)
    listed = needed = 0
    for case in range(40):
        n = [int(v) for v in rng.integers(1, 60, 3)]
        hi = 6.0 if case % 8 == 7 else 0.6
        spacing = [float(v) for v in rng.uniform(0.1, hi, 3)]
        if case % 5 == 4:
            n[2] = int(rng.choice([1, 2, 300]))
        ext = [a * b for a, b in zip(n, spacing)]
        origin = [-e / 2 + rng.uniform(-4, 4) for e in ext]
        src = Source()
        src.gantry = float(rng.choice([0.0, 90.0, 180.0, rng.uniform(0, 360)]))
        src.collimator = float(rng.choice([0.0, rng.uniform(0, 90)]))
        if case % 10 == 9:
            origin[1] = -100.0 + rng.uniform(-5, 25)
        h, off = rng.uniform(0.05, 12, 2), rng.uniform(-6, 6, 2)
        jaws = (max(off[0] - h[0], -20.0), min(off[0] + h[0], 20.0), max(off[1] - h[1], -20.0), min(off[1] + h[1], 20.0))
        c = beam_consts(src, jaws, spacing, int(rng.choice([1, 3, 5])))
        cen = [(F(o) + F(s) * np.arange(k).astype(F)).astype(F) for o, s, k in zip(origin, spacing, n)]
        X, Y = np.meshgrid(cen[0], cen[1], indexing="ij")
        px, py = X.ravel(), Y.ravel()
        z0, z1 = line_span(c, px, py, cen[2])
        if not c["enable"]:
            assert (z0 == 0).all() and (z1 == n[2]).all()
            continue
        cand = voxel_candidates(c, px[:, None], py[:, None], cen[2][None, :])
        z = np.arange(n[2])
        inside = (z >= z0[:, None]) & (z < z1[:, None])
        assert not (cand & ~inside).any(), case
        if not (n[2] == 1 or case % 8 == 7 or case % 10 == 9):
            listed += int(inside.sum())
            needed += int(cand.sum())
    assert needed > 0 and listed <= 1.15 * needed, listed / needed
