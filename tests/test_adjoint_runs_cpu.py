"""The run sums of blocked_adjoint_kernel (prologue.cu), restated lane by lane
(CPU): 32 voxels with shares g and sample counts in the 2 x 2 beamlets from
(a, k) on, lanes with the same first beamlet summed and added once.

Whatever the shares hold, an add goes to a beamlet of the grid that has a sample
of one of the run's voxels; finite shares give each beamlet its sum.
"""
import numpy as np
import pytest

F = np.float32


def _adds(a, k, cnt, g, cols):
    """(index, value) of every add; cnt[lane, f] is 0 off the grid."""
    id0 = a * cols + k
    ghi = g.astype(F)
    glo = (g - ghi.astype(np.float64)).astype(F)
    same = np.append(id0[1:] == id0[:-1], False)
    run = np.array([next(r for r in range(32 - i) if not same[i + r]) for i in range(32)])
    first = np.append(True, ~same[:-1])
    out = []
    for f in range(4):
        n = cnt[:, f].astype(F)
        has = n > 0
        if not has.any():
            continue
        hi = np.where(has, ghi * n, F(0))
        lo = np.where(has, (ghi.astype(np.float64) * n - (ghi * n)).astype(F) + glo * n, F(0))
        for o in (1, 2, 4, 8, 16):
            h2, l2 = np.append(hi[o:], hi[-o:]), np.append(lo[o:], lo[-o:])
            t2 = hi + h2
            bb = t2 - hi
            l3 = (lo + l2) + ((hi - (t2 - bb)) + (h2 - bb))
            take = o <= run
            hi, lo = np.where(take, t2, hi), np.where(take, l3, lo)
        for i in range(32):
            total = float(hi[i]) + float(lo[i]) if abs(hi[i]) <= np.finfo(F).max else float(hi[i])
            if first[i] and has[i:i + run[i] + 1].any() and total != 0.0:
                out.append((int(id0[i]) + (f >> 1) * cols + (f & 1), total))
    return out


def _warp(rng, rows, cols):
    """32 voxels along a line that may enter or leave the grid on any side."""
    a = np.full(32, rng.integers(-1, rows))
    k = np.clip(np.sort(rng.integers(-2, cols + 1, 32)), -1, cols - 1)
    if rng.random() < 0.5:
        a, k = np.clip(np.sort(rng.integers(-2, rows + 1, 32)), -1, rows - 1), np.full(32, rng.integers(-1, cols))
    cnt = np.zeros((32, 4), int)
    for i in range(32):
        if rng.random() < 0.2:
            continue                                   # a voxel without TERMA or gradient
        for f in range(4):
            if 0 <= a[i] + (f >> 1) < rows and 0 <= k[i] + (f & 1) < cols and rng.random() < 0.6:
                cnt[i, f] = rng.integers(1, 28)
    return a, k, cnt


@pytest.mark.parametrize("rows,cols", [(1, 1), (2, 3), (5, 1), (7, 6)])
@pytest.mark.parametrize("bad", [None, np.nan, np.inf, -np.inf])
def test_adds_stay_on_sampled_beamlets(rows, cols, bad):
    rng = np.random.default_rng(rows * 100 + cols)
    with np.errstate(invalid="ignore", over="ignore"):
        for _ in range(60):
            a, k, cnt = _warp(rng, rows, cols)
            g = rng.standard_normal(32) * 10.0 ** rng.uniform(-6, 6, 32)
            if bad is not None:
                g[rng.random(32) < 0.3] = bad
            want = np.zeros(rows * cols)
            sampled, tainted = set(), set()
            for i in range(32):
                for f in range(4):
                    if cnt[i, f]:
                        j = (a[i] + (f >> 1)) * cols + k[i] + (f & 1)
                        sampled.add(int(j))
                        want[j] += g[i] * cnt[i, f]
                        if not np.isfinite(g[i]):
                            tainted.add(int(j))
            got = np.zeros(rows * cols)
            for j, v in _adds(a, k, cnt, g, cols):
                assert 0 <= j < rows * cols and j in sampled
                got[j] += v
            assert {int(j) for j in np.flatnonzero(~np.isfinite(got))} == tainted
            ok = np.isfinite(want)
            # a pair carries 48 bits, a run has at most 32 of them
            assert np.all(np.abs(got - want)[ok] <= 2.0 ** -40 * 32 * 27 * np.abs(g[np.isfinite(g)]).max(initial=0.0))
