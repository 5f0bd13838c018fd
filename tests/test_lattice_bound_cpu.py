"""How large the lattice's error bound may be (prologue.cu, LATTICE_DELTA_MAX; CPU).

A map sample is accepted on its float32 coordinate when the cell next to it, per
axis and on its side, holds the same value; a beamlet sample when no edge lies
within the bound.  Both are right for bounds up to the limit and wrong for
some coordinate beyond half a cell, where blocked_fraction and the adjoint take
the mirrored samples instead.
"""
import os
import re

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(__file__), "..", "conehead_gb300", "csrc", "prologue.cu")
LIMIT = float(re.search(r"LATTICE_DELTA_MAX = ([0-9.]+)f", open(SRC).read()).group(1))


def _samples(delta):
    rng = np.random.default_rng(int(delta * 1000))
    u = rng.uniform(2.0, 18.0, 200000)
    edge = np.round(u) + rng.uniform(-1.0, 1.0, u.size) * delta      # near the edges, from either side
    u = np.where(rng.random(u.size) < 0.5, u, edge)
    return u, u + rng.choice([-1.0, 1.0, 0.3], u.size) * delta * 0.999


def _map_wrong(delta):
    """Samples accepted without the mirror whose reference cell holds another value."""
    v = np.random.default_rng(3).integers(0, 2, 24)
    u, ref = _samples(delta)
    i = np.floor(u).astype(int)
    du = u - i - 0.5
    j = np.where(np.abs(du) >= 0.5 - delta, i + np.where(du < 0, -1, 1), i)
    accepted = v[i] == v[j]
    return int((accepted & (v[np.floor(ref).astype(int)] != v[i])).sum())


def _beamlet_wrong(delta, cell):
    u, ref = _samples(delta)
    q = np.floor(u / cell)
    d = u - q * cell
    accepted = ~((d < delta) | (d > cell - delta))
    return int((accepted & (np.floor(ref / cell) != q)).sum())


@pytest.mark.parametrize("delta", [0.002, 0.05, LIMIT])
def test_bounds_up_to_the_limit(delta):
    assert _map_wrong(delta) == 0
    assert all(_beamlet_wrong(delta, cell) == 0 for cell in (1, 2, 5))


def test_larger_bounds_are_wrong_somewhere():
    assert _map_wrong(0.75) > 0 and LIMIT < 0.5
