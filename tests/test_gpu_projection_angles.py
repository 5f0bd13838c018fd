"""GPU: a dose-only call (pairs of float32 in the off-axis projection) against the
call that returns every intermediate (float64 projection), at right angles.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gantry", [0.0, 90.0, 180.0, 270.0])
@pytest.mark.parametrize("collimator", [0.0, 90.0])
@pytest.mark.parametrize("n", [(40, 37, 31), (100, 98, 30)])       # the one-launch prologue, the list
def test_right_angles(settings, gantry, collimator, n):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conehead_gb300 import Block, Conehead, GridPhantom, Source
    rho = np.random.default_rng(sum(n)).uniform(0.3, 1.7, n).astype(np.float32)
    ph = GridPhantom(rho, tuple(-(k - 1) * 0.4 / 2 for k in n), (0.4, 0.4, 0.4))
    src = Source()
    src.gantry, src.collimator = gantry, collimator
    blk = Block()
    blk.set_rect(-5.1, 4.4, -3.9, 4.7)
    a = np.asarray(Conehead().calculate(src, blk, ph, settings))
    b = Conehead().calculate(src, blk, ph, settings, return_intermediates=True)["dose"]
    assert b.max() > 0
    # two float32 transforms of TERMA volumes that differ by an ulp of the off-axis distance at most
    assert np.abs(a - b).max() <= 2e-6 * b.max()
