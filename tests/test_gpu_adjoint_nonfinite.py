"""GPU: beamlet gradients of objectives whose dose gradient holds a NaN or an
infinity: beamlets without a sample of a voxel stay 0, no other call notices.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conehead_gb300.build import build
    build()
    from conehead_gb300.conehead import engine
    return engine(0)


@pytest.mark.parametrize("gantry,rows,cols,cell", [(0.0, 20, 20, 40), (33.0, 9, 20, 50), (90.0, 1, 3, 200),
                                                   (250.0, 5, 1, 60)])
def test_nonfinite_dose_gradient(eng, settings, gantry, rows, cols, cell):
    import torch
    from conehead_gb300 import Source
    from conehead_gb300.adjoint import BeamletDose, BeamletGrid
    from conehead_gb300.phantoms import slab_phantom
    ph = slab_phantom(24, 0.25, seed=3, n_inserts=2)
    src = Source()
    src.gantry = gantry
    src.collimator = 0.0
    op = BeamletDose(eng, ph, src, BeamletGrid(rows, cols, cell), settings)
    w = torch.rand((rows, cols), generator=torch.Generator().manual_seed(1)).cuda() + 0.5
    dose = op.forward(w)
    g = torch.rand(tuple(ph.size), generator=torch.Generator().manual_seed(2)).cuda()
    want = op.backward(g, weights=w)
    for bad in (float("nan"), float("inf")):
        gb = g.clone()
        gb[11, 12, 13] = bad
        got = op.backward(gb, weights=w)
        # the transform spreads it over all of dL/dTERMA: every beamlet the finite gradient reaches
        assert torch.equal(~torch.isfinite(got), want != 0)
        assert torch.equal(got[want == 0], want[want == 0])
        assert torch.equal(op.forward(w), dose)
        again = op.backward(g, weights=w)
        assert torch.allclose(again, want, rtol=1e-5, atol=0)
    assert bool((want != 0).any())
    if rows * cols > 40:                     # wider than the phantom's shadow
        assert bool((want == 0).any())
