"""GPU: the blocked fraction's lattice path and the beamlet adjoint's two ways
of adding, where they can go wrong.

* blocked is bit-exact against the float32-mirrored oracle for 1 to 5
  sub-samples per axis, for a jaw opening, a map of graded values and a map
  open to its last row and column (which the wrapped index also reads).
* The gradient of small beamlets, summed over the coarse beamlet that holds
  them, is the coarse beamlet's: the same samples through the per-change adds
  and through the per-warp byte counts.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _phantom(n, sp):
    from conehead_gb300 import GridPhantom
    rng = np.random.default_rng(sum(n))
    rho = rng.uniform(0.2, 1.9, n).astype(np.float32)
    return GridPhantom(rho, tuple(-(k - 1) * s / 2 for k, s in zip(n, sp)), sp)


def _source(g, c):
    from conehead_gb300 import Source
    src = Source()
    src.gantry, src.collimator = g, c
    return src


def _blocks():
    from conehead_gb300 import Block
    jaw = Block()
    jaw.set_rect(-3.13, 2.58, -4.02, 3.77)
    rng = np.random.default_rng(4)
    graded = Block()
    v = np.zeros((4000, 4000), dtype=np.float32)
    v[1700:2350, 1650:2300] = np.repeat(np.repeat(rng.random((13, 26)), 50, 0), 25, 1)
    v[1900:1915, 1650:2300] *= np.linspace(1, 0, 15, dtype=np.float32)[:, None]
    graded.block_values = v
    wrap = Block()
    v = np.zeros((4000, 4000), dtype=np.float32)
    v[1500:, 1800:] = 1.0
    v[3999, :] = 0.5
    wrap.block_values = v
    return {"jaw": jaw, "graded": graded, "wrap": wrap}


@pytest.mark.parametrize("samples", [1, 2, 3, 5])
@pytest.mark.parametrize("kind", ["jaw", "graded", "wrap"])
def test_blocked_bitexact(settings, oracle_lib, kind, samples):
    from conehead_gb300 import Conehead
    ph = _phantom((33, 28, 47), (0.5, 0.6, 0.9))          # reaches 21 cm off axis: past the map's edge
    src, blk = _source(37.0, 22.0), _blocks()[kind]
    s = dict(settings, fluenceResampling=samples)
    got = Conehead().calculate(src, blk, ph, s, return_intermediates=True)["blocked"]
    ref = oracle_lib.prologue(src, blk, ph, s, oracle_lib.MODE_F32)["blocked"]
    assert (ref > 0).any()
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("coarse,cell,fine", [(8, 50, 10), (4, 25, 25), (6, 21, 3)])
def test_fine_beamlets_sum_to_coarse_ones(settings, coarse, cell, fine):
    import torch
    from conehead_gb300.adjoint import BeamletDose, BeamletGrid
    from conehead_gb300.conehead import engine
    eng = engine(0)
    ph = _phantom((40, 37, 30), (0.25, 0.25, 0.25))
    src = _source(61.0, 13.0)
    g = torch.Generator().manual_seed(coarse)
    w = torch.rand((coarse, coarse), generator=g) + 0.1
    up = torch.randn(tuple(ph.size), generator=g).cuda()
    r0 = 2000 - coarse * cell // 2
    big = BeamletDose(eng, ph, src, BeamletGrid(coarse, coarse, cell, r0=r0, c0=r0), settings)
    k = fine
    small = BeamletDose(eng, ph, src, BeamletGrid(coarse * k, coarse * k, cell // k, r0=r0, c0=r0), settings)
    a = big.backward(up, weights=w.cuda()).double()
    b = small.backward(up, weights=w.cuda().repeat_interleave(k, 0).repeat_interleave(k, 1)).double()
    b = b.reshape(coarse, k, coarse, k).sum((1, 3))
    assert float(a.abs().max()) > 0
    # float32 stores of the fine gradients: 2^-24 of each, k^2 of them
    assert float((a - b).abs().max()) <= 2e-6 * float(a.abs().max())
