"""GPU: blocking on a grid whose extent makes the float32 error bound exceed a
quarter of a cell near the source (45 m along the beam, from 21 cm off the source
on): every sample is mirrored there, and blocked stays bit-exact.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _phantom():
    from conehead_gb300 import GridPhantom
    n, sp = (6, 1500, 5), (0.7, 3.0, 0.9)
    rho = np.random.default_rng(5).uniform(0.01, 0.05, n).astype(np.float32)
    ph = GridPhantom(rho, (-1.75, -79.0, -1.8), sp)
    # the bound of lattice_centre at the nearest voxels (gantry 0: the source at y = -100)
    P = -79.0 + 1500 * 3.0
    err = 2.0 ** -24 * (np.sqrt(3) * P + P + 100 + 8 * (P + 4))
    assert 100 * 100 / (21 + 1) * err > 0.25 and 100 * 100 / 1000 * err < 0.25
    return ph


def _source():
    from conehead_gb300 import Source
    src = Source()
    src.gantry, src.collimator = 0.0, 31.0
    return src


@pytest.mark.parametrize("samples", [2, 3])
def test_blocked_bitexact_far_from_the_origin(settings, oracle_lib, samples):
    from conehead_gb300 import Block, Conehead
    rng = np.random.default_rng(6)
    v = np.zeros((4000, 4000), dtype=np.float32)
    v[1000:3000, 1000:3000] = np.repeat(np.repeat(rng.random((80, 200)), 25, 0), 10, 1)
    graded = Block()
    graded.block_values = v
    jaw = Block()
    jaw.set_rect(-3.13, 2.58, -4.02, 3.77)
    ph, src = _phantom(), _source()
    s = dict(settings, fluenceResampling=samples)
    for blk in (graded, jaw):
        got = Conehead().calculate(src, blk, ph, s, return_intermediates=True)["blocked"]
        ref = oracle_lib.prologue(src, blk, ph, s, oracle_lib.MODE_F32)["blocked"]
        assert ((ref > 0) & (ref < 1)).any()
        assert np.array_equal(got, ref)


@pytest.mark.parametrize("samples", [2, 3])
def test_fine_beamlets_sum_to_coarse_ones(settings, samples):
    import torch
    from conehead_gb300.adjoint import BeamletDose, BeamletGrid
    from conehead_gb300.conehead import engine
    eng = engine(0)
    ph, src = _phantom(), _source()
    s = dict(settings, fluenceResampling=samples)
    g = torch.Generator().manual_seed(4)
    w = torch.rand((8, 8), generator=g) + 0.1
    up = torch.rand(tuple(ph.size), generator=g).cuda()
    big = BeamletDose(eng, ph, src, BeamletGrid(8, 8, 20), s)
    small = BeamletDose(eng, ph, src, BeamletGrid(32, 32, 5), s)
    a = big.backward(up, weights=w.cuda()).double()
    b = small.backward(up, weights=w.cuda().repeat_interleave(4, 0).repeat_interleave(4, 1)).double()
    b = b.reshape(8, 4, 8, 4).sum((1, 3))
    assert float(a.abs().max()) > 0
    # float32 stores of the fine gradients: 2^-24 of each, 16 of them, of one sign
    assert float((a - b).abs().max()) <= 2e-6 * float(a.abs().max())
