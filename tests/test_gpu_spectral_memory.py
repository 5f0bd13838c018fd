"""GPU: the spectral work arena of large grids is bounded, and beams past the
bound take another launch.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ARENA = 16 << 30


@pytest.fixture(scope="module")
def eng(settings):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conehead_gb300.build import build
    build()
    from conehead_gb300.engine import DoseEngine
    e = DoseEngine(0)
    e.set_kernel(settings["energy_weights"])
    yield e
    e.close()


def _total(eng, n, beams, method):
    from conehead_gb300 import _native as N
    eng.set_tuning(cone_method=method)
    try:
        grids = (N.Grid * beams)(*[N.grid_struct(n, (0.0, 0.0, 0.0), (0.2, 0.2, 0.2))] * beams)
        total = ctypes.c_size_t()
        N.check(eng.L.ch_batch_scratch_bytes(eng.plan, beams, grids, None, ctypes.byref(total)), "scratch")
        return total.value
    finally:
        eng.set_tuning()


# 350^3 transforms at 768 x 768 x 384: 1.2 GB a beam
@pytest.mark.parametrize("n", [(201, 201, 201), (256, 256, 256), (350, 350, 350), (500, 400, 100)])
def test_arena_is_bounded(eng, n):
    voxels = n[0] * n[1] * (-(-n[2] // 4) * 4)
    for beams in (1, 32, 64):
        # TERMA and the voxel list are 8 bytes a voxel (and the line flags a byte a line)
        rest = beams * (8 * voxels + n[0] * n[1] + 8192)
        assert _total(eng, n, beams, 0) <= rest + ARENA


def test_beams_past_the_bound(eng, settings):
    import torch
    from conehead_gb300 import Block, GridPhantom, Source
    n = (240, 400, 256)           # 0.65 GiB a beam: 24 fit
    rho = np.random.default_rng(1).uniform(0.5, 1.5, n).astype(np.float32)
    ph = GridPhantom(rho, tuple(-(k - 1) * 0.1 for k in n), (0.2, 0.2, 0.2))
    r = eng.upload_densities(ph.densities)
    blk = Block()
    blk.set_rect(-2.0, 2.4, -1.6, 2.2)
    db = eng.block_for(blk)
    jobs = []
    for k in range(26):
        src = Source()
        src.gantry, src.collimator = 13.0 * k, 0.0
        jobs.append(eng.job(ph, r, src, db, settings))
    eng.run_batch(jobs)
    eng.sync()
    got = [jobs[k].dose.clone() for k in (0, 23, 24, 25)]
    for k, a in zip((0, 23, 24, 25), got):
        eng.run(jobs[k])
        eng.sync()
        assert float(a.max()) > 0
        # the same transforms of the same TERMA
        assert float((a - jobs[k].dose).abs().max()) <= 2e-6 * float(a.max())
    torch.cuda.empty_cache()
