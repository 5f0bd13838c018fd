"""GPU: device paths chosen by size, at the sizes where they can go wrong.

* One-launch prologue (few small beams) against the list of a larger batch.
* Rows without TERMA, which are neither written nor read between the z and y
  passes: a narrow beam after wide ones equals the narrow beam on a new plan.
* Passes that ask L2 for lines ahead (large batches) against one beam at a time.
* A ray parallel to the blocking plane is reported by the call that met it.
* The radiological scatter with an axis above 512 voxels.
* All intermediates (every voxel in order, no list) against the plain dose, for
  both cone methods.
* Map rasters of every row length modulo 4 and of an unaligned buffer.
"""
import ctypes
import os
import sys

import numpy as np
import pytest

from conftest import GOLDEN

sys.path.insert(0, GOLDEN)

pytestmark = pytest.mark.gpu
TOL = 2e-6      # fraction of the largest dose: two float32 transforms of one TERMA


def _phantom(n, sp=(0.4, 0.4, 0.4)):
    from conehead_gb300 import GridPhantom
    rng = np.random.default_rng(sum(n))
    rho = rng.uniform(0.3, 1.7, n).astype(np.float32)
    return GridPhantom(rho, tuple(-(k - 1) * s / 2 for k, s in zip(n, sp)), sp)


def _engine(settings):
    from conehead_gb300.engine import DoseEngine
    eng = DoseEngine(0)
    eng.set_kernel(settings["energy_weights"])
    return eng


def _job(eng, ph, settings, gantry, collimator, field):
    from conehead_gb300 import Block, Source
    src = Source()
    src.gantry, src.collimator = gantry, collimator
    blk = Block()
    blk.set_rect(*field)
    return eng.job(ph, eng.upload_densities(ph.densities), src, eng.block_for(blk), settings)


def _doses(eng, jobs):
    eng.run_batch(jobs)
    eng.sync()
    return [j.dose.cpu().numpy() for j in jobs]


# 8192 lines are the most of the one-launch prologue; 91 x 91 is past it
@pytest.mark.parametrize("n", [(5, 6, 7), (1, 1, 40), (40, 1, 33), (33, 28, 47), (64, 128, 32), (91, 91, 20)])
@pytest.mark.parametrize("beams", [1, 4])
def test_one_launch_prologue_equals_the_list(settings, n, beams):
    eng = _engine(settings)
    ph = _phantom(n)
    field = (-3.1, 2.4, -1.9, 2.7)
    jobs = [_job(eng, ph, settings, 40.0 * k + 11.0, 17.0 * k, field) for k in range(beams)]
    more = jobs + [_job(eng, ph, settings, 200.0 + 9.0 * k, 5.0, field) for k in range(5 - beams)]
    few = _doses(eng, jobs)
    many = _doses(eng, more)
    for a, b in zip(few, many):
        assert b.max() > 0
        assert np.abs(a - b).max() <= TOL * b.max()


@pytest.mark.parametrize("n", [(36, 41, 30), (60, 75, 33), (17, 150, 66)])
@pytest.mark.parametrize("beams", [1, 6])
def test_rows_without_terma(settings, n, beams):
    ph = _phantom(n, (0.3, 0.3, 0.3))
    wide, narrow = (-9.0, 9.0, -9.0, 9.0), (-0.6, 0.7, -0.8, 0.5)
    used, new = _engine(settings), _engine(settings)

    def jobs(eng, field):
        return [_job(eng, ph, settings, 61.0 * k, 8.0 * k, field) for k in range(beams)]
    _doses(used, jobs(used, wide))
    for a, b in zip(_doses(used, jobs(used, narrow)), _doses(new, jobs(new, narrow))):
        assert b.max() > 0
        assert np.array_equal(a, b)


# the batch's work array is past 18 << 20 values, one beam's is not
@pytest.mark.parametrize("n,beams", [((150, 131, 155), 3), ((70, 250, 129), 4), ((33, 40, 200), 32)])
def test_lines_asked_for_ahead(settings, n, beams):
    eng = _engine(settings)
    ph = _phantom(n, (0.2, 0.2, 0.2))
    field = (-3.1, 2.4, -1.9, 2.7)
    jobs = [_job(eng, ph, settings, 23.0 * k % 360.0, 5.0 * k, field) for k in range(beams)]
    together = _doses(eng, jobs)
    for job, a in zip(jobs, together):
        b = _doses(eng, [job])[0]
        assert b.max() > 0
        assert np.abs(a - b).max() <= TOL * b.max()


def test_parallel_ray_is_reported_once(settings):
    from conehead_gb300 import GridPhantom
    from conehead_gb300 import _native as N
    eng = _engine(settings)
    bad_ph = GridPhantom(np.ones((4, 4, 4), np.float32), (-1.0, -101.0, -1.0), (1.0, 1.0, 1.0))
    bad = _job(eng, bad_ph, settings, 0.0, 0.0, (-5.0, 5.0, -5.0, 5.0))
    good = _job(eng, _phantom((12, 10, 9)), settings, 0.0, 0.0, (-2.0, 2.0, -2.0, 2.0))
    ref = _doses(eng, [good])[0]
    for trim in (False, True, False):
        with pytest.raises(RuntimeError, match="plane"):
            _doses(eng, [bad])
        assert np.array_equal(_doses(eng, [good])[0], ref)
        if trim:
            N.check(eng.L.ch_plan_trim(eng.plan), "ch_plan_trim")
            assert np.array_equal(_doses(eng, [good])[0], ref)


@pytest.mark.parametrize("n", [(3, 4, 520), (513, 3, 5), (4, 600, 2), (8, 9, 512)])
def test_radiological_scatter_of_long_axes(settings, n):
    from conehead_gb300 import GridPhantom
    sp = (0.2, 0.2, 0.2)
    ph = GridPhantom(np.ones(n, np.float32), tuple(-(k - 1) * s / 2 for k, s in zip(n, sp)), sp)
    eng = _engine(settings)
    jobs = [_job(eng, ph, dict(settings, coneDistance=d), 25.0, 0.0, (-30.0, 30.0, -30.0, 30.0))
            for d in ("geometric", "radiological")]
    geo, rad = (_doses(eng, [j])[0] for j in jobs)
    # water: the same taps and weights, summed in another order
    assert geo.max() > 0
    assert np.abs(rad - geo).max() <= 2e-5 * geo.max()


@pytest.mark.parametrize("n", [(2, 3, 5), (1, 1, 33), (31, 9, 29), (40, 28, 47)])
@pytest.mark.parametrize("method", [0, 1])
def test_dose_with_all_intermediates(settings, n, method):
    eng = _engine(settings)
    eng.set_tuning(cone_method=method)
    ph = _phantom(n)
    a = _doses(eng, [_job(eng, ph, settings, 33.0, 12.0, (-3.1, 2.4, -1.9, 2.7))])[0]
    job = _job(eng, ph, settings, 33.0, 12.0, (-3.1, 2.4, -1.9, 2.7))
    for _ in range(2):
        _, inter = eng.run(job, intermediates=True)
        eng.sync()
        # the gather adds each voxel's work units in arrival order
        assert np.abs(job.dose.cpu().numpy() - a).max() <= 1e-5 * a.max()
    blocked, terma = inter["blocked"].cpu().numpy(), inter["terma"].cpu().numpy()
    assert terma.max() > 0 and not terma[blocked == 0].any()


@pytest.mark.parametrize("cols", [1, 2, 3, 127, 129, 402, 403, 404])
@pytest.mark.parametrize("offset", [0, 1])
def test_map_raster_rows(settings, cols, offset):
    import torch
    from conehead_gb300 import _native as N
    from conehead_gb300 import dicom
    from conehead_gb300.block import MLCField
    eng = _engine(settings)
    mlc = MLCField.from_plan(dicom.read(os.path.join(GOLDEN, "RP.3DCRT.dcm"), force=True))
    r0, c0, rows = 1700, 1790, 61
    out = torch.full((rows * cols + 2,), -7.0, dtype=torch.float32, device="cuda")
    m = mlc.struct()
    N.check(eng.L.ch_block_from_mlc(ctypes.byref(m), out.data_ptr() + 4 * offset, rows, cols, r0, c0, eng.stream()),
            "ch_block_from_mlc")
    got = out.cpu().numpy()
    expect = np.full(rows * cols + 2, -7.0, np.float32)
    expect[offset:offset + rows * cols] = mlc.values()[r0:r0 + rows, c0:c0 + cols].ravel()
    assert np.array_equal(got, expect)
