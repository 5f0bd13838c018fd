"""GPU: block maps with infinities, NaN and values near the end of float32's range:
a dose-only call (samples summed as pairs of float32) gives what the call with
intermediates (float64 sums) gives.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
VALUES = [float("inf"), float("nan"), 3.0e38, -3.0e38, -float("inf"), 1.0e-42]


@pytest.mark.parametrize("value", VALUES)
@pytest.mark.parametrize("samples", [2, 3])
@pytest.mark.parametrize("n", [(20, 21, 17), (96, 95, 9)])       # the one-launch prologue with spectral; the list
def test_map_values(settings, value, samples, n):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conehead_gb300 import Block, GridPhantom, Source
    from conehead_gb300.engine import DoseEngine
    # every spectrum bin has a weight: 0 times infinity would hide what is compared
    s = dict(settings, fluenceResampling=samples, energy_weights={"1.0": 0.5, "2.0": 0.3})
    eng = DoseEngine(0)
    eng.set_kernel(s["energy_weights"])
    ph = GridPhantom(np.ones(n, np.float32), tuple(-(k - 1) * 0.2 for k in n), (0.4, 0.4, 0.4))
    src = Source()
    src.gantry, src.collimator = 20.0, 10.0
    v = np.zeros((4000, 4000), np.float32)
    v[1800:2200, 1800:2200] = 0.5
    v[1950:1975, 1960:1990] = value
    blk = Block()
    blk.block_values = v
    rho, db = eng.upload_densities(ph.densities), eng.block_for(blk)
    out = {}
    for method in (1, 0):            # the gather keeps what is not finite where its cones reach
        eng.set_tuning(cone_method=method)
        job = eng.job(ph, rho, src, db, s)
        eng.run(job)
        eng.sync()
        a = job.dose.cpu().numpy()
        b, inter = eng.run(eng.job(ph, rho, src, db, s), intermediates=True)
        eng.sync()
        b = b.cpu().numpy()
        T = inter["terma"].cpu().numpy()
        with np.errstate(invalid="ignore"):
            assert np.array_equal(np.isnan(a), np.isnan(b))
            assert np.array_equal(np.isposinf(a), np.isposinf(b)) and np.array_equal(np.isneginf(a), np.isneginf(b))
            ok = np.isfinite(b)
            if ok.any():
                assert np.abs(a[ok] - b[ok]).max() <= 1e-5 * np.abs(b[ok]).max()
        out[method] = T
    if value == float("inf"):
        assert np.isposinf(T).any() and not np.isnan(T).any()
