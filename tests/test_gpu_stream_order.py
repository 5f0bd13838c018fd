"""GPU: calls on a busy stream.  Kernels that start while their predecessors end
must not read densities, maps or gradients that a caller's own kernel just before
them is still writing, nor write a dose that one after them still reads.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(settings):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conehead_gb300.engine import DoseEngine
    eng = DoseEngine(0)
    eng.set_kernel(settings["energy_weights"])
    return eng


def _setup(eng, settings, n, beams, gantry=20.0):
    import torch
    from conehead_gb300 import Block, GridPhantom, Source
    rng = np.random.default_rng(sum(n))
    ph = GridPhantom(rng.uniform(0.3, 1.7, n).astype(np.float32), tuple(-(k - 1) * 0.15 for k in n), (0.3, 0.3, 0.3))
    blk = Block()
    blk.set_rect(-3.0, 2.5, -2.0, 2.8)
    rho = eng.upload_densities(ph.densities)
    jobs = []
    for k in range(beams):
        src = Source()
        src.gantry, src.collimator = gantry + 31.0 * k, 7.0
        jobs.append(eng.job(ph, rho, src, eng.block_for(blk), settings))
    vols = [torch.from_numpy(rng.uniform(0.3, 1.7, n).astype(np.float32)).cuda() for _ in range(3)]
    return rho, jobs, vols


# one-launch prologue and early starts; the list with early starts; the plane path; a large launch
@pytest.mark.parametrize("n,beams", [((40, 37, 31), 1), ((64, 61, 50), 5), ((100, 99, 60), 2), ((130, 128, 90), 3)])
def test_densities_written_just_before(settings, n, beams):
    import torch
    eng = _engine(settings)
    rho, jobs, vols = _setup(eng, settings, n, beams)
    want = []
    for v in vols:
        rho.copy_(v)
        torch.cuda.synchronize()
        eng.run_batch(jobs)
        eng.sync()
        want.append([j.dose.clone() for j in jobs])
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        got = []
        for k in range(24):
            v = vols[k % 3]
            rho.fill_(50.0)                    # what an early read would find
            for part in torch.arange(0, n[0], 8).tolist():
                rho[part:part + 8].copy_(v[part:part + 8])
            eng.run_batch(jobs)
            got.append([j.dose * 1.0 for j in jobs])       # read while the next call begins
        eng.sync()
    for k, doses in enumerate(got):
        for a, b in zip(doses, want[k % 3]):
            assert torch.equal(a, b)


def test_gradients_written_just_before(settings):
    import torch
    from conehead_gb300 import GridPhantom, Source
    from conehead_gb300.adjoint import BeamletDose, BeamletGrid
    eng = _engine(settings)
    n = (40, 37, 31)
    rng = np.random.default_rng(3)
    ph = GridPhantom(rng.uniform(0.3, 1.7, n).astype(np.float32), tuple(-(k - 1) * 0.15 for k in n), (0.3, 0.3, 0.3))
    src = Source()
    src.gantry, src.collimator = 50.0, 0.0
    op = BeamletDose(eng, ph, src, BeamletGrid(8, 8, 60), settings)
    w = torch.rand((8, 8), generator=torch.Generator().manual_seed(1)).cuda() + 0.2
    ups = [torch.from_numpy(rng.uniform(0.1, 1.0, n).astype(np.float32)).cuda() for _ in range(3)]
    want = [op.backward(u, weights=w) for u in ups]
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        g = torch.empty_like(ups[0])
        got = []
        for k in range(24):
            g.fill_(1.0e6)
            for part in range(0, n[0], 8):
                g[part:part + 8].copy_(ups[k % 3][part:part + 8])
            got.append(op.backward(g, weights=w))
        eng.sync()
    for k, a in enumerate(got):
        # float64 adds in arrival order, stored in float32
        assert torch.allclose(a, want[k % 3], rtol=1e-6, atol=0)


def test_two_plans_on_two_streams(settings):
    import threading

    import torch
    engines = [_engine(settings) for _ in range(2)]
    setups = [_setup(e, settings, n, b, 20.0 + 90.0 * i)
              for i, (e, n, b) in enumerate(zip(engines, ((40, 37, 31), (64, 61, 50)), (1, 6)))]
    want = []
    for e, (rho, jobs, vols) in zip(engines, setups):
        e.run_batch(jobs)
        e.sync()
        want.append([j.dose.clone() for j in jobs])
    torch.cuda.synchronize()
    bad = [0, 0]

    def work(i):
        torch.cuda.set_device(0)
        eng, jobs = engines[i], setups[i][1]
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(40):
                for j in jobs:
                    j.dose.fill_(-1.0)
                eng.run_batch(jobs)
                eng.sync()
                bad[i] += sum(not torch.equal(j.dose, w) for j, w in zip(jobs, want[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert bad == [0, 0]
