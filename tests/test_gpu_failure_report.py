"""GPU: which call a device-side failure is reported to, and the statistics that
go with it.

* Captured batches of one plan, waited for by two threads at the same time, each
  report their own failure.
* A call of several beams fails where any of them does, whatever launches it
  takes for each; the next call does not, and a refused call reports nothing.
* Statistics are the last call's, whatever method the call before it used.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(settings):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conehead_gb300.build import build
    build()
    from conehead_gb300.engine import DoseEngine
    eng = DoseEngine(0)
    eng.set_kernel(settings["energy_weights"])
    return eng


def _job(eng, settings, parallel=False, n=12):
    """A beam; parallel: its source plane runs through a layer of voxel centres."""
    from conehead_gb300 import Block, GridPhantom, Source
    rho = np.ones((4, 4, 4) if parallel else (n, n - 1, n - 2), np.float32)
    origin = (-1.0, -101.0, -1.0) if parallel else (-5.0, -5.0, -5.0)
    ph = GridPhantom(rho, origin, (1.0, 1.0, 1.0))
    src = Source()
    src.gantry = 0.0
    src.collimator = 0.0
    blk = Block()
    blk.set_rect(-5.0, 5.0, -5.0, 5.0)
    return eng.job(ph, eng.upload_densities(ph.densities), src, eng.block_for(blk), settings, swap_xy=0)


def test_two_threads_wait_for_batches_of_one_plan(settings):
    import torch
    eng = _engine(settings)
    eng.prepare((12, 12, 12), (1.0, 1.0, 1.0))
    kinds = (True, False)
    batches = [eng.capture([_job(eng, settings, parallel=k)]) for k in kinds]
    streams = [torch.cuda.Stream() for _ in kinds]
    torch.cuda.synchronize()
    wrong = [0, 0]
    start = threading.Barrier(2)

    def wait(i):
        torch.cuda.set_device(0)
        with torch.cuda.stream(streams[i]):
            batches[i].launch()
            torch.cuda.current_stream().synchronize()
            start.wait()
            for _ in range(4000):
                try:
                    batches[i].sync()
                    wrong[i] += kinds[i]
                except RuntimeError as e:
                    wrong[i] += not (kinds[i] and "plane" in str(e))

    threads = [threading.Thread(target=wait, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == [0, 0]


@pytest.mark.parametrize("n", [12, 100])    # the one-launch prologue, the list
def test_statistics_after_a_method_switch(settings, n):
    eng = _engine(settings)
    job = _job(eng, settings, n=n)
    for _ in range(2):
        eng.set_tuning(cone_method=1)
        eng.run(job)
        eng.sync()
        gather = eng.stats()
        assert gather["updates"] > 0 and gather["n_units"] > 0
        eng.set_tuning(cone_method=0)
        eng.run(job)
        eng.sync()
        spectral = eng.stats()
        assert spectral["updates"] == 0 and spectral["n_units"] == 0
        assert spectral["ms_prologue"] > 0 and spectral["ms_cone"] > 0


# geometric beams in the room frame take the one-launch prologue, the others a list
KINDS = ({}, {"coneFrame": "beam"}, {"coneDistance": "radiological"})


@pytest.mark.parametrize("first", range(3))
@pytest.mark.parametrize("second", range(3))
def test_any_beam_of_a_call_may_fail(settings, first, second):
    eng = _engine(settings)
    options = [dict(settings, **KINDS[k]) for k in (first, second)]
    # a beam with options makes the call run beam by beam
    last = _job(eng, dict(settings, **KINDS[1]), n=9)
    for bad in (None, 0, 1):
        jobs = [_job(eng, o, parallel=(i == bad)) for i, o in enumerate(options)] + [last]
        eng.run_batch(jobs)
        if bad is None:
            eng.sync()
            continue
        for _ in range(2):
            with pytest.raises(RuntimeError, match="plane"):
                eng.sync()
        broken = _job(eng, settings)
        broken.grid.n[0] = 0
        with pytest.raises(Exception, match="invalid argument"):
            eng.run(broken)
        with pytest.raises(RuntimeError, match="plane"):
            eng.sync()
        for o in options:
            eng.run(_job(eng, o))
            eng.sync()
