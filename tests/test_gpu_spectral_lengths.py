"""GPU: every transform length of the spectral cone stage, at the last size it
holds and the first of the next, against the stencil gather.

x and y of n voxels take a period >= 2 n - 1, z a length >= n; lengths above 512
take the general passes; 97-128 voxels along x and y take the plane path with any
length along z."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 2e-6     # fraction of the largest output: both methods are float32

SIZES = [(24, 120, 48), (25, 96, 64), (32, 97, 80), (33, 80, 96), (40, 72, 128), (48, 64, 144), (49, 48, 160),
         (64, 40, 192), (65, 32, 240), (72, 24, 256), (80, 144, 49), (81, 160, 33), (97, 161, 30), (120, 20, 320),
         (121, 192, 20), (144, 25, 257), (145, 26, 385), (193, 30, 24), (216, 18, 40), (217, 22, 20), (256, 20, 24),
         (18, 216, 31), (20, 217, 26), (12, 20, 433), (257, 12, 20), (14, 260, 18), (16, 13, 513), (9, 400, 12),
         (97, 128, 49), (128, 100, 17), (101, 99, 145), (5, 6, 7)]


@pytest.mark.parametrize("size", SIZES)
def test_operator_matches_the_gather(settings, size):
    import torch
    from conehead_gb300.adjoint import cone
    from conehead_gb300.conehead import engine
    eng = engine(0)
    eng.set_kernel(settings["energy_weights"])
    spacing = (0.3, 0.3, 0.3)
    g = torch.Generator().manual_seed(sum(size))
    x = torch.rand(size, generator=g) * (torch.rand(size, generator=g) > 0.95)
    x[0, 0, 0] = x[-1, -1, -1] = 1.0
    x = x.cuda()
    out = {}
    for method in (0, 1):
        eng.set_tuning(cone_method=method)
        try:
            out[method] = [cone(eng, size, spacing, x, transpose=t).cpu().numpy() for t in (False, True)]
        finally:
            eng.set_tuning()
    for a, b in zip(out[0], out[1]):
        assert np.abs(a - b).max() <= TOL * np.abs(b).max()
