"""The adjoint's light terms in a kernel of their own (k_medium_replay) and the
medium kernels' deal of their queues: several lights against the oracle, and
a wavefront large enough that lanes claim entries beyond the first deal
against the sum of its frames in wavefronts of their own."""
import numpy as np
import pytest

import cupbr_b200 as cb
import cupbr_b200.medium as M
from cupbr_b200 import scenes
from oracle.bridge import CheckerScene
from test_gpu_medium import ALB, BOX, BOXF, G, MAJ, gpu_backward

pytestmark = pytest.mark.gpu


def three_lights():
    desc = scenes.medium_scene()
    desc.lights = list(desc.lights) + [
        scenes.LightDesc(scenes.POINT, (0.4, 0.6, 1.5), intensity=(0.6, 0.0, 0.3)),
        scenes.LightDesc(scenes.POINT, (-0.5, 0.2, 1.2), intensity=(0.2, 0.5, 0.1)),
    ]
    return desc


@pytest.mark.parametrize("w,h,spp", [(3, 2, 1), (45, 31, 3)])
def test_several_lights_match_oracle(w, h, spp):
    desc, grid = three_lights(), scenes.perlin_grid(32, seed=2, sigma_max=8.0)
    sc = desc.build()
    med = M.Medium(grid.shape, BOX, MAJ, ALB, G, 0.5)
    wgt = np.random.default_rng(4).random((h, w, 3)).astype(np.float32)
    gd, gp = gpu_backward(med, sc, grid, w, h, spp, 0, 5, wgt)
    rd, rp = CheckerScene(desc, "oracle").medium_backward(grid, BOXF, MAJ, ALB, G, 0.5, cb.Camera(w, h).flat(), w,
                                                          h, spp, 0, 5, wgt.reshape(-1, 3), gp.size)
    # the bounds of the single-light comparison
    touched = (rd != 0) | (gd != 0)
    close = np.abs(gd - rd) <= 1e-3 * np.abs(rd) + 1e-6 * np.abs(rd).max()
    assert close[touched].mean() >= 0.95
    assert np.allclose(gp, rp, rtol=1e-3, atol=1e-6 * np.abs(rp).max()), (gp, rp)
    assert med.error_count() == 0


def test_one_wavefront_equals_its_frames():
    """More than 32 queue entries per warp (4736 warps on 148 SMs).  The two
    sides add the same terms in another order: with up to a few thousand terms
    per entry of random sign their difference stays below 1e-4 of the largest."""
    desc, grid = three_lights(), scenes.perlin_grid(32, seed=2, sigma_max=8.0)
    sc = desc.build()
    w, h, spp = 256, 160, 5
    med = M.Medium(grid.shape, BOX, MAJ, ALB, G, 0.5)
    wgt = np.random.default_rng(4).random((h, w, 3)).astype(np.float32)
    gd, gp = gpu_backward(med, sc, grid, w, h, spp, 0, 4, wgt)
    parts = [gpu_backward(med, sc, grid, w, h, 1, k, 4, wgt) for k in range(spp)]
    sd = sum(p[0].astype(np.float64) for p in parts) / spp
    sp = sum(p[1].astype(np.float64) for p in parts) / spp
    assert np.abs(gd - sd).max() <= 1e-4 * np.abs(sd).max()
    assert np.abs(gp - sp).max() <= 1e-4 * np.abs(sp).max()
    assert med.error_count() == 0
