"""A wavefront of the medium large enough that every one of its persistent
kernels -- transmittance, with 6 blocks of 8 warps per SM the widest, among
them -- claims queue entries beyond the first deal: its image and gradients
against those of its frames in wavefronts of their own."""
import numpy as np
import pytest

import cupbr_b200 as cb
import cupbr_b200.medium as M
from cupbr_b200 import scenes
from test_gpu_medium import ALB, BOX, G, MAJ, gpu_backward

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_large_wavefront_equals_its_frames():
    grid, sc = scenes.perlin_grid(32, seed=2, sigma_max=8.0), scenes.medium_scene().build()
    warps = 48 * torch.cuda.get_device_properties(0).multi_processor_count
    w, h, spp = 512, 320, 5
    density = torch.from_numpy(grid).cuda()
    med = M.Medium(grid.shape, BOX, MAJ, ALB, G, 0.5)

    def forward(frames, frame0, depth):
        img = torch.zeros((h, w, 3), device="cuda")
        med.forward(sc, density.data_ptr(), cb.Camera(w, h), w, h, frames, frame0, depth, img.data_ptr())
        torch.cuda.synchronize()
        return img.double()

    med.set_instrumented(True)
    forward(spp, 0, 1)
    assert med.stats()["shadow_rays"] > 32 * warps  # of the first depth alone
    med.set_instrumented(False)
    whole, mean = forward(spp, 0, 4), sum(forward(1, k, 4) for k in range(spp)) / spp
    # a sum of five frames and a division, rounded to 24 bits each
    assert (whole - mean).abs().max() <= 6 * 2.0 ** -24 * mean.abs().max()
    wgt = np.random.default_rng(4).random((h, w, 3)).astype(np.float32)
    gd, gp = gpu_backward(med, sc, grid, w, h, spp, 0, 4, wgt)
    parts = [gpu_backward(med, sc, grid, w, h, 1, k, 4, wgt) for k in range(spp)]
    sd = sum(p[0].astype(np.float64) for p in parts) / spp
    sp = sum(p[1].astype(np.float64) for p in parts) / spp
    # sums of the same terms in another order, some thousands of either sign each
    assert np.abs(gd - sd).max() <= 1e-4 * np.abs(sd).max()
    assert np.abs(gp - sp).max() <= 1e-4 * np.abs(sp).max()
    assert med.error_count() == 0
