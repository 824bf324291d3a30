"""cupbr_gdpt_reconstruct on images with tiles that lie inside the border, which
take a kernel branch without bounds, beside tiles at the edges, for both of its
regions (tiles of 22 x 22 while 444 of them cover the image, else of 54 x 38):
bit-exact against the restatement of the 50 passes."""
import ctypes as C

import numpy as np
import pytest

from cupbr_b200 import _native as N
from test_gpu_gdpt_tiles import reconstruct

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# 22 x 22: tile edges, the last sizes without an interior tile and the first
# with one, several, ragged ones; the last image of the small tiles (444) and the
# first of the large; 54 x 38: as many tiles as fit exactly, a pixel more and
# less, a single row and column of tiles
@pytest.mark.parametrize("w,h", [(21, 22), (22, 22), (23, 23), (32, 32), (44, 45), (49, 50), (50, 49), (50, 50),
                                 (113, 82), (114, 81), (114, 82), (162, 152), (200, 150), (331, 241), (264, 814),
                                 (265, 814), (540, 456), (541, 457), (539, 455), (10001, 23), (23, 10001)])
def test_reconstruct_interior_tiles(w, h):
    rng = np.random.default_rng(100 * w + h)
    images = [rng.random((h, w, 3), dtype=np.float32) for _ in range(2)]
    images[1:1] = [(0.2 * (rng.random((h, w, 3), dtype=np.float32) - 0.5)).astype(np.float32) for _ in range(4)]
    base, gxf, gxb, gyf, gyb, temp = [torch.from_numpy(a.copy()).cuda() for a in images]
    gx, gy, out = (torch.zeros((h, w, 3), device="cuda") for _ in range(3))
    N.call("cupbr_gdpt_reconstruct", w, h,
           *[C.c_void_p(t.data_ptr()) for t in (base, gxf, gxb, gyf, gyb, gx, gy, temp, out)], None)
    torch.cuda.synchronize()
    for got, want in zip((out, gx, gy), reconstruct(*images)):
        assert np.array_equal(got.cpu().numpy(), want)
