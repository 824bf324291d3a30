"""cupbr_gdpt_reconstruct on images with tiles that lie inside the border, which
take a kernel branch without bounds (from 114 x 82 on), beside tiles at the
edges: bit-exact against the restatement of the 50 passes."""
import ctypes as C

import numpy as np
import pytest

from cupbr_b200 import _native as N
from test_gpu_gdpt_tiles import reconstruct

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# the last size without such a tile and the first with one; several; ragged ones
@pytest.mark.parametrize("w,h", [(113, 82), (114, 81), (114, 82), (162, 152), (200, 150), (331, 241)])
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
