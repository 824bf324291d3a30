"""cupbr_gdpt_reconstruct at the edges of its kernel's tiles (54 x 38 output
pixels of a 64 x 48 region) against a numpy restatement of the 50 passes
(GradientDomain.cu:248-350, 379-401) in the same float operations.  Bar:
bit-exact."""
import ctypes as C

import numpy as np
import pytest

from cupbr_b200 import _native as N

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def reconstruct(base, gxf, gxb, gyf, gyb, temp):
    f = np.float32
    h, w, _ = base.shape
    inner = (slice(1, h - 1), slice(1, w - 1))
    gx, gy = np.zeros_like(base), np.zeros_like(base)
    gx[inner], gy[inner] = gxf[inner] + gxb[inner], gyf[inner] + gyb[inner]
    cur, border = base.copy(), temp.copy()
    for i in range(50):
        nxt = border.copy()  # from the second pass on the border is temp's
        if w > 2 and h > 2:
            v1 = cur[1:-1, :-2] + gx[1:-1, :-2]
            v2 = cur[:-2, 1:-1] + gy[:-2, 1:-1]
            v3 = cur[1:-1, 2:] - gx[1:-1, 1:-1]
            v4 = cur[2:, 1:-1] - gy[1:-1, 1:-1]
            lo = np.minimum(np.minimum(v1, v2), np.minimum(v3, v4))
            hi = np.maximum(np.maximum(v1, v2), np.maximum(v3, v4))
            nxt[inner] = ((((v1 + v2) + v3) + v4) - lo - hi) / f(2)
        cur = nxt
    return cur, gx, gy


@pytest.mark.parametrize("w,h", [(1, 1), (2, 5), (3, 3), (4, 3), (53, 37), (54, 38), (55, 39), (59, 43), (60, 44),
                                 (64, 48), (108, 76), (109, 77), (200, 31), (31, 200)])
def test_reconstruct_tile_edges(w, h):
    rng = np.random.default_rng(100 * w + h)
    base = rng.random((h, w, 3), dtype=np.float32)
    g = [(0.2 * (rng.random((h, w, 3), dtype=np.float32) - 0.5)).astype(np.float32) for _ in range(4)]
    temp = rng.random((h, w, 3), dtype=np.float32)
    dev = lambda a: torch.from_numpy(a.copy()).cuda()
    ptr = lambda t: C.c_void_p(t.data_ptr())
    d_base, d_g, d_temp = dev(base), [dev(a) for a in g], dev(temp)
    d_gx, d_gy, d_out = (torch.zeros((h, w, 3), device="cuda") for _ in range(3))
    N.call("cupbr_gdpt_reconstruct", w, h, ptr(d_base), *[ptr(a) for a in d_g], ptr(d_gx), ptr(d_gy), ptr(d_temp),
           ptr(d_out), None)
    torch.cuda.synchronize()
    out, gx, gy = reconstruct(base, *g, temp)
    assert np.array_equal(d_gx.cpu().numpy(), gx) and np.array_equal(d_gy.cpu().numpy(), gy)
    assert np.array_equal(d_out.cpu().numpy(), out)
    assert np.array_equal(d_base.cpu().numpy(), base)
