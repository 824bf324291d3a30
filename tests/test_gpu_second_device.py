"""Kernels that opt in to more than 48 KB of dynamic shared memory, on two
devices of one process: the opt-in is the device's, not the process's."""
import ctypes as C

import numpy as np
import pytest

from cupbr_b200 import _native as N

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_reconstruct_on_two_devices():
    h, w = 90, 130
    base = np.random.default_rng(1).random((h, w, 3), dtype=np.float32)
    out = []
    for device in (0, 1):
        torch.cuda.set_device(device)
        src = torch.from_numpy(base).cuda()
        zero = [torch.zeros((h, w, 3), device="cuda") for _ in range(8)]
        N.call("cupbr_gdpt_reconstruct", w, h, *[C.c_void_p(t.data_ptr()) for t in (src, *zero)], None)
        torch.cuda.synchronize()
        out.append(zero[-1].cpu().numpy())
    torch.cuda.set_device(0)
    assert out[0].any() and np.array_equal(out[0], out[1])
