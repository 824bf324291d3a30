"""PostProcessor.register_image with an image of the same size allocates
nothing; another size gets a buffer of its own."""
import numpy as np
import pytest

import cupbr_b200 as cb
from cupbr_b200 import _native as N

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_same_size_keeps_its_buffer():
    images = [torch.rand(s, device="cuda") for s in ((30, 50, 3), (30, 50, 3), (50, 30, 3), (61, 33, 3))]
    pp, fresh = cb.PostProcessor(), []
    wrap = lambda t: cb.DeviceImage(t.data_ptr(), t.shape[1], t.shape[0], 3, np.float32, owner=t)
    threshold = cb.threshold_curve(0.8, 0.4)
    for t in images:
        p = cb.PostProcessor()
        p.register_image(wrap(t))
        p.bloom(threshold)
        fresh.append(p.get_post_process_buffer().numpy())
    pp.register_image(wrap(images[0]))
    for k, t in enumerate(images):
        try:
            N.call("cupbr_debug_fail_allocation", 0 if k < 3 else -1)
            pp.register_image(wrap(t))
        finally:
            N.call("cupbr_debug_fail_allocation", -1)
        pp.bloom(threshold)
        assert np.array_equal(pp.get_post_process_buffer().numpy(), fresh[k])
