"""The texture adjoint of few paths, one thread per path, against the same
gradient through wavefronts (which a view of three frames without an image
gradient brings about), and the wavefronts when memory runs out: halved, or no
more than one thread per path.  Bar: the order of the float additions (a texel
sums at most a few thousand terms: 1e-5 of the largest)."""
import numpy as np
import pytest

import cupbr_b200 as cb
from cupbr_b200 import _native as N
from cupbr_b200 import scenes

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def gradient(built, sizes, spp, extra=False, fail_at=None, calls=1):
    g = torch.Generator(device="cuda").manual_seed(4)
    views, grads, keep = [], [], []
    for i, (w, h) in enumerate(sizes):
        img = torch.zeros((h, w, 3), device="cuda")
        grad = torch.rand((h, w, 3), generator=g, device="cuda") - 0.5
        grad[: h // 3] = 0.0  # paths of weight 0 are not traced
        keep += [img, grad]
        views.append(dict(scene=built[i % len(built)], camera=cb.Camera(w, h), width=w, height=h, spp=spp, frame0=i,
                          image=img.data_ptr()))
        grads.append(grad.data_ptr())
    if extra:
        img = torch.zeros((8, 8, 3), device="cuda")
        keep.append(img)
        views.append(dict(scene=built[0], camera=cb.Camera(8, 8), width=8, height=8, spp=3, frame0=0,
                          image=img.data_ptr()))
        grads.append(0)
    batch = cb.Batch(views, 5)
    try:
        if fail_at is not None:
            N.call("cupbr_debug_fail_allocation", fail_at)
        for k in range(calls):
            batch.backward(grads)
    finally:
        N.call("cupbr_debug_fail_allocation", -1)
    torch.cuda.synchronize()
    assert batch.error_count() == 0
    return [torch.as_tensor(batch.texture_gradient(s), device="cuda").cpu().numpy() for s in built[:2]]


@pytest.fixture(scope="module")
def built():
    return [scenes.with_texture(scenes.cornell_variant(5), 16, seed=17).build(),
            scenes.with_texture(scenes.cornell_variant(6), 33, seed=3).build(),
            scenes.cornell_box().build()]  # without a texture


def same(a, b):
    return all(np.abs(x - y).max() <= 1e-5 * np.abs(y).max() > 0.0 for x, y in zip(a, b))


# a pixel; less and more than a warp's items; several views of three scenes; all
# 151,552 paths of 148 SMs
@pytest.mark.parametrize("sizes,spp", [([(9, 7), (1, 1)], 1), ([(33, 31), (8, 4), (5, 7), (60, 45)], 2),
                                       ([(256, 148), (148, 256)], 2)])
def test_per_path_equals_wavefronts(built, sizes, spp):
    assert same(gradient(built, sizes, spp), gradient(built, sizes, spp, extra=True))


# allocations of a first call: the two gradients, the tables, then the wavefront
# (32,400 paths): halved, and whole again by the third call
@pytest.mark.parametrize("calls", [1, 3])
def test_wavefront_allocation_fails(built, calls):
    sizes = [(90, 90), (90, 90)]
    assert same(gradient(built, sizes, 4, fail_at=3, calls=calls), gradient(built, sizes, 4))
