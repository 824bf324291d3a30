"""Texture adjoint split into several wavefronts: an allocation that fails
inside cupbr_batch_backward halves its wavefronts instead of failing the call.
Bar: the gradient of the undisturbed call up to the order of the float
additions (a texel sums at most a few thousand terms: 1e-5 of the largest)."""
import numpy as np
import pytest

import cupbr_b200 as cb
from cupbr_b200 import _native as N
from cupbr_b200 import scenes

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def gradient(scene, grads, fail_at=None):
    sizes = [(96, 80), (75, 61)]
    imgs = [torch.zeros((h, w, 3), device="cuda") for w, h in sizes]
    batch = cb.Batch([dict(scene=scene, camera=cb.Camera(w, h), width=w, height=h, spp=3 + i, frame0=0,
                           image=img.data_ptr()) for i, ((w, h), img) in enumerate(zip(sizes, imgs))], 5)
    try:
        if fail_at is not None:
            N.call("cupbr_debug_fail_allocation", fail_at)
        batch.backward([g.data_ptr() if g is not None else 0 for g in grads])
    finally:
        N.call("cupbr_debug_fail_allocation", -1)
    torch.cuda.synchronize()
    return torch.as_tensor(batch.texture_gradient(scene), device="cuda").cpu().numpy()


@pytest.mark.parametrize("skip", [None, 0, 1])  # the view without an image gradient
def test_split_wavefronts_give_the_same_gradient(skip):
    scene = scenes.with_texture(scenes.cornell_variant(5), 16, seed=17).build()
    g = torch.Generator(device="cuda").manual_seed(2)
    grads = [torch.rand((h, w, 3), generator=g, device="cuda") - 0.5 for w, h in ((96, 80), (75, 61))]
    grads[0][:40] = 0.0  # paths of weight 0 are not traced
    if skip is not None:
        grads[skip] = None
    ref = gradient(scene, grads)
    assert np.abs(ref).max() > 0.0
    # allocations of the call: the gradient, the image table, the segments, then the wavefront's buffers
    for fail_at in (3, 5, 11):
        got = gradient(scene, grads, fail_at)
        assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()
