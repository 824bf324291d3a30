"""How few paths are dealt out over the device: the per-path launch (a warp per
path up to full warps), the choice between it and the stage kernels by the
size of the frame, and the first deal of the traversal queues.  Every path
computes the same whatever warp carries it, so images are bit-identical."""
import numpy as np
import pytest

import cupbr_b200 as cb
from cupbr_b200 import scenes

pytestmark = pytest.mark.gpu


def render(w, h, frames=1, tail=None, pipelined=False, stream=None):
    r = cb.PBRenderer(cb.RenderingMethod.PATHTRACER)
    r.set_output_size(w, h)
    r.register_scene(scenes.cornell_box().build())
    r.set_method(cb.RenderingMethod.PATHTRACER)
    r.set_max_trace_depth(4)
    if tail is not None:
        r.set_tail_paths(tail)
    r.set_pipelined(pipelined)
    if stream is not None:
        r.set_stream(stream)
    cam = cb.Camera(w, h)
    for _ in range(frames):
        r.render(cam)
    if stream is not None:
        stream.synchronize()
    img = r.get_output_image().numpy()
    assert r.error_count() == 0
    return img


# four paths; fewer, as many and more paths than warps fit at once on 148 SMs
# (16 or 20 per SM); 16 paths per warp, where full warps take over, and one
# path less; around 4 and 32 queue entries per traversal warp (32 per SM)
SIZES = [(2, 2), (67, 35), (37, 64), (23, 103), (80, 37), (219, 173), (148, 256), (148, 320), (148, 128), (149, 129),
         (148, 1024), (1031, 147)]


@pytest.mark.parametrize("w,h", SIZES)
def test_few_paths_same_image(w, h):
    assert np.array_equal(render(w, h, tail=0), render(w, h, tail=1 << 30))


# the last frame that is one launch, the first that is not, and one in between
# the two limits of the tail
@pytest.mark.parametrize("w,h", [(627, 627), (768, 512), (256, 129)])
@pytest.mark.parametrize("pipelined", [False, True])
def test_default_choice_same_image(w, h, pipelined):
    assert np.array_equal(render(w, h, 3, 0), render(w, h, 3, None, pipelined))


# the same pipelined on a stream of its own, where frames overlap
@pytest.mark.parametrize("w,h", [(312, 315), (384, 256)])
def test_overlapping_choice_same_image(w, h):
    torch = pytest.importorskip("torch")
    assert np.array_equal(render(w, h, 6, 0), render(w, h, 6, None, True, torch.cuda.Stream()))
