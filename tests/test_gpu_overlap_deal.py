"""Pipelined frames on a stream of their own, whose traversal warps take 32 rays
of a short queue where others deal the whole queue out a few rays to a warp:
images are bit-identical to those of frames rendered one by one."""
import numpy as np
import pytest

import cupbr_b200 as cb
from cupbr_b200 import scenes

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SCENES = {"cornell": scenes.cornell_box, "mixed": lambda: scenes.material_test_scene(0),
          "volume": scenes.volume_test_scene}


def render(scene, method, w, h, stream, **k):
    r = cb.PBRenderer(method)
    r.set_output_size(w, h)
    r.register_scene(scene)
    r.set_method(method)
    r.set_max_trace_depth(5)
    r.set_russian_roulette(k.get("rr", False))
    if k.get("physical"):
        r.set_estimator("physical")
    if stream is not None:
        r.set_pipelined(True)
        r.set_stream(stream)
        r.set_tail_paths(0)
    for _ in range(6):
        r.render(cb.Camera(w, h))
    if stream is not None:
        stream.synchronize()
    assert r.error_count() == 0
    return r.get_output_image().numpy()


# queues of less than a ray, of 4 to 32 and of more than 32 rays per warp (4,736 warps on 148 SMs)
@pytest.mark.parametrize("name,method,w,h,options", [
    ("cornell", "PATHTRACER", 61, 43, {}), ("cornell", "PATHTRACER", 400, 301, {}),
    ("mixed", "PATHTRACER", 333, 222, dict(rr=True, physical=True)), ("mixed", "PATHTRACER", 640, 360, dict(rr=True)),
    ("volume", "VOLUME", 251, 187, {}), ("cornell", "GRADIENTDOMAIN", 150, 101, {})])
def test_overlapping_frames_same_image(name, method, w, h, options):
    scene = SCENES[name]().build()
    m = cb.RenderingMethod[method]
    assert np.array_equal(render(scene, m, w, h, None, **options), render(scene, m, w, h, torch.cuda.Stream(), **options))
