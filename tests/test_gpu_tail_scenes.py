"""The per-path launch against the stage kernels where rays differ most: all
materials, an environment and a terrain, Russian roulette, the physical
estimator, more paths than one per warp.  Every path computes the same either
way, so images are bit-identical."""
import numpy as np
import pytest

import cupbr_b200 as cb
from cupbr_b200 import scenes

pytestmark = pytest.mark.gpu

SCENES = {"mixed": lambda: scenes.material_test_scene(0),
          "terrain": lambda: scenes.heightfield_spheres(0, 65, 64 * 64, 9, 2, env_size=(128, 64))}
_built = {}


def render(name, w, h, tail, rr, physical):
    if name not in _built:
        _built[name] = SCENES[name]().build()
    r = cb.PBRenderer(cb.RenderingMethod.PATHTRACER)
    r.set_output_size(w, h)
    r.register_scene(_built[name])
    r.set_method(cb.RenderingMethod.PATHTRACER)
    r.set_max_trace_depth(7)
    r.set_russian_roulette(rr)
    if physical:
        r.set_estimator("physical")
    r.set_tail_paths(tail)
    for _ in range(2):
        r.render(cb.Camera(w, h))
    assert r.error_count() == 0
    return r.get_output_image().numpy()


# a few paths per warp, and warps full of them with a tail at every depth
@pytest.mark.parametrize("name", sorted(SCENES))
@pytest.mark.parametrize("rr,physical", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("w,h", [(117, 71), (401, 307)])
def test_per_path_launch_same_image(name, w, h, rr, physical):
    stages = render(name, w, h, 0, rr, physical)
    assert stages.any()
    for tail in (1 << 30, 40_000):
        assert np.array_equal(stages, render(name, w, h, tail, rr, physical))
