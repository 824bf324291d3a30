"""Primitive tests of an instrumented frame's shadow rays: a ray that the first
primitive of a leaf blocks has tested that one, not the whole leaf."""
import numpy as np
import pytest

import cupbr_b200 as cb
from cupbr_b200 import scenes

pytestmark = pytest.mark.gpu


def test_blocked_rays_count_the_tests_they_make():
    sc = scenes.SceneDesc(name="blocked")
    white = scenes.MaterialDesc(scenes.LAMBERT)
    sc.add(scenes.ObjectDesc(scenes.QUAD, white, p0=(0, -1, 2), p1=(0, 1, 0), p2=(1, 0, 0), p3=(0, 0, 1)))
    # four times the same tilted triangle, above the camera and the floor, seen from its back
    v = np.array([(-60, 0.3, -40), (0, 0.9, 90), (60, 0.4, -40)], np.float32)
    sc.add(scenes.ObjectDesc(scenes.MESH, white, vertices=v, indices=np.array([[0, 1, 2]] * 4, np.uint32)))
    sc.lights.append(scenes.LightDesc(scenes.POINT, position=(0.0, 3.0, 2.0), intensity=(1.0, 1.0, 1.0)))
    r = cb.PBRenderer(cb.RenderingMethod.PATHTRACER)
    r.set_output_size(64, 48)
    r.register_scene(sc.build(dict(max_leaf_size=4)))
    r.set_method(cb.RenderingMethod.PATHTRACER)
    r.set_max_trace_depth(1)
    r.set_instrumented(True)
    r.render(cb.Camera(64, 48))
    s = r.stats()
    assert s["shadow_rays"] > 200 and not r.get_output_image().numpy().any()
    # one triangle, and the floor the ray starts on
    assert s["shadow_rays"] <= s["shadow_prims"] <= 2 * s["shadow_rays"]
