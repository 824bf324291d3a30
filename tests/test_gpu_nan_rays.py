"""Rays that are no numbers, among ordinary ones: Scene.trace and visible
report what the oracle does (nothing is hit), lanes beside them keep their own
hits, and frames of a camera at NaN end without an error on every path a frame
can take through the traversal."""
import dataclasses

import numpy as np
import pytest

import cupbr_b200 as cb
from cupbr_b200 import scenes
from oracle.bridge import CheckerScene

pytestmark = pytest.mark.gpu

SCENES = {"cornell": scenes.cornell_box, "mixed": lambda: scenes.material_test_scene(0),
          "terrain": lambda: scenes.heightfield_spheres(0, 33, 1000, 5, 1, env_size=(64, 32))}


@pytest.mark.parametrize("name", sorted(SCENES))
def test_trace_and_visible(name):
    desc = SCENES[name]()
    rng = np.random.default_rng(7)
    n = 4099
    o = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32) + np.float32([0.0, 1.0, 2.0])
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    odd = rng.integers(0, 3, n) == 0
    values = np.float32([np.nan, np.nan, 1e19, -1e19, 0.5])
    o[odd] = values[rng.integers(0, 5, (odd.sum(), 3))]
    o[odd & (rng.integers(0, 6, n) == 0)] = np.inf
    o[odd & (rng.integers(0, 6, n) == 0)] = -np.inf
    d[odd & (rng.integers(0, 3, n) == 0)] = np.float32([0.0, 1.0, 0.0])
    d[odd & (rng.integers(0, 6, n) == 0)] = np.nan
    d[odd & (rng.integers(0, 6, n) == 0)] = np.inf
    dist = np.full(n, 3.0, np.float32)
    sc, ref = desc.build(), CheckerScene(desc, "oracle")
    t, obj, tri = sc.trace(o, d)
    rt, robj, rtri, _, _ = ref.trace(o, d)
    assert np.array_equal(t, rt) and np.array_equal(obj, robj) and np.array_equal(tri, rtri)
    assert np.array_equal(sc.visible(o, d, dist), ref.visible(o, d, dist))
    assert (obj[odd] < 0).mean() > 0.9 and (obj[~odd] >= 0).any()


def renderer(desc, method, w=67, h=45):
    r = cb.PBRenderer(method)
    r.set_output_size(w, h)
    r.register_scene(desc.build())
    r.set_method(method)
    r.set_max_trace_depth(4)
    return r


def nan_camera(w, h):
    c = cb.Camera(w, h)
    return cb.Camera.from_axes((float("nan"),) * 3, c.x_axis(), c.y_axis(), c.z_axis())


@pytest.mark.parametrize("name", sorted(SCENES))
@pytest.mark.parametrize("tail", [None, 0])
@pytest.mark.parametrize("frames", [1, 3])
def test_pathtracer_camera_at_nan(name, tail, frames):
    r = renderer(SCENES[name](), cb.RenderingMethod.PATHTRACER)
    if tail is not None:
        r.set_tail_paths(tail)
    r.render_frames(nan_camera(67, 45), frames)
    r.get_output_image().numpy()
    assert r.error_count() == 0


@pytest.mark.parametrize("method", ["VOLUME", "GRADIENTDOMAIN", "RAYTRACER"])
def test_other_methods_camera_at_nan(method):
    r = renderer(scenes.cornell_box(), cb.RenderingMethod[method])
    r.render(nan_camera(67, 45))
    r.get_output_image().numpy()
    assert r.error_count() == 0


@pytest.mark.parametrize("mode", ["wavefront", "persistent", "cooperative"])
def test_batch_camera_at_nan(mode):
    torch = pytest.importorskip("torch")
    sc = scenes.cornell_box().build()
    images = [torch.zeros((45, 67, 3), device="cuda") for _ in range(2)]
    cams = [cb.Camera(67, 45), nan_camera(67, 45)]
    b = cb.Batch([dict(scene=sc, camera=c, width=67, height=45, spp=2, frame0=0, image=i.data_ptr())
                  for c, i in zip(cams, images)], 4)
    b.set_mode(mode)
    b.launch()
    torch.cuda.synchronize()
    assert b.error_count() == 0
    assert torch.isfinite(images[0]).all() and images[0].mean() > 0.0


# a GGX surface of NaN roughness sends its paths on from NaN positions
@pytest.mark.parametrize("tail", [None, 0])
def test_paths_that_turn_nan(tail):
    desc = scenes.cornell_box()
    objects = [dataclasses.replace(o) for o in desc.objects]
    for o in objects[::2]:
        o.material = dataclasses.replace(o.material, type=scenes.GGX, roughness=float("nan"))
    r = renderer(dataclasses.replace(desc, objects=objects), cb.RenderingMethod.PATHTRACER)
    if tail is not None:
        r.set_tail_paths(tail)
    r.render(cb.Camera(67, 45))
    r.get_output_image().numpy()
    assert r.error_count() == 0
