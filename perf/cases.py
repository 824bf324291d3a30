"""The measured work: what a program that renders with cupbr_b200 has it do.

Twelve listed cases, one per way the framework is used, and draw(), which
gives more of the same kinds with sizes spread over the ranges below.  Every
case goes through the public entry points (PBRenderer, ToneMapper,
PostProcessor, Batch, medium.Medium / medium.render, cache.RadianceCache).

prepare() is what such a program holds before it renders: a committed scene,
a renderer with its output size, device images and buffers.  Geometry that
does not depend on the seed (the terrain meshes, the sky) is generated once
per process, as a program loads its meshes once; materials, wall colours,
camera poses, density grids, images and training samples come from the seed.
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

import cupbr_b200 as cb
from cupbr_b200 import medium as grid_medium
from cupbr_b200 import scenes
from cupbr_b200.cache import LAYERS, RadianceCache

METHOD = cb.RenderingMethod
CURVE = (1.0, 1.0)  # bloom threshold and knee


def listed():
    return [
        # the smallest call: one interactive preview sample of a small scene, tone mapped for display
        dict(name="preview_cornell_256", kind="viewer", scene="cornell", w=256, h=256, depth=5, frames=1,
             pipelined=False, physical=False, rr=False),
        # an interactive viewer: one sample per displayed frame, pipelined, each tone mapped; the physical
        # estimator (environment sampling with MIS) and Russian roulette on, a ragged window size
        dict(name="viewer_terrain_physical_1273x717", kind="viewer", scene="terrain", grid=257, spheres=40, subdiv=3,
             w=1273, h=717, depth=8, frames=4, pipelined=True, physical=True, rr=True),
        # offline rendering of the Cornell box: 512 x 512, 64 samples per pixel, depth 5
        dict(name="render_cornell_512", kind="render", scene="cornell", w=512, h=512, depth=5, frames=64),
        # offline rendering of the 2,024,000-triangle scene: 1080p, depth 8, 16 samples per pixel
        dict(name="render_terrain_1080p", kind="render", scene="terrain", grid=1024, spheres=200, subdiv=4, w=1920,
             h=1080, depth=8, frames=16),
        # the VOLUME method on its test scene (homogeneous media, glass, mirror, point and area light)
        dict(name="volume_512", kind="volume", w=512, h=512, depth=5, frames=32),
        # gradient-domain rendering: base and shift paths and the reconstruction of every frame
        dict(name="gdpt_512", kind="gdpt", w=512, h=512, depth=5, frames=8),
        # the density-grid medium, forward: 256^3 voxels, analog delta tracking
        dict(name="medium_forward_256", kind="medium", res=256, w=512, h=512, depth=5, spp=16),
        # inverse rendering of the medium: forward, L2 loss and the gradients of every voxel and scene parameter
        dict(name="medium_gradient_128", kind="medium_grad", res=128, w=256, h=256, depth=5, spp=16),
        # post-processing of a large still: bloom with the fused Reinhard tone map, 7680 x 4320
        dict(name="post_fused_8k", kind="post_fused", w=7680, h=4320, gamma=False),
        # post-processing of a viewer's frame at a laptop panel's width: bloom to HDR, then the tone map
        dict(name="post_separate_1366x768", kind="post_separate", w=1366, h=768, gamma=True),
        # many views of textured scenes in one launch, and the gradient of the textures
        dict(name="batch_texture_gradient", kind="batch", scenes=3, views=4, grid=257, side=256, spp=16, depth=5),
        # the radiance cache: answers a batch of records, renders cached frames, takes a frame's four Adam steps
        dict(name="cache_terrain_960x540", kind="cache", grid=513, spheres=100, subdiv=3, w=960, h=540, depth=8,
             frames=4, records=1 << 20, batch=1 << 14, steps=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["viewer", "viewer", "render", "render", "volume", "gdpt", "medium", "medium_grad", "post_fused",
                       "post_separate", "batch", "cache"])
    w = _log(rng, 200, 1900)
    h = max(64, int(w * rng.uniform(0.5, 1.0)))
    depth = rng.randint(3, 8)

    def frames(budget, most):  # whole frames of w x h within a budget of paths
        return max(1, min(_log(rng, 1, most), budget // (w * h)))

    if kind in ("viewer", "render"):
        case = dict(kind=kind, scene=rng.choice(["cornell", "terrain", "mixed"]), w=w, h=h, depth=depth)
        if case["scene"] == "terrain":
            case.update(grid=_log(rng, 100, 700), spheres=rng.randint(10, 100), subdiv=rng.choice([2, 3]))
        if kind == "render":
            case.update(frames=frames(16_000_000, 64))
        else:
            case.update(frames=frames(8_000_000, 6), pipelined=rng.random() < 0.5, physical=rng.random() < 0.5,
                        rr=rng.random() < 0.5)
        return case
    if kind == "volume":
        return dict(kind=kind, w=w, h=h, depth=depth, frames=frames(8_000_000, 32))
    if kind == "gdpt":
        return dict(kind=kind, w=w, h=h, depth=depth, frames=frames(2_000_000, 12))
    if kind == "medium":
        w = _log(rng, 128, 900)
        return dict(kind=kind, res=_log(rng, 48, 256), w=w, h=max(64, int(w * rng.uniform(0.5, 1.0))),
                    depth=rng.randint(3, 6), spp=max(1, min(_log(rng, 1, 32), 4_000_000 // (w * w))))
    if kind == "medium_grad":
        w = _log(rng, 96, 400)
        return dict(kind=kind, res=_log(rng, 32, 160), w=w, h=max(64, int(w * rng.uniform(0.5, 1.0))),
                    depth=rng.randint(3, 6), spp=max(1, min(_log(rng, 2, 32), 1_200_000 // (w * w))))
    if kind in ("post_fused", "post_separate"):
        w = _log(rng, 300, 7680)
        return dict(kind=kind, w=w, h=max(2, int(w * rng.uniform(0.45, 0.75))), gamma=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(1, 3), views=rng.randint(1, 4), grid=_log(rng, 100, 300),
                    side=_log(rng, 90, 260), spp=_log(rng, 2, 16), depth=rng.randint(3, 5))
    w = _log(rng, 200, 960)
    return dict(kind="cache", grid=_log(rng, 100, 513), spheres=rng.randint(10, 100), subdiv=rng.choice([2, 3]), w=w,
                h=max(64, int(w * rng.uniform(0.5, 1.0))), depth=depth, frames=rng.randint(1, 4),
                records=_log(rng, 1 << 12, 1 << 20), batch=128 * rng.randint(8, 128), steps=rng.randint(1, 4))


# ------------------------------------------------------------------ scenes

@functools.lru_cache(maxsize=6)
def _terrain(grid, spheres, subdiv):
    """The seeded heightfield with icospheres, its chunks scaled so that a
    smaller terrain keeps the large one's extent; cropped as the
    2,024,000-triangle scene is (1,000,000 of its 2,093,058 triangles)."""
    crop = 1_000_000 if grid == 1024 else (grid - 1) * (grid - 1)
    return scenes.heightfield_spheres(seed=0, grid=grid, crop=crop, n_spheres=spheres, subdiv=subdiv)


@functools.lru_cache(maxsize=1)
def _mixed():
    return scenes.material_test_scene(env_size=(512, 256))


def _desc(name, seed, case):
    """A scene description with the seed's materials."""
    if name == "cornell":
        return scenes.cornell_variant(seed)
    rng = np.random.default_rng(seed)
    if name == "terrain":
        base = _terrain(case["grid"], case.get("spheres", 20), case.get("subdiv", 2))
        return dataclasses.replace(base, objects=[dataclasses.replace(o, material=scenes.random_material(rng))
                                                  for o in base.objects])
    base = _mixed()
    objects = []
    for o in base.objects:
        m = o.material
        if m.type in (scenes.LAMBERT, scenes.PHONG):
            m = dataclasses.replace(m, albedo_d=tuple(rng.uniform(0.1, 0.9, 3).astype(np.float32).tolist()))
        elif m.type == scenes.GGX:
            m = dataclasses.replace(m, roughness=float(np.float32(rng.uniform(0.05, 0.5))))
        objects.append(dataclasses.replace(o, material=m))
    return dataclasses.replace(base, objects=objects)


def _camera(name, w, h, seed):
    """The default camera, moved a little: within the open side of the room,
    or over the terrain."""
    rng = np.random.default_rng((seed, 7))
    base = cb.Camera(w, h)
    p = (rng.uniform(-4, 4), rng.uniform(0.5, 2.0), rng.uniform(-1, 3)) if name == "terrain" else \
        rng.uniform(-0.3, 0.3, 3)
    return cb.Camera.from_axes(tuple(float(v) for v in p), base.x_axis(), base.y_axis(), base.z_axis())


def _renderer(method, scene, case):
    r = cb.PBRenderer(method)
    r.set_output_size(case["w"], case["h"])
    r.register_scene(scene)
    r.set_method(method)
    r.set_max_trace_depth(case["depth"])
    r.set_russian_roulette(bool(case.get("rr", False)))
    if case.get("physical"):
        r.set_estimator("physical")
    if case.get("pipelined"):
        r.set_pipelined(True)
    return r


def _view(image):
    return torch.as_tensor(image, device="cuda")


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _density(res, seed, sigma_max=8.0, octaves=4):
    """(res, res, res) densities in [0, sigma_max]: octaves of smooth noise,
    the lattice doubling and the amplitude halving from one to the next."""
    g = _generator(seed)
    total = torch.zeros((1, 1, res, res, res), device="cuda")
    n, amp = 5, 1.0
    for _ in range(octaves):
        lattice = torch.randn((1, 1, n, n, n), generator=g, device="cuda")
        total += amp * torch.nn.functional.interpolate(lattice, size=(res,) * 3, mode="trilinear", align_corners=True)
        n, amp = min(2 * n, res), 0.5 * amp
    total -= total.min()
    return (total * (sigma_max / total.max())).clamp_(0.0, sigma_max)[0, 0].contiguous()


# ------------------------------------------------------------------ states

def prepare(case, seed):
    return _PREPARE[case["kind"]](case, int(seed))


def run(state):
    return state["run"](state)


def _prepare_viewer(case, seed):
    scene = _desc(case["scene"], seed, case).build()
    r = _renderer(METHOD.PATHTRACER, scene, case)
    tone = cb.ToneMapper(cb.ToneMappingType.REINHARD)
    hdr = r.get_output_image()
    tone.register_image(hdr)
    return dict(run=_run_viewer, renderer=r, tone=tone, camera=_camera(case["scene"], case["w"], case["h"], seed),
                frames=case["frames"], out=(_view(hdr), _view(tone.get_render_buffer())))


def _run_viewer(s):
    for _ in range(s["frames"]):
        s["renderer"].render(s["camera"])
        s["tone"].tone_map()
    return s["out"]


def _prepare_render(case, seed):
    scene = _desc(case["scene"], seed, case).build()
    r = _renderer(METHOD.PATHTRACER, scene, case)
    return dict(run=_run_frames, renderer=r, camera=_camera(case["scene"], case["w"], case["h"], seed),
                frames=case["frames"], out=_view(r.get_output_image()))


def _run_frames(s):
    s["renderer"].render_frames(s["camera"], s["frames"])
    return s["out"]


def _prepare_volume(case, seed):
    rng = np.random.default_rng(seed)
    medium = (tuple(rng.uniform(0.02, 0.08, 3)), tuple(rng.uniform(0.01, 0.03, 3)), float(rng.uniform(0.0, 0.5)))
    scene = scenes.volume_test_scene(medium).build()
    r = _renderer(METHOD.VOLUME, scene, case)
    return dict(run=_run_frames, renderer=r, camera=_camera("volume", case["w"], case["h"], seed),
                frames=case["frames"], out=_view(r.get_output_image()))


def _prepare_gdpt(case, seed):
    scene = scenes.cornell_variant(seed).build()
    r = _renderer(METHOD.GRADIENTDOMAIN, scene, case)
    return dict(run=_run_gdpt, renderer=r, camera=_camera("cornell", case["w"], case["h"], seed), frames=case["frames"])


def _run_gdpt(s):
    r = s["renderer"]
    r.render_frames(s["camera"], s["frames"])
    # the gradient images are there once a frame has been rendered
    return _view(r.get_output_image()), _view(r.get_gradient_x()), _view(r.get_gradient_y())


BOX = ((-1.0, -1.0, 1.0), (1.0, 1.0, 3.0))  # the inside of the Cornell box


def _prepare_medium(case, seed):
    scene = scenes.cornell_variant(seed).build()
    res = case["res"]
    m = grid_medium.Medium((res, res, res), BOX, 8.0, albedo=0.9, g=0.3, q=0.0)
    return dict(run=_run_medium, medium=m, scene=scene, density=_density(res, seed), case=case,
                camera=_camera("cornell", case["w"], case["h"], seed),
                image=torch.zeros((case["h"], case["w"], 3), device="cuda"))


def _run_medium(s):
    c = s["case"]
    s["medium"].forward(s["scene"], s["density"].data_ptr(), s["camera"], c["w"], c["h"], c["spp"], 0, c["depth"],
                        s["image"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return s["image"]


def _prepare_medium_grad(case, seed):
    scene = scenes.cornell_variant(seed).build()
    res = case["res"]
    m = grid_medium.Medium((res, res, res), BOX, 8.5, albedo=0.9, g=0.3, q=0.5)
    target = torch.rand((case["h"], case["w"], 3), generator=_generator(seed), device="cuda")
    return dict(run=_run_medium_grad, medium=m, scene=scene, density=_density(res, seed).requires_grad_(True),
                params=torch.from_numpy(m.params(scene)).cuda().requires_grad_(True), target=target, case=case,
                camera=_camera("cornell", case["w"], case["h"], seed))


def _run_medium_grad(s):
    c = s["case"]
    s["density"].grad = s["params"].grad = None
    image = grid_medium.render(s["density"], s["params"], s["medium"], s["scene"], s["camera"], c["w"], c["h"],
                               c["spp"], 0, c["depth"])
    ((image - s["target"]) ** 2).mean().backward()
    return image.detach(), s["density"].grad, s["params"].grad


def _hdr(w, h, seed):
    """A smooth image with bright spots, values up to 8 as a path tracer's frame of the terrain has."""
    g = _generator(seed)
    low = torch.rand((1, 3, max(2, h // 24), max(2, w // 24)), generator=g, device="cuda")
    img = torch.nn.functional.interpolate(low, size=(h, w), mode="bilinear", align_corners=True)[0].permute(1, 2, 0)
    noise = torch.rand((h, w, 3), generator=g, device="cuda")
    return ((2.0 * img * (0.75 + 0.5 * noise)).clamp(0.0, 2.0) ** 3).contiguous()


def _tone_type(case):
    return cb.ToneMappingType.GAMMA if case["gamma"] else cb.ToneMappingType.REINHARD


def _prepare_post_fused(case, seed):
    w, h = case["w"], case["h"]
    hdr = _hdr(w, h, seed)
    rgba = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
    pp = cb.PostProcessor()
    pp.register_image(cb.DeviceImage(hdr.data_ptr(), w, h, 3, np.float32, owner=hdr))
    return dict(run=_run_post_fused, pp=pp, hdr=hdr, type=_tone_type(case), rgba=rgba, curve=cb.threshold_curve(*CURVE),
                target=cb.DeviceImage(rgba.data_ptr(), w, h, 4, np.uint8, owner=rgba))


def _run_post_fused(s):
    s["pp"].bloom_tonemap(s["curve"], s["type"], 1.0, s["target"])
    return s["rgba"]


def _prepare_post_separate(case, seed):
    w, h = case["w"], case["h"]
    hdr = _hdr(w, h, seed)
    pp = cb.PostProcessor()
    pp.register_image(cb.DeviceImage(hdr.data_ptr(), w, h, 3, np.float32, owner=hdr))
    bloomed = pp.get_post_process_buffer()
    tone = cb.ToneMapper(_tone_type(case))
    tone.register_image(bloomed)
    return dict(run=_run_post_separate, pp=pp, hdr=hdr, tone=tone, curve=cb.threshold_curve(*CURVE),
                out=(_view(bloomed), _view(tone.get_render_buffer())))


def _run_post_separate(s):
    s["pp"].bloom(s["curve"])
    s["tone"].tone_map()
    return s["out"]


def _prepare_batch(case, seed):
    """Views of textured Cornell boxes and one textured terrain, the sides
    between half and the whole of `side`, the samples between a quarter and
    the whole of `spp`; the stage kernels' wavefronts (the mode the autotuner
    picks for such views)."""
    rng = np.random.default_rng(seed)
    size = 512
    built, views, images, grads = [], [], [], []
    for k in range(case["scenes"]):
        name = "terrain" if k == 2 else "cornell"
        d = _desc(name, seed + k, case)
        d = dataclasses.replace(d, objects=[dataclasses.replace(o) for o in d.objects])
        built.append(scenes.with_texture(d, size, seed=(seed, k)).build())
        for v in range(case["views"]):
            side = case["side"] if v == 0 else int(case["side"] * (0.5 + 0.5 * ((v * 5) % 7) / 7))
            spp = max(1, case["spp"] >> (v % 3))
            images.append(torch.zeros((side, side, 3), device="cuda"))
            grads.append(torch.from_numpy(rng.uniform(-0.5, 0.5, (side, side, 3)).astype(np.float32)).cuda())
            views.append(dict(scene=built[-1], camera=_camera(name, side, side, seed + 31 * k + v), width=side,
                              height=side, spp=spp, frame0=0, image=images[-1].data_ptr()))
    b = cb.Batch(views, case["depth"])
    b.set_mode("wavefront")
    return dict(run=_run_batch, batch=b, scenes=built, images=images, grads=grads,
                pointers=[g.data_ptr() for g in grads])


def _run_batch(s):
    s["batch"].launch()
    s["batch"].backward(s["pointers"])
    return s["images"], [_view(s["batch"].texture_gradient(sc)) for sc in s["scenes"]]


def _records(n, lo, hi, seed):
    """n vertex records inside the scene's box, with targets (their layout: cupbr_b200/cache.py)."""
    g = _generator(seed)
    unit = lambda: torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)
    uniform = lambda k: torch.rand((n, k), generator=g, device="cuda")
    lo, hi = (torch.from_numpy(np.asarray(v, np.float32)).cuda() for v in (lo, hi))
    r = torch.zeros((n, 20), device="cuda")
    r[:, 0:3] = lo + (hi - lo) * uniform(3)
    r[:, 4:7], r[:, 7:8] = unit(), uniform(1)
    r[:, 8:11] = unit()
    r[:, 11] = torch.randint(1, 9, (n,), generator=g, device="cuda").float()
    r[:, 12:15] = uniform(3)
    # a smooth radiance with noise, as single path samples have
    r[:, 16:19] = r[:, 12:15] * (0.5 + r[:, 1:2].sin().abs()) * (2.0 * uniform(1))
    r[:, 19] = 1.0
    return r


def _prepare_cache(case, seed):
    scene = _desc("terrain", seed, case).build()
    c = RadianceCache(scene, cache_depth=1, batch=case["batch"], samples_per_frame=case["batch"] * case["steps"],
                      seed=seed)
    lo, inv = c.bounds()
    w, h = case["w"], case["h"]
    return dict(run=_run_cache, cache=c, scene=scene, case=case, records=_records(case["records"], lo, lo + 1 / inv, seed),
                samples=_records(case["batch"] * case["steps"], lo, lo + 1 / inv, seed + 1),
                answers=torch.zeros((case["records"], 4), device="cuda"), image=torch.zeros((h, w, 3), device="cuda"),
                camera=_camera("terrain", w, h, seed))


def _run_cache(s):
    c, k = s["cache"], s["case"]
    c.infer(s["records"].data_ptr(), k["records"], s["answers"].data_ptr())
    c.render(s["scene"], s["camera"], k["w"], k["h"], 0, k["frames"], k["depth"], s["image"].data_ptr(), train=False)
    for i in range(k["steps"]):
        c.train_step(s["samples"][i * k["batch"]].data_ptr(), k["batch"])
    return s["answers"], s["image"], c.params()


_PREPARE = {"viewer": _prepare_viewer, "render": _prepare_render, "volume": _prepare_volume, "gdpt": _prepare_gdpt,
            "medium": _prepare_medium, "medium_grad": _prepare_medium_grad, "post_fused": _prepare_post_fused,
            "post_separate": _prepare_post_separate, "batch": _prepare_batch, "cache": _prepare_cache}


# -------------------------------------------------------------------- work

# Mean rays of a path (closest hit and shadow) per bounce it is allowed, and
# floating-point operations of a ray: box tests of the nodes on its way
# (4 boxes of 12 operations each) and a few primitive tests of about 45.
_RAYS_PER_BOUNCE = {"cornell": 1.6, "terrain": 0.45, "mixed": 0.9}
_RAY_FLOPS = {"cornell": 4 * 48 + 4 * 45, "terrain": 14 * 48 + 5 * 45, "mixed": 5 * 48 + 3 * 45}
_TRI_BYTES = 64 + 22  # vertices, edges and normal, and its share of the tree


def _scene_bytes(name, case):
    if name != "terrain":
        return 4096 + (512 * 256 * 12 if name == "mixed" else 0)
    grid = case["grid"]
    terrain = 1_000_000 if grid == 1024 else (grid - 1) ** 2
    return _TRI_BYTES * (terrain + case.get("spheres", 20) * 20 * 4 ** case.get("subdiv", 2)) + 2048 * 1024 * 12


def work(case):
    kind = case["kind"]
    pixels = case.get("w", 0) * case.get("h", 0)
    if kind in ("viewer", "render"):
        rays = pixels * case["frames"] * case["depth"] * _RAYS_PER_BOUNCE[case["scene"]]
        shown = 28 * case["frames"] if kind == "viewer" else 24  # the mean read and written; 4 B shown per frame
        return {"bytes": _scene_bytes(case["scene"], case) + shown * pixels,
                "flops": rays * (_RAY_FLOPS[case["scene"]] + 60)}
    if kind == "volume":
        return {"bytes": 24 * pixels, "flops": pixels * case["frames"] * case["depth"] * 1.6 * 500}
    if kind == "gdpt":
        paths = 5 * pixels * case["frames"] * case["depth"] * 1.6 * (_RAY_FLOPS["cornell"] + 60)
        # five running means, and per frame the reconstruction's inputs once and its output once (50 passes of 27)
        return {"bytes": (5 * 24 + 48) * pixels * case["frames"], "flops": paths + 50 * 81 * pixels * case["frames"]}
    if kind in ("medium", "medium_grad"):
        # about 8 tentative points per flight and per light term, 20 operations each
        paths = pixels * case["spp"] * case["depth"] * 0.8 * (16 * 20 + 2 * _RAY_FLOPS["cornell"] + 60)
        grid = 4 * case["res"] ** 3
        if kind == "medium":
            return {"bytes": grid + 12 * pixels, "flops": paths}
        return {"bytes": 3 * grid + 24 * pixels, "flops": 3 * paths}  # forward, and two replays
    if kind == "post_fused":
        return {"bytes": 16 * pixels, "flops": 70 * pixels}
    if kind == "post_separate":
        return {"bytes": 40 * pixels, "flops": 70 * pixels}
    if kind == "batch":
        flops, total = 0.0, 0.0
        for k in range(case["scenes"]):
            name = "terrain" if k == 2 else "cornell"
            for v in range(case["views"]):
                side = case["side"] if v == 0 else int(case["side"] * (0.5 + 0.5 * ((v * 5) % 7) / 7))
                n = side * side
                total += 24 * n
                flops += 2 * n * max(1, case["spp"] >> (v % 3)) * case["depth"] * _RAYS_PER_BOUNCE[name] * \
                    (_RAY_FLOPS[name] + 60)
            total += _scene_bytes(name, case) + 512 * 512 * (16 + 12)
        return {"bytes": total, "flops": flops}
    network = 2 * sum(o * i for o, i in LAYERS)
    trained = case["batch"] * case["steps"]
    rays = pixels * case["frames"] * 3 * (_RAY_FLOPS["terrain"] + 60)
    return {"bytes": _scene_bytes("terrain", case) + (80 + 16) * case["records"] + 80 * trained + 12 * pixels,
            "flops": network * (case["records"] + pixels * case["frames"] + 3 * trained) + rays}


# ------------------------------------------------------------------- exact

def exact(case, seed):
    """Values in 64 bits where they follow from the inputs by plain formulas:
    the bloomed image and the network's answers.  A rendered image is a sum
    over paths whose every turn depends on single-precision decisions, and
    tone-mapped pixels are whole numbers: None."""
    if case["kind"] == "post_separate":
        return _exact_bloom(_hdr(case["w"], case["h"], int(seed)).double()), None
    if case["kind"] == "cache":
        s = prepare(case, seed)
        lo, inv = s["cache"].bounds()
        return _exact_network(s["cache"].params(), s["records"].double(), lo, inv), None, None
    return None


def _exact_bloom(hdr):
    t, knee = CURVE
    h, w, _ = hdr.shape
    br = hdr.max(dim=2, keepdim=True).values
    rq = (br - (knee - t)).clamp(0.0, 2.0 * knee)
    rq = 0.25 / knee * rq * rq
    level0 = hdr * (torch.maximum(rq, br - t) / br.clamp_min(1e-5))
    x, y = torch.arange(w // 2, device=hdr.device), torch.arange(h // 2, device=hdr.device)
    level1 = sum(level0[2 * y + b][:, 2 * x + a] for a in (0, 1) for b in (0, 1)) / 4.0
    up = torch.zeros_like(hdr)
    cx, cy = torch.arange(w, device=hdr.device) // 2, torch.arange(h, device=hdr.device) // 2
    for du, ku in ((-1, 1.0), (0, 2.0), (1, 1.0)):
        for dv, kv in ((-1, 1.0), (0, 2.0), (1, 1.0)):
            rows, cols = (cy + dv).clamp(0, h // 2 - 1), (cx + du).clamp(0, w // 2 - 1)
            up += ku * kv * level1[rows][:, cols]
    return hdr + up / 16.0 + level0


def _exact_network(params, r, lo, inv):
    lo, inv = (torch.from_numpy(np.asarray(v, np.float64)).cuda() for v in (lo, inv))
    p = ((r[:, 0:3] - lo) * inv).clamp(0.0, 1.0)
    x = torch.zeros((len(r), 96), dtype=torch.float64, device="cuda")
    for a in range(3):
        for j in range(12):
            angle = math.pi * 2.0 ** j * p[:, a]
            x[:, 24 * a + 2 * j], x[:, 24 * a + 2 * j + 1] = angle.sin(), angle.cos()
    x[:, 72:75], x[:, 75:78], x[:, 78], x[:, 79:82] = r[:, 4:7], r[:, 8:11], r[:, 7], r[:, 12:15]
    x[:, 82], x[:, 83] = 1.0, r[:, 11].clamp(0.0, 16.0) / 16.0
    at = 0
    for k, (o, i) in enumerate(LAYERS):
        weight = torch.from_numpy(np.asarray(params[at:at + o * i], np.float64).reshape(o, i)).cuda()
        x = x @ weight.T
        x = x.clamp_min(0.0) if k + 1 < len(LAYERS) else x
        at += o * i
    return torch.cat([x, torch.zeros((len(x), 1), dtype=x.dtype, device=x.device)], dim=1)
