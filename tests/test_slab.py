"""The traversal's slab test (cupbr_b200/csrc/slab.hpp) on the CPU, for rays
whose components are no numbers, infinite, huge, zero or denormal as well as
ordinary ones: a ray that may walk a tree never enters a missing child, whose
reference leads out of the tables; a ray of ordinary numbers walks, and enters
a box exactly when it meets it."""
import itertools
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
BOX = np.array([1.0, 0.5, -2.0, 1.0, 3.0, 0.25], np.float32)  # x in [0.5, 1.5], y in [-3, -1], z in [2.75, 3.25]


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("slab")
    exe = str(d / "slab_harness")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "cupbr_b200", "csrc"),
                    os.path.join(HERE, "slab_harness.cpp"), "-o", exe], check=True, capture_output=True)

    def go(rays):
        np.ascontiguousarray(rays, np.float32).tofile(d / "rays.bin")
        BOX.tofile(d / "box.bin")
        subprocess.run([exe, str(d / "rays.bin"), str(d / "box.bin"), str(d / "out.bin")], check=True)
        return np.fromfile(d / "out.bin", np.int32).reshape(-1, 3).astype(bool)
    return go


def test_no_walking_ray_enters_a_missing_child(run):
    o = [np.nan, np.inf, -np.inf, 0.0, -0.0, 1.5, -3e38, 1e19, 1e-42]
    d = [np.nan, np.inf, -np.inf, 0.0, -0.0, 0.6, -3e38, 1e-42]
    rays = np.array([a + b for a in itertools.product(o, repeat=3) for b in itertools.product(d, repeat=3)], np.float32)
    walks, missing, _ = run(rays).T
    assert not (walks & missing).any()
    assert missing.any()  # it is the question slab_walks that keeps those out
    # a ray that is not a number, or nowhere, meets nothing and need not walk
    assert not walks[~np.isfinite(rays[:, :3]).all(axis=1)].any()


def test_ordinary_rays_walk_and_hit(run):
    rng = np.random.default_rng(3)
    n = 20000
    o = rng.uniform(-6.0, 6.0, (n, 3))
    target = BOX[[0, 2, 4]] + rng.uniform(-2.5, 2.5, (n, 3)) * BOX[[1, 3, 5]]
    d = target - o
    d[rng.integers(0, 40, n) == 0, 0] = 0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([o, d], axis=1).astype(np.float32)
    walks, missing, hit = run(rays).T
    assert walks.all() and not missing.any()
    # the interval in 64 bits for boxes 1e-4 smaller and larger, far above the
    # rounding of 12 operations on values below 100 (about 1e-5)
    o, d = rays[:, :3].astype(np.float64), rays[:, 3:].astype(np.float64)
    d = np.where(d == 0.0, 1e-20, d)
    for grow, wanted in ((-1e-4, lambda m: hit[m].all()), (1e-4, lambda m: not hit[~m].any())):
        lo = (BOX[[0, 2, 4]] - BOX[[1, 3, 5]] - grow - o) / d
        hi = (BOX[[0, 2, 4]] + BOX[[1, 3, 5]] + grow - o) / d
        inside = np.maximum(np.minimum(lo, hi).max(axis=1), 0.0) <= np.maximum(lo, hi).min(axis=1)
        assert 1000 < inside.sum() < n - 1000
        assert wanted(inside)
