"""Short queries, walked a warp a ray, of rays that are not unit vectors with an open interval: no,
infinite and NaN components, zero and denormal directions, bounded and empty intervals. They
answer as the FP32 brute force does and end. After a refit of moved points they answer from the
moved triangles, as probes do."""
import numpy as np
import pytest

import luce_render_b200 as lr
from luce_render_b200 import scenes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

COUNT = 1024


def _odd(kind, extent):
    rng = np.random.default_rng(9)
    rays = scenes.random_rays(COUNT, 5, -extent, extent)
    rays[:, 7] = np.inf
    rows, axis = np.arange(COUNT), rng.integers(0, 3, COUNT)
    if kind == "axis":
        rays[:, 4:7] = 0.0
        rays[rows, 4 + axis] = rng.choice([-1.0, 1.0], COUNT)
    elif kind == "zero direction":
        rays[:, 4:7] = 0.0
    elif kind == "denormal direction":
        rays[:, 4:7] *= 1e-42
    elif kind == "huge direction":
        rays[:, 4:7] *= 1e30
    elif kind == "NaN direction":
        rays[rows, 4 + axis] = np.nan
    elif kind == "infinite direction":
        rays[rows, 4 + axis] = np.inf
    elif kind == "NaN origin":
        rays[rows, axis] = np.nan
    elif kind == "infinite origin":
        rays[rows, axis] = -np.inf
    elif kind == "NaN interval":
        rays[rows, np.where(rows % 2 == 0, 3, 7)] = np.nan
    elif kind == "interval":
        rays[:, 3] = rng.uniform(0.0, extent, COUNT)
        rays[:, 7] = rays[:, 3] + extent
    elif kind == "empty interval":
        rays[:, 3], rays[:, 7] = 5.0, 1.0
    return rays


def _equal(hits, prim, t, u, v):
    assert np.array_equal(lr.hit_ids(hits), prim)
    assert np.array_equal(hits[:, 0].view(np.uint32), t.view(np.uint32))
    hit = prim >= 0
    assert np.array_equal(hits[hit, 2].view(np.uint32), u[hit].view(np.uint32))
    assert np.array_equal(hits[hit, 3].view(np.uint32), v[hit].view(np.uint32))


@pytest.mark.parametrize("kind", ["open interval", "axis", "zero direction", "denormal direction", "huge direction",
                                  "NaN direction", "infinite direction", "NaN origin", "infinite origin", "NaN interval",
                                  "interval", "empty interval"])
@pytest.mark.parametrize("meshes", [scenes.cornell_meshes, lambda: scenes.scene_of_size(6000, 3)[0]])
def test_odd_rays_equal_brute_force(ctx, kind, meshes):
    scene = lr.compile_scene(meshes())
    a = scene.arrays()
    rays = _odd(kind, float(np.abs(a["positions"]).max()))
    gpu = lr.GpuScene.upload(ctx, scene)
    try:
        hits = lr.trace_rays(ctx, gpu, rays)
    finally:
        gpu.destroy()
    _equal(hits, *orc.brute_watertight(a["positions"], a["indices"], a["order"], rays))


@pytest.mark.parametrize("triangles", [34, 6000, 60_000])
def test_short_queries_follow_a_refit(ctx, triangles):
    if triangles == 34:
        scene = lr.compile_scene(scenes.cornell_meshes())
    else:
        scene = lr.compile_scene(scenes.scene_of_size(triangles, 3)[0])
    before = scene.arrays()["positions"].astype(np.float64)
    extent = float(np.abs(before).max())
    moved = (before * 1.5 + 0.1 * extent * np.sin(3.0 / extent * before[:, [1, 2, 0]])).astype(np.float32)
    gpu = lr.GpuScene.upload(ctx, scene)
    frame = lr.look_frame((0.0, 0.0, 4.0 * extent), (0.02, -0.01, -1.0), (0.0, 1.0, 0.0), 0.4, 48, 40)
    rays = np.concatenate([scenes.random_rays(COUNT, 7, -extent, extent), scenes.frame_rays(frame)])
    try:
        gpu.refit(ctx, moved)
        hits = lr.trace_rays(ctx, gpu, rays)
        _, distances = lr.probe(ctx, gpu, frame)
    finally:
        gpu.destroy()
    scene.move_points(moved)
    a = scene.arrays()
    want = orc.brute_watertight(a["positions"], a["indices"], a["order"], rays)
    _equal(hits, *want)
    assert np.array_equal(distances.view(np.uint32), want[1][COUNT:].view(np.uint32))
