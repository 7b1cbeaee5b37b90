"""Rays from far away, where an entry's rounding exceeds the boxes' widening: the walks that
answer short queries, long ones and named widths all equal the FP32 brute force, on rays aimed
inside triangles and at the edges and corners they share (ties go to the smaller id)."""
import numpy as np
import pytest

import luce_render_b200 as lr
from luce_render_b200 import scenes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _sheets():
    """Three coincident grids: every hit a tie."""
    p, t, f = scenes.grid(2.0, 24)
    return [lr.MeshData(p, t, faces=f, face_count=int(f.max()) + 1) for _ in range(3)]


def _aimed(a, count, distance, corners, seed):
    """Rays of `count` random triangles from `distance` times the scene's extent away."""
    rng = np.random.default_rng(seed)
    tri = a["indices"][rng.integers(0, len(a["indices"]), count)]
    weight = rng.dirichlet((1, 1, 1), count)
    if corners:
        weight = np.eye(3)[rng.integers(0, 3, count)]
        weight[::2] = 0.5 * (weight[::2] + np.roll(weight[::2], 1, axis=1))
    target = (a["positions"][tri].astype(np.float64) * weight[:, :, None]).sum(1)
    d = rng.normal(size=(count, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.zeros((count, 8), np.float32)
    rays[:, 0:3] = target - d * distance * float(np.abs(a["positions"]).max())
    rays[:, 4:7] = target - rays[:, 0:3].astype(np.float64)
    rays[:, 7] = 3e38
    return rays


@pytest.mark.parametrize("meshes", [scenes.cornell_meshes, _sheets, lambda: scenes.scene_of_size(6000, 3)[0]])
@pytest.mark.parametrize("distance", [300.0, 1e4, 1e6])
@pytest.mark.parametrize("corners", [False, True])
def test_far_rays_equal_brute_force(ctx, meshes, distance, corners):
    scene = lr.compile_scene(meshes())
    a = scene.arrays()
    rays = _aimed(a, 4096, distance, corners, 3)
    prim, t, _, _ = orc.brute_watertight(a["positions"], a["indices"], a["order"], rays)
    gpu = lr.GpuScene.upload(ctx, scene)
    try:
        for width in (0, 2, 4, 8):
            hits = lr.trace_rays(ctx, gpu, rays, width=width)
            assert np.array_equal(lr.hit_ids(hits), prim), width
            assert np.array_equal(hits[:, 0].view(np.uint32), t.view(np.uint32)), width
    finally:
        gpu.destroy()
    assert np.count_nonzero(prim >= 0) > 3900
