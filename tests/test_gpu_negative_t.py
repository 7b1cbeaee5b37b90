"""Rays whose interval reaches behind their origin (t_min below zero): hits at negative t, ties
among them going to the smaller id, equal the FP32 brute force in every walk, short queries,
long ones and named widths."""
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


@pytest.mark.parametrize("meshes", [scenes.cornell_meshes, _sheets, lambda: scenes.scene_of_size(6000, 3)[0]])
@pytest.mark.parametrize("edges", [False, True])
def test_hits_behind_the_origin_equal_brute_force(ctx, meshes, edges):
    scene = lr.compile_scene(meshes())
    a = scene.arrays()
    extent = float(np.abs(a["positions"]).max())
    count, rng = 4096, np.random.default_rng(5)
    rays = scenes.random_rays(count, 5, -extent, extent)
    rays[:, 3] = -3.0 * extent
    if edges:  # away from points of shared edges behind the origin
        tri = a["indices"][rng.integers(0, len(a["indices"]), count)]
        weight = np.round(8.0 * rng.random((count, 1))) / 8.0
        target = weight * a["positions"][tri[:, 0]] + (1.0 - weight) * a["positions"][tri[:, 1]]
        rays[:, 0:3] = target + rays[:, 4:7] * 3.0 * extent
        rays[:, 4:7] = rays[:, 0:3] - target
        rays[:, 3], rays[:, 7] = -4.0, 0.0
    prim, t, _, _ = orc.brute_watertight(a["positions"], a["indices"], a["order"], rays)
    assert np.count_nonzero(t[prim >= 0] < 0.0) > 300
    gpu = lr.GpuScene.upload(ctx, scene)
    try:
        answers = {width: lr.trace_rays(ctx, gpu, rays, width=width) for width in (0, 2, 4, 8)}
        long = np.tile(rays, (200, 1))  # past the queries that vote
        answers["long"] = lr.trace_rays(ctx, gpu, long)[-count:]
    finally:
        gpu.destroy()
    for name, hits in answers.items():
        assert np.array_equal(lr.hit_ids(hits), prim), name
        assert np.array_equal(hits[prim >= 0, 0].view(np.uint32), t[prim >= 0].view(np.uint32)), name
