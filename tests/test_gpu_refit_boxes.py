"""A refit of unmoved points writes the upload's boxes again: the 8- and 4-wide trees and the
BVH2 are walked through the same nodes and triangle tests as before it, on trees whose node
counts leave the refit's last warp full, partly full and with one node."""
import numpy as np
import pytest

import luce_render_b200 as lr
from luce_render_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("meshes", [lambda: [lr.MeshData(*scenes._quad((-1, -1, 0), (1, -1, 0), (1, 1, 0), (-1, 1, 0)))],
                                    scenes.cornell_meshes, lambda: scenes.scene_of_size(3000, 2)[0],
                                    lambda: scenes.scene_of_size(40_000, 2)[0]])
def test_unmoved_points_keep_every_box(meshes):
    scene = lr.compile_scene(meshes())
    points = scene.arrays()["positions"]
    extent = float(np.abs(points).max())
    rays = scenes.random_rays(20_000, 3, -extent, extent)
    ctx = lr.Context(0)
    gpu = lr.GpuScene.upload(ctx, scene)

    def walks():
        out = []
        for width in (2, 4, 8):
            hits = lr.trace_rays(ctx, gpu, rays, width=width, count=True)
            out.append((hits.view(np.uint32).tobytes(), lr.trace_counts(ctx)))
        out.append(lr.trace_rays(ctx, gpu, rays).view(np.uint32).tobytes())
        return out

    before = walks()
    gpu.refit(ctx, points)
    assert walks() == before
    # Moved far away and back: nothing of the pose between stays.
    gpu.refit(ctx, points * np.float32(3.0) + np.float32(500.0))
    gpu.refit(ctx, points)
    assert walks() == before
    gpu.destroy()
    ctx.close()
