"""The BVH2 walk of long queues (a warp votes between nodes and leaves, and refills finished
lanes): a long query's answers are those of the same rays asked in short queries, which take
the plain walk, bit for bit -- any-hit ids included, since a ray's own order of visits is the
same. 800,003 rays are more than 2.5 times the lanes the GPU holds, and end inside a warp's batch;
50,000 are fewer."""
import numpy as np
import pytest

import luce_render_b200 as lr
from luce_render_b200 import scenes

pytestmark = pytest.mark.gpu

LONG, SHORT = 800_003, 50_000


@pytest.mark.parametrize("triangles", [34, 60_000, 150_000, 500_000])
@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("camera", [False, True])
def test_long_query_equals_short_ones(triangles, any_hit, camera):
    if triangles == 34:
        scene, extent = lr.compile_scene(scenes.cornell_meshes()), 0.6  # some rays start outside and miss
    else:
        meshes, materials, lights, cam = scenes.scene_of_size(triangles, 5)
        scene, extent = lr.compile_scene(meshes, [cam], lights, materials), 50.0 * (triangles / 2**20) ** (1 / 3)
    rays = scenes.random_rays(LONG, 11, -extent, extent)
    if camera:  # whole batches along one octant, which smaller scenes walk plainly, and mixed ones
        rays[:, 4:7] = np.abs(rays[:, 4:7]) * np.where(np.arange(LONG)[:, None] % 1000 < 900, 1.0, rays[:, 4:7])
    rays[::7, 7] = 0.25 * extent  # some end before what they would hit
    ctx = lr.Context(0)
    gpu = lr.GpuScene.upload(ctx, scene)
    whole = lr.trace_rays(ctx, gpu, rays, any_hit=any_hit)
    parts = [lr.trace_rays(ctx, gpu, rays[i:i + SHORT], any_hit=any_hit) for i in range(0, LONG, SHORT)]
    gpu.destroy()
    ctx.close()
    assert np.array_equal(whole.view(np.uint32), np.concatenate(parts).view(np.uint32))
    assert 0 < np.count_nonzero(lr.hit_ids(whole) >= 0) < LONG
