"""Small host-side queries stage in memory their context keeps (up to 8 MiB), and small probes
walk a warp a pixel: answers equal the reference path's frames and the larger queries', at sizes
around the staging's growth and its end, and the staging holds nothing over from call to call."""
import numpy as np
import pytest

import luce_render_b200 as lr
from luce_render_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def placed():
    meshes, materials, lights, cam = scenes.scene_of_size(20_000, 4)
    scene = lr.compile_scene(meshes, [cam], lights, materials)
    ctx = lr.Context(0)
    gpu = lr.GpuScene.upload(ctx, scene)
    yield ctx, gpu
    gpu.destroy()
    ctx.close()


def test_rays_around_the_staging_sizes(placed):
    ctx, gpu = placed
    most = (8 << 20) // 48
    rays = scenes.random_rays(most + 1, 6, -13.0, 13.0)
    whole = lr.trace_rays(ctx, gpu, rays)  # past the staging
    for count in (1, 1365, 1366, most, 7):  # 64 KiB is 1,365 rays
        assert np.array_equal(lr.trace_rays(ctx, gpu, rays[:count]).view(np.uint32), whole[:count].view(np.uint32))
        back = lr.trace_rays(ctx, gpu, rays[most + 1 - count:])
        assert np.array_equal(back.view(np.uint32), whole[most + 1 - count:].view(np.uint32))


@pytest.mark.parametrize("width, height", [(1, 1), (3, 1), (5, 7), (64, 63), (97, 95), (1024, 1024), (1024, 1025)])
@pytest.mark.parametrize("reference", [False, True])
def test_probes_equal_static_probes(placed, width, height, reference):
    ctx, gpu = placed
    frame = lr.look_frame((0.0, 0.0, 35.0), (0.02, -0.01, -1.0), (0.0, 1.0, 0.0), 0.34, width, height)
    faces, distances = lr.probe(ctx, gpu, frame, reference=reference)
    rays = scenes.frame_rays(frame)
    hits = lr.trace_rays(ctx, gpu, rays, reference=reference, width=0)
    assert np.array_equal(distances.view(np.uint32), hits[:, 0].view(np.uint32))
    assert np.array_equal(faces != 0xFFFFFFFF, lr.hit_ids(hits) >= 0)
    static = lr.probe_static(ctx, gpu, frame, reference=reference)
    assert np.array_equal(faces, static[0]) and np.array_equal(distances.view(np.uint32), static[1].view(np.uint32))
