"""Ray lists of more than 2^31 rays in device memory (the limit is 2^32 - 1): the last rays are
answered from their own records, in every width. All but a few rays are zero, of no reach and
outside the scene, so they end at its root box."""
import numpy as np
import pytest

import luce_render_b200 as lr
from luce_render_b200 import scenes

pytestmark = pytest.mark.gpu

COUNT = (1 << 31) + 97


def test_rays_past_two_to_the_31(ctx):
    need = COUNT * 48
    if ctx.memory()["free"] < need + (4 << 30):
        pytest.skip("the device has no room for the list")
    p, t, f = scenes.grid(2.0, 8)
    scene = lr.compile_scene([lr.MeshData(p + np.float32([0.0, 10.0, 0.0]), t, faces=f, face_count=int(f.max()) + 1)])
    last = np.zeros((97, 8), np.float32)
    last[:, 0] = np.linspace(-0.9, 0.9, 97)
    last[:, 1:3] = (11.0, 0.1)
    last[:, 5], last[:, 7] = -1.0, 100.0
    gpu = lr.GpuScene.upload(ctx, scene)
    want = lr.trace_rays(ctx, gpu, last)
    assert (lr.hit_ids(want) >= 0).all()
    rays = hits = None
    try:
        rays, hits = ctx.alloc(COUNT * 32), ctx.alloc(COUNT * 16)
        ctx.memset(rays, 0, COUNT * 32)
        ctx.upload(rays + (COUNT - 97) * 32, last)
        for width in (0, 4, 8):
            ctx.memset(hits, 0xFF, COUNT * 16)
            lr._check(lr.lib.lr_trace_rays_device(ctx.handle, gpu.handle, rays, COUNT, hits, lr.TRACE_BVH[width]))
            ctx.synchronize()
            got = ctx.download(hits + (COUNT - 97) * 16, np.empty((97, 4), np.float32))
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), width
    finally:
        for buffer in (rays, hits):
            if buffer is not None:
                ctx.free(buffer)
        gpu.destroy()
