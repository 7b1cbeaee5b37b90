"""The warp-a-ray walk of short queues (32 lanes share one ray on the 8-wide tree): closest
hits equal the FP32 brute force bit for bit, ties and misses included, at queue lengths around
a warp, a block and the length past which the plain walk takes over; renders through it equal
renders whose traversal counts its work, which never take it."""
import numpy as np
import pytest

import luce_render_b200 as lr
import render_cases
from luce_render_b200 import scenes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _wide_leaves():
    """Leaves of up to 16 triangles: a stack of coincident quads the SAH does not split."""
    quads = [scenes._quad((-1, -1, 0), (1, -1, 0), (1, 1, 0), (-1, 1, 0)) for _ in range(7)]
    return [lr.MeshData(p, t) for p, t in quads]


@pytest.mark.parametrize("meshes, extent", [(scenes.cornell_meshes, 0.6), (_wide_leaves, 1.5),
                                            (lambda: scenes.scene_of_size(6000, 3)[0], 12.0)])
@pytest.mark.parametrize("count", [1, 3, 4, 5, 127, 4097])
def test_short_queries_equal_brute_force(meshes, extent, count):
    scene = lr.compile_scene(meshes())
    a = scene.arrays()
    rays = scenes.random_rays(count, count, -extent, extent)
    rays[::5, 7] = 0.3 * extent
    ctx = lr.Context(0)
    gpu = lr.GpuScene.upload(ctx, scene)
    hits = lr.trace_rays(ctx, gpu, rays)
    prim, t, u, v = orc.brute_watertight(a["positions"], a["indices"], a["order"], rays)
    assert np.array_equal(lr.hit_ids(hits), prim)
    found = prim >= 0
    assert np.array_equal(hits[found, 0].view(np.uint32), t[found].view(np.uint32))
    assert np.array_equal(hits[found, 2].view(np.uint32), u[found].view(np.uint32))
    assert np.array_equal(hits[found, 3].view(np.uint32), v[found].view(np.uint32))
    assert np.array_equal(hits[~found, 0], rays[~found, 7])
    gpu.destroy()
    ctx.close()


def test_walks_agree_where_one_takes_over_from_the_other():
    meshes, materials, lights, cam = scenes.scene_of_size(30_000, 9)
    scene = lr.compile_scene(meshes, [cam], lights, materials)
    rays = scenes.random_rays(60_000, 2, -15.0, 15.0)
    ctx = lr.Context(0)
    gpu = lr.GpuScene.upload(ctx, scene)
    whole = lr.trace_rays(ctx, gpu, rays)
    parts = np.concatenate([lr.trace_rays(ctx, gpu, rays[i:i + 1000]) for i in range(0, 60_000, 1000)])
    gpu.destroy()
    ctx.close()
    assert np.array_equal(whole.view(np.uint32), parts.view(np.uint32))


@pytest.mark.parametrize("index", range(11))
def test_renders_equal_counted_renders(index):
    scene, settings = render_cases.cases()[index]
    ctx = lr.Context(0)
    images = []
    for profile in (0, 2):
        settings.profile = profile
        r = lr.Renderer.create(ctx, scene, settings)
        r.finish()
        images.append(r.read())
        r.destroy()
    ctx.close()
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))
