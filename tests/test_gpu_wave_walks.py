"""Every walk a pass can take makes the image of the plain BVH2 walk, bit for bit, on queues too
long for a warp a ray (8 rays a warp: 37,888 on 148 SMs): the 4- and 8-wide trees in warp batches
and with refilling warps, later rounds on the 8-wide tree, and BVH2 warps that vote, over queues
that mix members of different scenes, camera and light paths."""
import numpy as np
import pytest

import luce_render_b200 as lr
import render_cases
from luce_render_b200 import scenes

pytestmark = pytest.mark.gpu

SWITCHES = ("LUCE_RENDER_B200_BVH_WIDTH", "LUCE_RENDER_B200_REFILL", "LUCE_RENDER_B200_THIN")


def _members(scale):
    """A light-traced Cornell box, a scene of 20k triangles and a glossy box, films of `scale`."""
    box = lr.compile_scene(scenes.cornell_meshes(materials=True), [scenes.cornell_camera()],
                           [scenes.cornell_light()], scenes.cornell_materials())
    traced = render_cases.settings(256 * scale, 256 * scale, 1, 4, False, seed=13)
    traced.light_tracing = 0.5
    meshes, materials, lights, cam = scenes.scene_of_size(20_000, seed=11)
    objects = lr.compile_scene(meshes, [cam], lights, materials)
    meshes, cams, lights, materials = scenes.glossy_cornell(2)
    glossy = lr.compile_scene(meshes, cams, lights, materials)
    return [(box, traced), (objects, render_cases.settings(320 * scale, 200 * scale, 2, 5, True, seed=5)),
            (glossy, render_cases.settings(160 * scale, 120 * scale, 1, 6, False, seed=17))]


def _images(ctx, uploads, members, pool):
    b = lr.Batch(ctx, lr.BatchSettings.default(pool=pool, max_bounces=6, capacity=len(members)))
    try:
        slots = [b.add(gpu, scene, settings) for gpu, (scene, settings) in zip(uploads, members)]
        b.finish()
        return [b.read(m).view(np.uint32).copy() for m in slots]
    finally:
        b.destroy()


@pytest.fixture(scope="module")
def mix(ctx):
    members = _members(1)
    uploads = [lr.GpuScene.upload(ctx, scene) for scene, _ in members]
    yield members, uploads
    for gpu in uploads:
        gpu.destroy()


@pytest.fixture(scope="module")
def plain(ctx, mix):
    members, uploads = mix
    with pytest.MonkeyPatch.context() as m:
        m.setenv("LUCE_RENDER_B200_BVH_WIDTH", "2")
        m.setenv("LUCE_RENDER_B200_THIN", "-1")
        return _images(ctx, uploads, members, 1 << 18)


@pytest.mark.parametrize("width, refill, thin", [(4, 0, -1), (4, 32, -1), (4, 8, -1), (8, 0, -1), (8, 32, -1), (8, 8, -1),
                                                 (8, 1, -1), (2, 0, 1), (2, 8, 1)])
def test_wide_walks_equal_the_bvh2(ctx, mix, plain, width, refill, thin, monkeypatch):
    members, uploads = mix
    for name, value in zip(SWITCHES, (width, refill, thin)):
        monkeypatch.setenv(name, str(value))
    for got, want in zip(_images(ctx, uploads, members, 1 << 18), plain):
        assert np.array_equal(got, want)


def test_voting_warps_over_mixed_members_equal_plain_ones(ctx):
    # 726,016 paths a pass, past 2.5 rays a lane; in passes of 100,000 warps walk plain batches.
    members = _members(2)
    uploads = [lr.GpuScene.upload(ctx, scene) for scene, _ in members]
    try:
        for got, want in zip(_images(ctx, uploads, members, 1 << 20), _images(ctx, uploads, members, 100_000)):
            assert np.array_equal(got, want)
    finally:
        for gpu in uploads:
            gpu.destroy()
