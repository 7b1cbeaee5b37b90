"""A tuned refill point is a choice among kernels that differ: the tuner tries none when the passes
walk the BVH2 alone, whose warps refill by their own rule (every candidate would launch the same
kernels, and the winner would be noise)."""
import pytest

import luce_render_b200 as lr
import render_cases
from luce_render_b200 import scenes

pytestmark = pytest.mark.gpu


def test_no_refill_is_tried_on_the_bvh2(ctx):
    meshes, materials, lights, cam = scenes.scene_of_size(100_000, 3)  # no thin rounds by default
    scene = lr.compile_scene(meshes, [cam], lights, materials)
    gpu = lr.GpuScene.upload(ctx, scene)
    info = gpu.info
    # A width's stacks that hold the scene's bound, each in blocks of three sizes.
    stacks = (sum(k >= info.bvh2_depth + 2 for k in (32, 64, 96)) + sum(k >= info.wide4_stack + 1 for k in (32, 48)) +
              sum(k >= info.wide8_stack for k in (16, 32)))
    others = 3 * stacks + 3 + 2 + 4  # pool fills, sort intervals, first thin rounds
    on_bvh2 = 0
    try:
        for _ in range(8):
            b = lr.Batch(ctx, lr.BatchSettings.default(pool=1 << 20, max_bounces=4, capacity=1))
            b.add(gpu, scene, render_cases.settings(1024, 1024, 4, 4, False))
            t = b.tune()
            b.destroy()
            on_bvh2 += t["class_width"][1] == 2
            assert t["candidates"] == others + (0 if t["class_width"][1] == 2 else 3), t
            if t["class_width"][1] == 2 and t["thin_from"] == -1:
                assert t["refill_at"] == 0, t
    finally:
        gpu.destroy()
    assert on_bvh2 > 0
