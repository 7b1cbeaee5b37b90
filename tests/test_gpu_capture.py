"""What capturing and instantiating a pass's graph costs, which a batch does within its first pass
and a renderer when it is created: no more than a graph of as many empty launches in a chain takes
to capture, instantiate and launch six times. The least host time of twelve first passes, with the
batches made before still alive. (With streams made for every capture, and forked the other way
round, it took three times as long.)"""
import time

import pytest

import luce_render_b200 as lr
import render_cases
from luce_render_b200 import scenes

pytestmark = pytest.mark.gpu

KERNELS = 1 + 3 * 7  # a plain pass of six bounces


def test_a_pass_is_captured_as_fast_as_a_chain(ctx):
    scene = lr.compile_scene(scenes.cornell_meshes(materials=True), [scenes.cornell_camera()],
                             [scenes.cornell_light()], scenes.cornell_materials())
    gpu = lr.GpuScene.upload(ctx, scene)
    chain = first_pass = 1.0
    live = []
    for _ in range(12):
        start = time.perf_counter()
        ctx.launch_overhead(KERNELS, True)
        chain = min(chain, time.perf_counter() - start)
        live.append(lr.Batch(ctx, lr.BatchSettings.default(pool=1024, max_bounces=6, capacity=1)))
        live[-1].add(gpu, scene, render_cases.settings(16, 16, 1, 6, False))
        ctx.synchronize()
        start = time.perf_counter()
        live[-1].advance()
        first_pass = min(first_pass, time.perf_counter() - start)
        live[-1].finish()
    for b in live:
        b.destroy()
    gpu.destroy()
    assert first_pass < chain, (first_pass, chain)
