"""The passes of a render with light tracing or adaptive sampling queue as promptly as a plain
render's: what they need beyond it is ready when the renderer is created, not made in the first
pass that asks for it. Host time to queue one pass, the least of ten renderers; capturing and
instantiating a graph there took four times a plain pass's."""
import time

import pytest

import luce_render_b200 as lr
import render_cases
from luce_render_b200 import scenes

pytestmark = pytest.mark.gpu


def _queueing(ctx, scene, settings, done):
    """Seconds to queue the pass after the first `done` samples."""
    best = 1.0
    for _ in range(10):
        settings.c.samples = max(done, 1)
        r = lr.Renderer.create(ctx, scene, settings)
        if done:
            r.finish()
        r.set_samples(done + 1)
        ctx.synchronize()
        start = time.perf_counter()
        r.advance()
        best = min(best, time.perf_counter() - start)
        r.finish()
        r.destroy()
    return best


@pytest.mark.parametrize("kind, done", [("traced", 0), ("adaptive", 3)])
def test_a_pass_queues_as_a_plain_one(ctx, kind, done):
    scene = lr.compile_scene(scenes.cornell_meshes(materials=True), [scenes.cornell_camera()],
                             [scenes.cornell_light()], scenes.cornell_materials())
    plain = render_cases.settings(64, 64, 4, 4, False)
    other = render_cases.settings(64, 64, 4, 4, False)
    if kind == "traced":
        other.light_tracing = 0.5
    else:
        other.noise_threshold, other.adaptive_minimum = 0.05, 4
    assert _queueing(ctx, scene, other, done) < 2.0 * _queueing(ctx, scene, plain, done)
