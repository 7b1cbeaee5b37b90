"""Captured passes fork: a round's shadow rays beside the next round's closest hits, light
paths' shading beside the camera paths'. Profiled passes run the same kernels one after
another, so their images are the reference, bit for bit."""
import numpy as np
import pytest

import luce_render_b200 as lr
import render_cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("index", range(11))
def test_forked_pass_equals_serial_pass(index):
    scene, settings = render_cases.cases()[index]
    ctx = lr.Context(0)
    images = []
    for profile in (0, 1):
        settings.profile = profile
        r = lr.Renderer.create(ctx, scene, settings)
        r.finish()
        images.append(r.read())
        r.destroy()
    ctx.close()
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))
