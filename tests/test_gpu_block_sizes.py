"""Waves of different traversal block sizes in one process: each keeps the shared memory its
stacks need, whichever was set up last."""
import numpy as np
import pytest

import luce_render_b200 as lr
import render_cases

pytestmark = pytest.mark.gpu


def test_a_smaller_block_elsewhere_leaves_a_larger_one_its_stacks(monkeypatch):
    scene, settings = render_cases.cases()[3]
    ctx = lr.Context(0)
    want = render_cases.alone(ctx, scene, settings)
    monkeypatch.setenv("LUCE_RENDER_B200_TRACE_BLOCK", "256")
    large = lr.Renderer.create(ctx, scene, settings)
    large.advance_one()  # captured on the first lane
    monkeypatch.setenv("LUCE_RENDER_B200_TRACE_BLOCK", "64")
    small = lr.Renderer.create(ctx, scene, settings)
    small.finish()
    large.finish()  # captured on the second lane after the smaller block's set-up
    for r in (large, small):
        assert np.array_equal(r.read().view(np.uint32), want.view(np.uint32))
        r.destroy()
    ctx.close()
