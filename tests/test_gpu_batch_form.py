"""The form of a batch is the caller's to choose: on and off select it whatever the scenes'
sizes, luz_batch_fused says which one renders, and until a choice is made the faster one does."""
import numpy as np
import pytest

import luz_gb300 as L

pytestmark = pytest.mark.gpu


def _launches(ctx, b):
    before = ctx.launch_count()
    b.render(2)
    ctx.synchronize()
    assert ctx.device_status() == 0
    return ctx.launch_count() - before


@pytest.mark.parametrize("sizes,default", [([(64, 48)] * 4, True), ([(64, 48)] * 2, False), ([(1, 1)], False),
                                           ([(500, 400)] * 3, False)])
def test_the_chosen_form_renders(sizes, default):
    ctx = L.Context(0)
    try:
        ctx.set_blue_noise(L.blue_noise())
        b = L.Batch(ctx, [L.HostScene(1, seed=i, width=w, height=h, ao_samples=2) for i, (w, h) in enumerate(sizes)])
        assert b.fused == default
        assert (_launches(ctx, b) == 1) == default
        planes = [fr.read(L.PLANE_LIGHT).copy() for fr in b.frames]
        for fused in (True, False, True):
            b.set_fused(fused)
            assert b.fused == fused
            assert (_launches(ctx, b) == 1) == fused
            for fr, p in zip(b.frames, planes):
                assert np.array_equal(fr.read(L.PLANE_LIGHT).view(np.uint32), p.view(np.uint32))
    finally:
        ctx.close()
