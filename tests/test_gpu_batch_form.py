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


def test_a_recorded_batch_is_dropped_when_its_buffers_move():
    """A recorded render holds the addresses of the lanes' buffers: renders in between leave it
    valid, and one whose traces outgrow them drops it, so that a replay is refused."""
    torch = pytest.importorskip("torch")
    ctx = L.Context(0)
    try:
        ctx.set_stream(torch.cuda.Stream().cuda_stream)
        ctx.set_blue_noise(L.blue_noise())
        scenes = [L.HostScene(1, seed=i, width=96, height=64, ao_samples=2) for i in range(2)]
        b = L.Batch(ctx, scenes)
        b.set_fused(False)
        b.render(2)
        planes = [fr.read(L.PLANE_LIGHT).copy() for fr in b.frames]
        b.capture(2)
        for _ in range(3):
            b.render(2)
            b.replay()
        ctx.synchronize()
        for fr, p in zip(b.frames, planes):
            assert np.array_equal(fr.read(L.PLANE_LIGHT).view(np.uint32), p.view(np.uint32))
        more = scenes[0]
        more.set_sampling(24)
        b.frames[0].upload(more.block(), more.lights(), more.light_count, more.models(), more.instance_count)
        b.render(2)
        ctx.synchronize()
        with pytest.raises(L.LuzError):
            b.replay()
        b.capture(2)
        b.replay()
        ctx.synchronize()
        assert ctx.device_status() == 0
        g = L.GPUScene(ctx, more)
        g.render(2)
        ctx.synchronize()
        assert np.array_equal(b.frames[0].read(L.PLANE_AO_BITS), g.frame.read(L.PLANE_AO_BITS))
    finally:
        ctx.close()


@pytest.mark.parametrize("fused", [True, False])
def test_tuning_a_batch_leaves_the_contexts_frames_alone(fused):
    """The tuned shape is the batch's: the launch shape of single frames, and of other
    batches, stays what it was; a shape set on the context afterwards holds for all."""
    ctx = L.Context(0)
    try:
        ctx.set_blue_noise(L.blue_noise())
        scenes = [L.HostScene(1, seed=i, width=80, height=48, ao_samples=2) for i in range(3)]
        b = L.Batch(ctx, scenes)
        b.set_fused(fused)
        before = ctx.vis_tuning()
        tuned, ms = b.autotune(1)
        assert ms > 0 and ctx.vis_tuning() == before
        b.render(2)
        ctx.synchronize()
        g = L.GPUScene(ctx, scenes[1])
        g.render(2)
        ctx.synchronize()
        assert ctx.device_status() == 0
        assert np.array_equal(b.frames[1].read(L.PLANE_LIGHT).view(np.uint32),
                              g.frame.read(L.PLANE_LIGHT).view(np.uint32))
        ctx.set_vis_tuning(refill=32, steps=1, ctas_per_sm=1)
        b.autotune(1)
        assert ctx.vis_tuning() == {"smem_nodes": 0, "refill": 32, "steps": 1, "ctas_per_sm": 1}
        b.render(2)
        ctx.synchronize()
        assert ctx.device_status() == 0
    finally:
        ctx.close()


@pytest.mark.parametrize("fused", [True, False])
def test_shadow_cull_of_a_batchs_frame_holds_in_either_form(fused):
    ctx = L.Context(0)
    try:
        ctx.set_blue_noise(L.blue_noise())
        scenes = [L.HostScene(1, seed=i, width=96, height=64, ao_samples=2) for i in range(3)]
        b = L.Batch(ctx, scenes)
        b.set_fused(fused)
        bits = {}
        for cull in (True, False, True):
            for fr in b.frames:
                fr.set_shadow_cull(cull)
            b.render(2)
            ctx.synchronize()
            for i, (sc, fr) in enumerate(zip(scenes, b.frames)):
                g = L.GPUScene(ctx, sc)
                g.frame.set_shadow_cull(cull)
                g.render(2)
                ctx.synchronize()
                got = fr.read(L.PLANE_SHADOW_BITS).copy()
                assert np.array_equal(got, g.frame.read(L.PLANE_SHADOW_BITS))
                assert np.array_equal(got, bits.setdefault((i, cull), got))
            assert ctx.device_status() == 0
        assert any(not np.array_equal(bits[i, True], bits[i, False]) for i in range(3))
    finally:
        ctx.close()
