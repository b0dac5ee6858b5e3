"""Batches whose scenes run in lanes (streams forked from the context's): more scenes than
lanes, two scenes, scenes of 200,000 pixels on average, and the frame kernel just below
that; each scene's planes are those of its own render bit for bit, rendered, recorded and
replayed, and after the other form ran in between."""
import numpy as np
import pytest

import luz_gb300 as L

pytestmark = pytest.mark.gpu

PLANES = (L.PLANE_LIGHT, L.PLANE_SHADOW_BITS, L.PLANE_AO_BITS, L.PLANE_PRIMARY_HIT)


def _scene(i, w, h):
    if i % 3 == 0:
        return L.HostScene(1, seed=i, width=w, height=h, ao_samples=2)
    if i % 3 == 1:
        return L.HostScene(6, seed=i, width=w, height=h, triangles=2000 * (i + 1), ao_samples=4)
    return L.HostScene(2, seed=i, width=w, height=h, meshes=2, instances=30 * i, subdivisions=2, ao_samples=1)


@pytest.mark.parametrize("sizes,fused", [([(40 + 9 * i, 31 + i) for i in range(11)], False), ([(64, 48), (200, 33)], True),
                                         ([(500, 400)] * 3, True), ([(500, 399)] * 3, True), ([(1, 1)] * 9, False)])
def test_lanes_match_single_renders(sizes, fused):
    torch = pytest.importorskip("torch")
    ctx = L.Context(0)
    try:
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        scenes = [_scene(i, w, h) for i, (w, h) in enumerate(sizes)]
        ref = []
        for sc in scenes:
            g = L.GPUScene(ctx, sc)
            g.render(3)
            ctx.synchronize()
            ref.append([g.frame.read(p) for p in PLANES])
        ctx.set_blue_noise(L.blue_noise())
        b = L.Batch(ctx, scenes)
        b.set_fused(fused)

        def check():
            ctx.synchronize()
            assert ctx.device_status() == 0
            for fr, r in zip(b.frames, ref):
                for p, x in zip(PLANES, r):
                    assert np.array_equal(fr.read(p).view(np.uint32), x.view(np.uint32))
                fr.write(L.PLANE_LIGHT, np.zeros((fr.height, fr.width, 4), np.float32))

        b.render(3)
        check()
        b.render(3)
        b.render(3)
        check()
        b.capture(3)
        for _ in range(2):
            b.replay()
        check()
        counts = b.stats(3)
        check()
        b.set_fused(not fused)
        b.render(3)
        check()
        assert b.stats(3) == counts
    finally:
        ctx.close()
