"""The list of lit pixels at the edges of its blocks (32x32 pixels, 8x8 G-buffer tiles, 64x64
list tiles) and of its two forms (up to 4096 blocks each block adds up the counts before its
own, above that they are scanned): counted in the G-buffer pass, and counted again from a
normal plane that was written back. Both give the planes' number of lit pixels and the same
light and hit/miss planes, the background at every other pixel."""
import numpy as np
import pytest

import luz_gb300 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(1, 1), (7, 9), (31, 33), (64, 64), (65, 129), (511, 3), (4096, 1024), (4096, 1025)])
def test_counts_and_planes(width, height):
    ctx = L.Context(0)
    try:
        s = L.HostScene(1, seed=width + height, width=width, height=height, points=1, ao_samples=1)
        g = L.GPUScene(ctx, s)
        fr = g.frame
        planes = (L.PLANE_LIGHT, L.PLANE_SHADOW_BITS, L.PLANE_AO_BITS)
        runs = []
        for again in (False, True):
            if again:
                fr.write(L.PLANE_LIGHT, np.full((height, width, 4), 7.0, np.float32))
                fr.write(L.PLANE_NORMAL, normal)
                fr.trace(g.tlas, 2)
                fr.light_pass()
            else:
                g.render(2)
            ctx.synchronize()
            assert ctx.device_status() == 0
            normal = fr.read(L.PLANE_NORMAL)
            lit = (normal[..., :3] != 0).any(-1)
            assert fr.lit_count() == int(lit.sum())
            runs.append([fr.read(p) for p in planes])
        for a, b in zip(*runs):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        light = runs[0][0].reshape(height, width, 4)
        background = light[~lit]
        assert (background == background[:1]).all() and (background[:, 3] == 1).all()
        if width * height > 1000:
            assert 0 < lit.sum() < lit.size
    finally:
        ctx.close()
