"""The step cap counts the steps that a ray takes itself: a ray that fits it is traced to its
end however long it waits for others of its warp, and in launches that check it rarely; a cap
that the longest ray does not fit is reported."""
import numpy as np
import pytest

import luz_gb300 as L

pytestmark = pytest.mark.gpu

LUZ_DEV_TRAVERSAL_CAP = 1 << 2


def test_cap_counts_a_rays_own_steps():
    ctx = L.Context(0)
    try:
        s = L.HostScene(3, seed=6, width=24, height=12, instances=900, ao_samples=1)
        s.set_sampling(1, ao_max=1e4, light_samples=0)   # rays of any length, from the TLAS root
        g = L.GPUScene(ctx, s)
        g.render(1)
        ctx.synchronize()
        want = g.frame.read(L.PLANE_AO_BITS).copy()
        normal = g.frame.read(L.PLANE_NORMAL).copy()
        total = g.frame.trace_stats(g.tlas, 1)
        # the steps of each pixel's one ray, traced alone
        steps = []
        for y, x in np.argwhere(np.linalg.norm(normal[..., :3], axis=-1) > 0):
            only = np.zeros_like(normal)
            only[y, x] = normal[y, x]
            g.frame.write(L.PLANE_NORMAL, only)
            st = g.frame.trace_stats(g.tlas, 1)
            assert st["rays"] == 1
            steps.append(st["tlas_nodes"] + st["blas_nodes"] + st["tris"] + st["instances"])
        g.frame.write(L.PLANE_NORMAL, normal)
        assert sum(steps) == sum(total[k] for k in ("tlas_nodes", "blas_nodes", "tris", "instances"))
        fits = (max(steps) + 7) & ~7
        assert len(steps) > 100 and fits >= 32
        for tuning in ({}, {"refill": 8, "steps": 2, "ctas_per_sm": 2}, {"refill": 32, "steps": 8, "ctas_per_sm": 4},
                       {"refill": 1, "steps": 1, "ctas_per_sm": 1}):
            ctx.set_vis_tuning(**tuning)
            ctx.set_debug_step_cap(fits)
            g.frame.trace(g.tlas, 1)
            ctx.synchronize()
            assert ctx.device_status() == 0
            assert np.array_equal(g.frame.read(L.PLANE_AO_BITS), want)
            ctx.set_debug_step_cap(fits - 24)            # (rounds of up to 8 steps may pass it by those)
            g.frame.trace(g.tlas, 1)
            assert ctx.device_status() == LUZ_DEV_TRAVERSAL_CAP
    finally:
        ctx.close()
