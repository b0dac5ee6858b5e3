"""Instances whose transform is singular or not finite: no ray hits them, no access leaves its
buffer (a ray with a NaN overlaps the boxes of empty child slots too), and the frame is that of
the same scene with those instances masked out, in single frames and in both batch forms."""
import numpy as np
import pytest

import luz_gb300 as L

pytestmark = pytest.mark.gpu

INF, NAN = np.inf, np.nan
PLANES = (L.PLANE_PRIMARY_HIT, L.PLANE_NORMAL, L.PLANE_SHADOW_BITS, L.PLANE_AO_BITS)


def _spoil(t, kind):
    if kind == "flat":
        t[:, 1, :3] = 0.0
    elif kind == "zero":
        t[:, :, :3] = 0.0
    elif kind == "nan":
        t[:, 0, 1] = NAN
    elif kind == "nan translation":
        t[:, 2, 3] = NAN
    elif kind == "inf":
        t[:, 1, 1] = INF
    elif kind == "inf translation":
        t[:, 0, 3] = -INF
    elif kind == "all inf":
        t[:, :, :] = INF


class _Scene(L.HostScene):
    def transforms(self):
        t = super().transforms()
        if self.kind:
            sub = t[self.bad]
            _spoil(sub, self.kind)
            t[self.bad] = sub
        return t


@pytest.mark.parametrize("kind", ["flat", "zero", "nan", "nan translation", "inf", "inf translation", "all inf"])
@pytest.mark.parametrize("cfg,kw", [(1, {"instances": 40}), (2, {"meshes": 3, "instances": 2500, "subdivisions": 2}),
                                    (1, {"instances": 5000})])
def test_frames_without_the_bad_instances(cfg, kw, kind):
    ctx = L.Context(0)
    try:
        s = _Scene(cfg, seed=12, width=72, height=44, **kw)
        s.kind = None
        s.set_sampling(5, ao_max=3.0, light_samples=2)
        rng = np.random.default_rng(3)
        bad = rng.random(s.instance_count) < 0.2
        bad[0] = False                               # (config 1: the quad)
        s.bad = np.nonzero(bad)[0]
        s.kind = kind
        g = L.GPUScene(ctx, s)
        got = []
        for mask in (None, np.where(bad, 0, 0xFF)):
            g.instances, g.n_instances = L.Tlas.make_instances(g.blas, s.instance_mesh(), s.transforms(), mask=mask)
            g.render(1)
            ctx.synchronize()
            assert ctx.device_status() == 0
            got.append([g.frame.read(p).copy() for p in PLANES])
        assert g.frame.lit_count() > 100
        for a, b in zip(*got):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        if s.instance_count > 4096:
            return
        b = L.Batch(ctx, [s])
        for fused in (True, False):
            b.set_fused(fused)
            b.render(1)
            ctx.synchronize()
            for p, x in zip(PLANES, got[0]):
                assert np.array_equal(b.frames[0].read(p).view(np.uint32), x.view(np.uint32))
        b.stats(1)
        for p, x in zip(PLANES, got[0]):
            assert np.array_equal(b.frames[0].read(p).view(np.uint32), x.view(np.uint32))
        assert ctx.device_status() == 0
    finally:
        ctx.close()


def test_many_bad_instances_of_a_large_mesh_cost_a_ray_nothing():
    """A row of zeros beside rows of NaN leaves boxes to overlap along a plane of the mesh: were
    they walked, a ray over many such instances would run into its step cap."""
    ctx = L.Context(0)
    try:
        s = _Scene(2, seed=3, width=48, height=32, meshes=2, instances=4000, subdivisions=6)
        s.kind, s.bad = "inf", np.arange(1, 4000, 2)
        s.set_sampling(2, ao_max=3.0)
        g = L.GPUScene(ctx, s)
        g.render(1)
        ctx.synchronize()
        assert ctx.device_status() == 0
        st = g.frame.trace_stats(g.tlas, 1)
        assert st["rays"] > 0 and st["blas_nodes"] < 500 * st["rays"]
    finally:
        ctx.close()
