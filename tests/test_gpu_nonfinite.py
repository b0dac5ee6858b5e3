"""Meshes with a vertex that is infinite or not a number: the group bounds (shafts, horizons)
leave every hit/miss bit as a trace of each ray from the TLAS root gives it, also for the
finite triangles that share the boxes above such a vertex."""
import numpy as np
import pytest

import luz_gb300 as L
from tests.pathutil import bits_mismatch, oracle_frame, oracle_scene

pytestmark = pytest.mark.gpu

INF, NAN = np.float32(np.inf), np.float32(np.nan)
BAD = {"none": [],
       "inf_x": [[(0, 5, 0), (0, 5, 1), (INF, 5, 0)]],
       "inf_y": [[(0, 0.2, 0), (1, INF, 0), (0, 0.2, 1)]],
       "inf_all": [[(-INF, 5, 0), (-INF, 5, 1), (-INF, 6, 0)]],
       "nan_last": [[(2, 0.3, 0), (2, 0.3, 1), (NAN, 0.3, 0)], [(-2, 0.4, 2), (-2, 0.4, 1), (0, NAN, NAN)]],
       "nan_first": [[(NAN, 0.3, 2), (2, 0.3, 1), (1, 0.3, 0)], [(0, NAN, 2), (NAN, 0.4, 1), (-1, 1, NAN)]]}


def _quads(y, xs, z0, z1, n, up):
    out = []
    for x0, x1 in xs:
        zs = np.linspace(z0, z1, n + 1)
        for a, b in zip(zs[:-1], zs[1:]):
            p = [(x0, y, a), (x1, y, a), (x1, y, b), (x0, y, b)]
            out += [[p[0], p[2], p[1]], [p[0], p[3], p[2]]] if up else [[p[0], p[1], p[2]], [p[0], p[2], p[3]]]
    return out


def _room(bad):
    """A floor that faces +y under a canopy of strips, one mesh."""
    edges = np.linspace(-6, 6, 13)
    tris = _quads(0.0, list(zip(edges[:-1], edges[1:])), -6, 6, 12, True)
    n_floor = len(tris)
    tris += _quads(0.7, [(x, x + 0.5) for x in np.arange(-4, 4, 1.0)], -4, 4, 8, False) + BAD[bad]
    v = np.zeros((len(tris) * 3, 12), np.float32)
    v[:, :3] = np.asarray(tris, np.float32).reshape(-1, 3)
    v[:, 4] = -1.0                                   # normals: the floor's +y, the others -y
    v[: 3 * n_floor, 4] = 1.0
    return v, np.arange(v.shape[0], dtype=np.uint32)


class _Scene(L.HostScene):
    def meshes(self):
        n = len(super().meshes())
        return [_room(self.bad)] + [_room("none")] * (n - 1)

    def transforms(self):
        t = np.zeros((self.instance_count, 3, 4), np.float32)
        k = np.arange(len(t))
        a = np.float32(0.4 if self.turned else 0.0)
        t[:, 0, 0] = t[:, 2, 2] = np.cos(a)
        t[:, 0, 2], t[:, 2, 0] = np.sin(a), -np.sin(a)
        t[:, 1, 1] = 1.0
        t[:, 0, 3], t[:, 2, 3] = 13.0 * (k % 7 - (3 if len(t) > 7 else 0)), -13.0 * (k // 7)
        return t


@pytest.mark.parametrize("instances", [1, 40])
@pytest.mark.parametrize("turned", [False, True])
@pytest.mark.parametrize("bad", list(BAD))
def test_group_bounds_with_nonfinite_vertices(bad, turned, instances):
    ctx = L.Context(0)
    try:
        s = _Scene(1, seed=4, width=120, height=72, instances=instances)
        s.bad, s.turned = bad, turned
        s.set_sampling(8, ao_max=2.0, light_samples=2)
        c = s.camera()
        c.mode = 2
        c.eye[:], c.center[:] = (1.0, 2.5, 9.0), (0.0, 0.0, 0.0)
        s.set_camera(c)
        ctx.set_blue_noise(L.blue_noise())
        b = L.Batch(ctx, [s])
        b.set_fused(False)
        fr = b.frames[0]
        b.render(3)
        ctx.synchronize()
        assert ctx.device_status() == 0
        got = [fr.read(p).copy() for p in (L.PLANE_SHADOW_BITS, L.PLANE_AO_BITS)]
        b.stats(3)                                   # the same rays, each from the TLAS root
        want = [fr.read(p) for p in (L.PLANE_SHADOW_BITS, L.PLANE_AO_BITS)]
        assert fr.lit_count() > 1000 and want[0].any()
        assert [bits_mismatch(x, y) for x, y in zip(got, want)] == [0, 0]
        if bad in ("none", "inf_x") and not turned:
            _, tl = oracle_scene(s)
            f = oracle_frame(s, tl, 3)
            assert bits_mismatch(got[0], f.shadow_bits[: f.shadow_slots]) == 0
            assert bits_mismatch(got[1], f.ao_bits[: f.ao_samples]) == 0
    finally:
        ctx.close()
