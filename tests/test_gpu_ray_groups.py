"""Rays resolved in groups before the traversal: shadow groups by their shafts (and the
cuts of the BLASes that the rest start at), AO rays by their patch's horizon. Every case
compares the hit/miss planes with the oracle's per-ray traces bit for bit, at the edges of
the groups (patches of 32 lit pixels, blocks of 8 patches, groups of 4 samples, lists of 15
and 31 leaves, horizons from 4 AO samples on) and over instance transforms of every kind."""
import numpy as np
import pytest

import luz_gb300 as L
import oracle as O
from tests.pathutil import bits_mismatch, oracle_frame, oracle_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = L.Context(0)
    yield c
    c.close()


def _check(ctx, s, cull, transforms=None, frame=3):
    g = L.GPUScene(ctx, s)
    if transforms is not None:
        g.instances, g.n_instances = L.Tlas.make_instances(g.blas, s.instance_mesh(), transforms)
    g.frame.set_shadow_cull(cull)
    g.render(frame)
    ctx.synchronize()
    assert ctx.device_status() == 0
    ob, tl = oracle_scene(s)
    if transforms is not None:
        tl = O.OracleTlas([ob[m] for m in s.instance_mesh()], transforms)
    f = oracle_frame(s, tl, frame)
    if not cull:
        f.shadow_bits[:] = 0
        f.ao_bits[:] = 0
        f.visibility(frame, L.blue_noise(), cull=False)
    assert np.array_equal(g.frame.read(L.PLANE_PRIMARY_HIT).reshape(-1, 2), f.primary_hit)
    lit = int((f.primary_hit[:, 0] != 0xFFFFFFFF).sum())
    if f.shadow_slots:
        assert bits_mismatch(g.frame.read(L.PLANE_SHADOW_BITS), f.shadow_bits[: f.shadow_slots]) == 0
    if f.ao_samples:
        assert bits_mismatch(g.frame.read(L.PLANE_AO_BITS), f.ao_bits[: f.ao_samples]) == 0
    return lit


@pytest.mark.parametrize("w,h,instances,light_samples,ao,sampler,cull,ao_max", [
    (1, 1, 16, 1, 4, 0, True, 1.0),          # one pixel
    (31, 1, 30, 4, 5, 1, True, 1.0),         # a row shorter than a patch; a full sample group
    (33, 17, 64, 2, 3, 0, False, 1.0),       # below the horizon's sample limit
    (64, 40, 64, 5, 4, 1, True, 2.0),        # two sample groups of one light
    (97, 61, 64, 7, 9, 0, False, 30.0),      # AO lists and horizon instances run over
    (160, 90, 400, 1, 16, 1, True, 0.3),     # dense field, short rays
    (129, 65, 2500, 1, 6, 0, True, 6.0),     # lists of up to 31 leaves, running over
])
def test_cube_fields(ctx, w, h, instances, light_samples, ao, sampler, cull, ao_max):
    s = L.HostScene(3, seed=11, width=w, height=h, instances=instances, sampler=sampler)
    s.set_sampling(ao, ao_max=ao_max, light_samples=light_samples, sampler=sampler)
    _check(ctx, s, cull)


@pytest.mark.parametrize("subdivisions,instances,cull,ao", [(1, 40, True, 16), (3, 900, False, 4), (5, 300, True, 33)])
def test_displaced_spheres(ctx, subdivisions, instances, cull, ao):
    s = L.HostScene(2, seed=5, width=211, height=119, meshes=5, instances=instances, subdivisions=subdivisions,
                    point_lights=6, spot_lights=5)
    s.set_sampling(ao)
    assert _check(ctx, s, cull) > 32


@pytest.mark.parametrize("kind", ["stretched", "mirrored", "sheared", "far"])
def test_affine_instances(ctx, kind):
    """Shafts and horizons work in object space: transforms that stretch, mirror or shear the
    mesh, and a scene far from the origin (large coordinates, coarse rounding)."""
    rng = np.random.default_rng(3)
    s = L.HostScene(2, seed=9, width=200, height=112, meshes=4, instances=500, subdivisions=4, point_lights=5,
                    spot_lights=3)
    s.set_sampling(8)
    tr = s.transforms().reshape(-1, 3, 4).astype(np.float64)
    for m in tr:
        if kind == "stretched":
            m[:, :3] = m[:, :3] @ np.diag(rng.uniform(0.1, 3.0, 3))
        elif kind == "mirrored":
            m[:, :3] = m[:, :3] @ np.diag([-1.0, 1.0, rng.choice([-1.0, 1.0])])
        elif kind == "sheared":
            m[:, :3] = m[:, :3] @ (np.eye(3) + np.triu(rng.uniform(-2, 2, (3, 3)), 1))
    if kind == "far":
        tr[:, :, 3] += [4000.0, -3000.0, 2500.0]
        c = s.camera()
        for k, v in enumerate((4000.0, -3000.0, 2500.0)):
            c.eye[k] += v
            c.center[k] += v
        s.set_camera(c)
    assert _check(ctx, s, True, tr.astype(np.float32)) > 256
