"""Which form a group's start list takes, seen by the counting trace: rays that start at a list
visit no TLAS node. Every group's shaft ends at a light inside k boxes, so its list has k
leaves: up to 31 of them, above 2048 instances up to 62, and the TLAS root past that. And
frames of the smallest sizes with every pixel lit."""
import numpy as np
import pytest

import luz_gb300 as L
import oracle as O
from tests.pathutil import bits_mismatch, oracle_frame, oracle_scene

pytestmark = pytest.mark.gpu


def _above(s):
    c = s.camera()
    c.mode = 2
    c.eye[:], c.center[:] = (0.0, 9.0, 0.5), (0.0, 0.0, 0.0)
    s.set_camera(c)


@pytest.mark.parametrize("instances", [300, 2300])
@pytest.mark.parametrize("k", [1, 15, 16, 31, 32, 33, 61, 62, 63])
def test_lists_and_roots(instances, k):
    ctx = L.Context(0)
    try:
        s = L.HostScene(1, seed=k, width=64, height=40, instances=instances)
        s.set_sampling(0, light_samples=2)
        _above(s)
        lights = s.lights()
        lights[0].type = L.LIGHT_POINT
        lights[0].position[:], lights[0].radius = (0.5, 6.0, -0.25), 0.1
        t = s.transforms()
        cubes = np.nonzero(s.instance_mesh() == s.instance_mesh()[-1])[0]
        assert len(cubes) == instances
        rng = np.random.default_rng(k)
        t[cubes, 1, 3] = -5000.0                     # far below but for k around the light
        near = cubes[:k]
        t[near, :, :3] = np.eye(3, dtype=np.float32) * rng.uniform(0.5, 0.9, (k, 1, 1)).astype(np.float32)
        t[near, :, 3] = np.array(lights[0].position[:], np.float32) + rng.uniform(-0.1, 0.1, (k, 3)).astype(np.float32)
        g = L.GPUScene(ctx, s)
        block = s.block()
        block.num_lights = 1
        g.frame.upload(block, lights, 1, g.models, s.instance_count)
        inst, n = L.Tlas.make_instances(g.blas, s.instance_mesh(), t)
        g.tlas.build(inst, n)
        g.frame.gbuffer(g.tlas)
        st = g.frame.trace_stats(g.tlas, 1)
        ctx.synchronize()
        assert ctx.device_status() == 0
        assert g.frame.lit_count() > 2000 and st["rays"] > 2000 and st["instances"] > 0
        assert (st["tlas_nodes"] == 0) == (k <= (62 if instances > 2048 else 31))
        counted = g.frame.read(L.PLANE_SHADOW_BITS).copy()
        assert counted.any()
        g.frame.trace(g.tlas, 1)
        assert np.array_equal(g.frame.read(L.PLANE_SHADOW_BITS), counted)
        ob, _ = oracle_scene(s)
        f = O.OracleFrame(O.OracleTlas([ob[m] for m in s.instance_mesh()], t), block, lights, 1, s.models(),
                          s.instance_count, s.width, s.height)
        f.gbuffer()
        f.visibility(1, L.blue_noise())
        assert bits_mismatch(counted, f.shadow_bits[: f.shadow_slots]) == 0
    finally:
        ctx.close()


@pytest.mark.parametrize("w,h", [(1, 1), (1, 33), (19, 17)])
@pytest.mark.parametrize("cull", [True, False])
def test_small_frames_with_every_pixel_lit(w, h, cull):
    ctx = L.Context(0)
    try:
        s = L.HostScene(1, seed=w, width=w, height=h)
        s.set_sampling(5, ao_max=2.0, light_samples=5)
        _above(s)
        g = L.GPUScene(ctx, s)
        g.frame.set_shadow_cull(cull)
        g.render(1)
        ctx.synchronize()
        assert ctx.device_status() == 0 and g.frame.lit_count() == w * h
        _, tl = oracle_scene(s)
        f = oracle_frame(s, tl, 1)
        if not cull:
            f.shadow_bits[:] = 0
            f.ao_bits[:] = 0
            f.visibility(1, L.blue_noise(), cull=False)
        assert bits_mismatch(g.frame.read(L.PLANE_SHADOW_BITS), f.shadow_bits[: f.shadow_slots]) == 0
        assert bits_mismatch(g.frame.read(L.PLANE_AO_BITS), f.ao_bits[: f.ao_samples]) == 0
    finally:
        ctx.close()
