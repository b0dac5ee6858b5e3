"""Start lists around their lengths: up to 15 leaves with cuts at every size, to 31 with them
above 2048 instances and without below, to 62 without above 2048, the TLAS root past that. A
cluster of small instances around a light gives every group's shaft to that light as many
leaves, a few more where it passes others; the hit/miss planes are the oracle's bit for bit."""
import numpy as np
import pytest

import luz_gb300 as L
import oracle as O
from tests.pathutil import bits_mismatch, oracle_frame, oracle_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("instances,cluster", [(n, k) for n in (300, 2300) for k in (13, 15, 29, 30, 31)] +
                         [(2300, k) for k in (32, 45, 60, 61, 62, 63, 90)])
@pytest.mark.parametrize("cull", [True, False])
def test_lists_of_a_cluster(instances, cluster, cull):
    ctx = L.Context(0)
    try:
        s = L.HostScene(2, seed=cluster, width=88, height=56, meshes=3, instances=instances, subdivisions=2,
                        point_lights=2, spot_lights=1, ao_samples=4)
        t = s.transforms()
        at = np.array(s.lights()[0].position[:], np.float32)
        rng = np.random.default_rng(cluster)
        scene = 150                                  # instances left where they are, grown to be seen
        t[:scene, :, :3] *= 4.0
        near = slice(scene, scene + cluster)
        t[near, :, :3] *= 0.05
        t[near, :, 3] = at + rng.uniform(-1, 1, (cluster, 3)).astype(np.float32)
        t[scene + cluster:, 1, 3] -= 5000.0          # the others far below
        g = L.GPUScene(ctx, s)
        g.instances, g.n_instances = L.Tlas.make_instances(g.blas, s.instance_mesh(), t)
        g.frame.set_shadow_cull(cull)
        g.render(2)
        ctx.synchronize()
        assert ctx.device_status() == 0
        ob, _ = oracle_scene(s)
        f = oracle_frame(s, O.OracleTlas([ob[m] for m in s.instance_mesh()], t), 2)
        if not cull:
            f.shadow_bits[:] = 0
            f.ao_bits[:] = 0
            f.visibility(2, L.blue_noise(), cull=False)
        assert int((f.primary_hit[:, 0] != 0xFFFFFFFF).sum()) > 32
        assert bits_mismatch(g.frame.read(L.PLANE_SHADOW_BITS), f.shadow_bits[: f.shadow_slots]) == 0
        assert bits_mismatch(g.frame.read(L.PLANE_AO_BITS), f.ao_bits[: f.ao_samples]) == 0
    finally:
        ctx.close()
