"""TLAS builds at the edges of their three forms (one block; one block for the tree between
two grid-wide kernels from 769 instances on; grid-wide kernels above 4096) and of the sort
network and the breadth-first ranks inside them (warps, powers of two, equal Morton codes):
nodes, codes and order against the oracle's build bit for bit, and a small frame's primary
hits and hit/miss planes for the 4-wide nodes."""
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


@pytest.mark.parametrize("instances,equal", [(3, 0), (31, 0), (33, 33), (64, 20), (65, 0), (512, 0), (768, 5), (769, 300),
                                             (1025, 0), (2049, 2049), (4095, 100), (4097, 0), (6000, 3000)])
def test_tlas_and_its_traversal(ctx, instances, equal):
    s = L.HostScene(2, seed=instances, width=40, height=24, meshes=2, instances=instances, subdivisions=1, points=1,
                    spots=1, ao_samples=4)
    g = L.GPUScene(ctx, s)
    t = s.transforms()
    t[:equal] = t[0]   # equal boxes: equal Morton codes, split by index
    g.instances, g.n_instances = L.Tlas.make_instances(g.blas, s.instance_mesh(), t)
    g.render(1)
    ctx.synchronize()
    assert ctx.device_status() == 0
    ob, _ = oracle_scene(s)
    tl = O.OracleTlas([ob[m] for m in s.instance_mesh()], t)
    gn, gm, go = g.tlas.download()
    on, om, oo = tl.arrays()
    assert np.array_equal(gm[:instances], om)
    assert np.array_equal(go[:instances], oo)
    assert np.array_equal(gn.view(np.uint32), on.view(np.uint32))
    f = oracle_frame(s, tl, 1)
    assert np.array_equal(g.frame.read(L.PLANE_PRIMARY_HIT).reshape(-1, 2), f.primary_hit)
    assert bits_mismatch(g.frame.read(L.PLANE_SHADOW_BITS), f.shadow_bits[: f.shadow_slots]) == 0
    assert bits_mismatch(g.frame.read(L.PLANE_AO_BITS), f.ao_bits[: f.ao_samples]) == 0
