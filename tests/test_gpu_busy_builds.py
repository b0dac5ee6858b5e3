"""BLAS and TLAS builds while other streams keep the device busy: the sort's tiles wait only on
tiles that run, so the trees are those of a build alone and no status bit is raised."""
import threading

import numpy as np
import pytest

import luz_gb300 as L

pytestmark = pytest.mark.gpu


def _mesh(rng, n):
    v = np.zeros((3 * n, 12), np.float32)
    v[:, :3] = (rng.uniform(-9, 9, (n, 1, 3)) + rng.uniform(-0.2, 0.2, (n, 3, 3))).reshape(-1, 3)
    return v, np.arange(3 * n, dtype=np.uint32)


# one segment of 2, 3, 40, 128 and 129 tiles of 2048 keys, and several in one sort
@pytest.mark.parametrize("sizes", [[2049], [4097], [81920], [128 * 2048], [128 * 2048 + 1], [5000, 1, 70000, 30000]])
def test_builds_beside_a_rendering_batch(sizes):
    rng = np.random.default_rng(sum(sizes))
    meshes = [_mesh(rng, n) for n in sizes]
    ctx, other = L.Context(0), L.Context(0)
    try:
        want = [b.download() for b in ctx.build_blas(meshes)]
        other.set_blue_noise(L.blue_noise())
        batch = L.Batch(other, [L.HostScene(2, seed=i, width=640, height=360, meshes=2, instances=5000, subdivisions=3,
                                            ao_samples=2) for i in range(8)])
        stop, failed = threading.Event(), []

        def render():
            try:
                while not stop.is_set():
                    for _ in range(4):
                        batch.render(1)
                    other.synchronize()
            except Exception as e:                   # noqa: BLE001 (reported by the main thread)
                failed.append(e)

        t = threading.Thread(target=render)
        t.start()
        try:
            for _ in range(6):
                for b, w in zip(ctx.build_blas(meshes), want):
                    for x, y in zip(b.download(), w):
                        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
        finally:
            stop.set()
            t.join()
        assert not failed, failed
        assert ctx.device_status() == 0 and other.device_status() == 0
    finally:
        ctx.close()
        other.close()
