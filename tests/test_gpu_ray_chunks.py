"""Traces of more rays than one chunk holds (2^27 shadow rays, 2^26 AO rays): the bit planes are
those of a trace of every ray from the TLAS root, with as many shadow as AO chunks, more or
fewer, and an uneven last one; and where the device has no memory for whole chunks."""
import numpy as np
import pytest

import luz_gb300 as L

pytestmark = pytest.mark.gpu


def _batch(ctx, w, h, lights, light_samples, ao):
    """One scene whose every pixel is lit: the quad under its cubes, from above."""
    s = L.HostScene(1, seed=8, width=w, height=h, point_lights=lights - 1)
    s.set_sampling(ao, ao_max=2.0, light_samples=light_samples)
    c = s.camera()
    c.mode = 2
    c.eye[:], c.center[:] = (0.0, 9.0, 0.5), (0.0, 0.0, 0.0)
    s.set_camera(c)
    ctx.set_blue_noise(L.blue_noise())
    b = L.Batch(ctx, [s])
    b.set_fused(False)
    return b


def _compare(ctx, b, lit):
    fr = b.frames[0]
    b.render(1)
    ctx.synchronize()
    assert ctx.device_status() == 0 and fr.lit_count() >= lit
    got = [fr.read(p).copy() for p in (L.PLANE_SHADOW_BITS, L.PLANE_AO_BITS)]
    b.stats(1)                                       # the same rays, each from the TLAS root
    for p, x in zip((L.PLANE_SHADOW_BITS, L.PLANE_AO_BITS), got):
        assert x.any() and np.array_equal(x, fr.read(p))
    assert ctx.device_status() == 0


@pytest.mark.parametrize("w,h,lights,light_samples,ao", [
    (128, 72, 1024, 16, 4),       # 1.13 chunks of shadow rays (4 samples a group), 1 of AO rays
    (131, 139, 3, 1, 4096),       # 1 and 1.11
    (131, 139, 630, 25, 4096),    # 2.5 (groups of 4 and 1 sample) and 1.11
    (97, 403, 1500, 3, 1800),     # 1.75 (groups of 3) and 1.05
])
def test_more_rays_than_a_chunk(w, h, lights, light_samples, ao):
    ctx = L.Context(0)
    try:
        _compare(ctx, _batch(ctx, w, h, lights, light_samples, ao), w * h)
    finally:
        ctx.close()


def test_chunks_shrink_to_the_memory_there_is():
    torch = pytest.importorskip("torch")
    ctx = L.Context(0)
    try:
        b = _batch(ctx, 64, 64, 3, 1, 4)
        b.render(1)
        ctx.synchronize()
        free, _ = torch.cuda.mem_get_info()
        held = torch.empty(free - (5 << 30), dtype=torch.uint8, device="cuda")   # a whole chunk takes 7 GB and more
        try:
            big = _batch(ctx, 128, 72, 1024, 16, 4)
            _compare(ctx, big, 128 * 72)
            del held
            torch.cuda.empty_cache()
            _compare(ctx, big, 128 * 72)
        finally:
            held = None
            torch.cuda.empty_cache()
    finally:
        ctx.close()


def test_lanes_take_an_eighth_of_the_memory_at_most():
    torch = pytest.importorskip("torch")
    ctx = L.Context(0)
    try:
        before, total = torch.cuda.mem_get_info()
        s = L.HostScene(1, seed=8, width=128, height=72, point_lights=1023)
        s.set_sampling(4, light_samples=16)
        b = L.Batch(ctx, [s] * 8)                    # 7 GB a scene in whole chunks
        b.set_fused(False)
        b.render(1)
        ctx.synchronize()
        assert ctx.device_status() == 0
        assert before - torch.cuda.mem_get_info()[0] < total // 8 + (1 << 30)
    finally:
        ctx.close()
