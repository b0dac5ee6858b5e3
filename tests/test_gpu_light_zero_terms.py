"""Lights whose terms the light pass leaves out: a light behind every surface and a light
with every sample occluded change no bit of the light plane, in front of surfaces of every
roughness (roughness 0 takes the full evaluation); a light of infinite radiance is evaluated
in full and gives NaN where its weight is 0, as the products of light.frag do."""
import numpy as np
import pytest

import luz_gb300 as L
from luz_gb300 import _abi

pytestmark = pytest.mark.gpu

W, H = 72, 40


@pytest.mark.parametrize("samples", [1, 2, 3])
@pytest.mark.parametrize("kind", ["behind", "occluded", "infinite"])
def test_zero_terms(kind, samples):
    rng = np.random.default_rng(samples)
    ctx = L.Context(0)
    try:
        s = _abi.Scene()
        s.ambient_light_color[:], s.ambient_light_intensity = [1.0, 0.9, 0.8], 0.1
        for name in ("proj", "view", "inverse_proj", "inverse_view"):
            getattr(s, name)[:] = np.eye(4, dtype=np.float32).reshape(-1).tolist()
        s.cam_pos[:] = [0.0, 3.0, 0.0]
        s.ao_min, s.ao_max, s.shadow_type = 1e-4, 2.0, L.SHADOW_RAYTRACING
        depth = rng.uniform(0.1, 0.9, (H, W)).astype(np.float32)
        normal = np.zeros((H, W, 4), np.float32)
        normal[..., 1] = 1.0                                     # every surface faces +y
        normal[rng.random((H, W)) < 0.2] = 0.0
        words = lambda: rng.integers(0, 2**32, (H, W), dtype=np.uint32)  # noqa: E731
        material = words()
        material[: H // 2] &= np.uint32(0xFFFFFF00)              # roughness 0
        planes = {L.PLANE_ALBEDO: words(), L.PLANE_MATERIAL: material, L.PLANE_EMISSION: words()}
        bits = rng.integers(0, 2**32, (4 * samples, (W * H + 31) // 32), dtype=np.uint32)

        def render(count):
            lights = (_abi.Light * count)()
            for i, lt in enumerate(lights):
                lt.color[:], lt.intensity, lt.type = [1.0, 0.5, 0.25], 40.0, i % 3
                lt.position[:], lt.direction[:] = [i - 1.0, 5.0 + i, 2.0], [0.1 * i, -1.0, 0.2]
                lt.inner_angle, lt.outer_angle, lt.num_shadow_samples, lt.shadow_map = 0.95, 0.7, samples, -1
            if count == 4 and kind != "occluded":
                lights[3].type, lights[3].position[:] = L.LIGHT_POINT, [0.3, -50.0, 0.4]
                if kind == "infinite":
                    lights[3].intensity = float("inf")
            s.num_lights = count
            f = ctx.frame(W, H)
            f.upload(s, lights, count, None, 0)
            for p, x in planes.items():
                f.write(p, x)
            f.write(L.PLANE_NORMAL, normal)
            f.write(L.PLANE_DEPTH, depth)
            b = bits[: count * samples].copy()
            if count == 4 and kind == "occluded":
                b[3 * samples:] = 0xFFFFFFFF
            f.write(L.PLANE_SHADOW_BITS, b)
            f.light_pass()
            ctx.synchronize()
            assert ctx.device_status() == 0
            return f.read(L.PLANE_LIGHT).reshape(H, W, 4)

        base, more = render(3), render(4)
        lit = normal[..., 1] != 0
        assert (base[lit][:, :3].max(-1) > 0).all()
        if kind == "infinite":
            assert np.isnan(more[lit][:, :3]).all()
            assert np.array_equal(more[~lit].view(np.uint32), base[~lit].view(np.uint32))
        else:
            smooth = lit & ((material & 255) == 0)
            same = (more.view(np.uint32) == base.view(np.uint32)).all(-1)
            nan = np.isnan(base).any(-1)
            assert same[~nan].all() and smooth.any()
    finally:
        ctx.close()
