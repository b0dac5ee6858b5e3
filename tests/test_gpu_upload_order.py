"""Scene constants uploaded again and again: each upload is what the work after it reads,
without waits between, as blocks grow and shrink and from a context other than the one that
renders; during a stream capture an upload is refused."""
import ctypes as C

import numpy as np
import pytest

import luz_gb300 as L
from luz_gb300 import _abi

pytestmark = pytest.mark.gpu

W, H = 72, 40


def _block(scene):
    s = _abi.Scene()
    s.ambient_light_color[:], s.ambient_light_intensity = [1.0, 1.0, 1.0], 0.0
    for name in ("proj", "view", "inverse_proj", "inverse_view"):
        getattr(s, name)[:] = np.eye(4, dtype=np.float32).reshape(-1).tolist()
    s.cam_pos[:] = [0.0, 3.0, 0.0]
    s.ao_min, s.ao_max, s.shadow_type = 1e-4, 2.0, L.SHADOW_RAYTRACING
    s.num_lights = scene
    return s


def _lights(count, intensity):
    lights = (_abi.Light * max(count, 1))()
    for i in range(count):
        lt = lights[i]
        lt.color[:], lt.intensity, lt.type = [1.0, 0.5, 0.25], intensity / count, L.LIGHT_POINT
        lt.position[:], lt.direction[:] = [0.0, 5.0, 2.0], [0.0, -1.0, 0.0]
        lt.num_shadow_samples, lt.shadow_map = 0, -1
    return lights


def _frame(ctx):
    f = ctx.frame(W, H)
    f.upload(_block(1), _lights(1, 1.0), 1, None, 0)
    normal = np.zeros((H, W, 4), np.float32)
    normal[..., 1] = 1.0
    f.write(L.PLANE_NORMAL, normal)
    f.write(L.PLANE_DEPTH, np.full((H, W), 0.5, np.float32))
    f.write(L.PLANE_ALBEDO, np.full((H, W), 0xFFFFFFFF, np.uint32))
    f.write(L.PLANE_MATERIAL, np.full((H, W), 0xFFFFFF80, np.uint32))
    f.write(L.PLANE_EMISSION, np.zeros((H, W), np.uint32))
    return f


def _light(f):
    return f.read(L.PLANE_LIGHT)[..., :3].copy()


def test_uploads_follow_one_another_and_outgrow_their_block():
    torch = pytest.importorskip("torch")
    ctx = L.Context(0)
    try:
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        f = _frame(ctx)
        f.light_pass()
        one = _light(f)
        assert (one > 0).all()
        frames = [_frame(ctx) for _ in range(4)]
        with torch.cuda.stream(stream):
            torch.cuda._sleep(50_000_000)            # the copies queue up behind it
        for n, intensity in ((1, 2.0), (3, 4.0), (200, 8.0), (2, 16.0), (500, 32.0), (1, 64.0)):
            models = (_abi.Model * n)()
            for k, fr in enumerate(frames):
                fr.upload(_block(n), _lights(n, intensity * 2.0 ** k), n, models, n)
                fr.light_pass()
        for k, fr in enumerate(frames):
            assert np.array_equal(_light(fr), one * np.float32(64.0 * 2.0 ** k))
        ctx.synchronize()
        assert ctx.device_status() == 0
    finally:
        ctx.close()


def test_upload_by_another_context_is_there_when_the_call_returns():
    torch = pytest.importorskip("torch")
    loader, ctx = L.Context(0), L.Context(0)
    try:
        stream = torch.cuda.Stream()
        loader.set_stream(stream.cuda_stream)
        f = _frame(loader)
        lib, h = L.lib, f.handle
        loader.synchronize()
        assert lib.luz_light_pass(ctx.handle, h, 0) == 0
        ctx.synchronize()
        one = _light(f)
        with torch.cuda.stream(stream):
            torch.cuda._sleep(400_000_000)           # the loader's stream is busy for a while
        f.upload(_block(1), _lights(1, 2.0), 1, None, 0)
        assert lib.luz_light_pass(ctx.handle, h, 0) == 0
        ctx.synchronize()
        out = np.zeros((H, W, 4), np.float32)
        assert lib.luz_frame_read(ctx.handle, h, L.PLANE_LIGHT, _abi.ptr(out), C.c_size_t(out.nbytes)) == 0
        assert np.array_equal(out[..., :3], one * np.float32(2.0))
        loader.synchronize()
    finally:
        ctx.close()
        loader.close()


def test_upload_during_a_capture_is_refused():
    torch = pytest.importorskip("torch")
    ctx = L.Context(0)
    try:
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        f = _frame(ctx)
        f.light_pass()
        ctx.synchronize()
        one = _light(f)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="relaxed")
            try:
                with pytest.raises(L.LuzError):
                    f.upload(_block(1), _lights(1, 2.0), 1, None, 0)
                f.light_pass()
            finally:
                graph.capture_end()
            graph.replay()
        ctx.synchronize()
        assert np.array_equal(_light(f), one)        # the refused upload left nothing behind
    finally:
        ctx.close()


def test_a_frame_is_created_while_the_stream_is_busy():
    torch = pytest.importorskip("torch")
    ctx = L.Context(0)
    try:
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        _frame(ctx)
        ctx.synchronize()
        busy = torch.cuda.Event()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1_000_000_000)         # half a second
            busy.record()
        f = ctx.frame(W, H)
        f.upload(_block(1), _lights(1, 1.0), 1, None, 0)
        assert not busy.query()                      # neither call waited for the stream
        ctx.synchronize()
    finally:
        ctx.close()
