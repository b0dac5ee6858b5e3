"""Timed workloads of the library: what a program does with it, through its public entry points.

A case is a dict of plain values. ``kind`` names the path it takes:

* ``frame``    one frame: uploads, TLAS rebuild, G-buffer, shadow / AO trace, light pass,
               optionally through the denoiser or followed by the post passes
* ``light``    the light pass alone over given G-buffer and visibility planes
* ``train``    the denoiser's forward and backward pass over a batch of images
* ``infer``    the denoiser over every pixel of a batch of images
* ``blas``     one BLAS build into the caller's device buffers
* ``batch``    many scenes of uneven size as one unit
"""
import ctypes as C
import math
from pathlib import Path

import numpy as np
import torch

import luz_gb300 as L
from luz_gb300 import _abi, denoiser as D

WEIGHTS = Path(__file__).resolve().parent.parent / "luz_gb300" / "weights" / "denoiser_config3.bin"

FRAME = {"kind": "frame", "denoise": False, "post": False, "cull": True, "sampler": 0, "light_samples": 1}


def listed():
    return [
        # A thumbnail / material preview: the smallest frame a user asks for, where launches,
        # copies and single-block kernels are the whole cost.
        dict(FRAME, name="frame_tiny", scene="cubes", width=96, height=64, instances=16, ao=4, points=4),
        # The default test scene at its default size: an ordinary interactive frame.
        dict(FRAME, name="frame_cubes_512", scene="cubes", width=512, height=512, instances=64, ao=4, points=4),
        # A crowd of small meshes above the single-block TLAS build's limit, odd sizes, several
        # shadow samples per light, the stratified sampler, every shadow ray traced.
        dict(FRAME, name="frame_crowd_odd", scene="spheres", width=1021, height=573, instances=8000, meshes=16,
             subdivisions=3, ao=8, points=11, spots=3, light_samples=2, sampler=1, cull=False),
        # The headline frame: 1024 instances of 64 meshes of 81,920 triangles, 41 lights, 16 AO rays.
        dict(FRAME, name="frame_1080p", scene="spheres", width=1920, height=1080, instances=1024, meshes=64,
             subdivisions=6, ao=16, points=32, spots=8),
        # The same frame as the renderer shows it: 1 AO ray, denoised, then composed.
        dict(FRAME, name="frame_1080p_denoised", scene="spheres", width=1920, height=1080, instances=1024, meshes=64,
             subdivisions=6, ao=1, points=32, spots=8, sampler=1, denoise=True),
        # The largest frame: 4K, 4096 instances, 145 lights, 64 AO rays.
        dict(FRAME, name="frame_4k", scene="spheres", width=3840, height=2160, instances=4096, meshes=64,
             subdivisions=6, ao=64, points=128, spots=16),
        # A viewer's frame: cubes at 720p followed by TAA, tone mapping and the exposure histogram.
        dict(FRAME, name="frame_viewer_720p", scene="cubes", width=1280, height=720, instances=200, ao=8, points=6,
             post=True),
        # Relighting: the light pass again over planes that are in place (a light editor's change).
        {"kind": "light", "name": "light_pass_900p", "width": 1601, "height": 899, "lights": 24, "ao": 8,
         "light_samples": 2},
        # One step of denoiser training: a batch of 16 images of 256x256, forward and backward.
        {"kind": "train", "name": "train_16x256", "width": 256, "height": 256, "images": 16},
        # The denoiser over whole images of a batch (offline use).
        {"kind": "infer", "name": "infer_2x720p", "width": 1280, "height": 720, "images": 2},
        # A mesh that changed: its BVH rebuilt in place, near the entry point's largest size.
        {"kind": "blas", "name": "blas_81920", "subdivisions": 6, "keep": 81920},
        # A set of uneven scenes rendered as one unit (dataset rendering).
        {"kind": "batch", "name": "batch_12", "scenes": 12, "triangles": 300000, "ao": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cubes", "spheres", "spheres", "denoised", "viewer", "light", "train", "infer", "blas",
                       "batch"])
    if kind in ("cubes", "viewer"):
        return dict(FRAME, scene="cubes", width=_log(rng, 64, 1600), height=_log(rng, 48, 900),
                    instances=_log(rng, 4, 1000), ao=_log(rng, 1, 32), points=_log(rng, 1, 16),
                    light_samples=rng.choice([1, 1, 2, 4]), sampler=rng.choice([0, 1]),
                    cull=rng.random() < 0.75, post=kind == "viewer")
    if kind in ("spheres", "denoised"):
        denoise = kind == "denoised"
        return dict(FRAME, scene="spheres", width=_log(rng, 160, 2560), height=_log(rng, 90, 1440),
                    instances=_log(rng, 16, 10000), meshes=_log(rng, 1, 32), subdivisions=rng.randint(2, 6),
                    ao=1 if denoise else _log(rng, 1, 64), points=_log(rng, 1, 64), spots=_log(rng, 1, 16),
                    light_samples=1 if denoise else rng.choice([1, 1, 2]), sampler=1 if denoise else rng.choice([0, 1]),
                    cull=rng.random() < 0.75, denoise=denoise)
    if kind == "light":
        return {"kind": "light", "width": _log(rng, 64, 2560), "height": _log(rng, 48, 1440),
                "lights": _log(rng, 1, 145), "ao": rng.choice([0, 1, 4, 16, 33]),
                "light_samples": rng.choice([1, 1, 2, 4])}
    if kind in ("train", "infer"):
        return {"kind": kind, "width": _log(rng, 33, 512), "height": _log(rng, 33, 512), "images": rng.randint(1, 8)}
    if kind == "blas":
        level = rng.randint(0, 6)
        return {"kind": "blas", "subdivisions": level, "keep": _log(rng, 1, 20 * 4 ** level)}
    return {"kind": "batch", "scenes": rng.randint(2, 14), "triangles": _log(rng, 20000, 500000),
            "ao": rng.randint(1, 8)}


# ---------------------------------------------------------------------------- common parts
_stream = None


def _use_stream():
    """The torch stream that all work runs on, so that torch's and the library's are ordered."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    torch.cuda.set_stream(_stream)
    return _stream


def _context():
    stream = _use_stream()
    ctx = L.Context(0)
    ctx.set_stream(stream.cuda_stream)
    return ctx


class _Plane:
    """A plane's memory for torch.as_tensor; the tensor keeps it, and it the plane's owner."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 2}


_FORMATS = {L.PLANE_LIGHT: (4, "<f4"), L.PLANE_TAA: (4, "<f4"), L.PLANE_NORMAL: (4, "<f4"), L.PLANE_DEPTH: (1, "<f4"),
            L.PLANE_DENOISED: (4, "<f4"), L.PLANE_PRIMARY_HIT: (2, "<i4"), L.PLANE_SIGNAL: (4, "<f4")}


def _plane(frame, plane, owner=None):
    """A plane of the frame as a torch tensor over its own memory (owner: what holds the frame)."""
    comps, typestr = _FORMATS.get(plane, (1, "<i4"))
    n = frame.plane_bytes(plane) // (4 * comps)
    shape = (n, comps) if comps > 1 else (n,)
    return torch.as_tensor(_Plane(owner or frame, frame.device_ptr(plane), shape, typestr), device="cuda")


def _slots(case):
    if case["scene"] == "cubes":
        lights = 1 + case["points"]
    else:
        lights = 1 + case["points"] + case["spots"]
    return lights * case["light_samples"]


# ---------------------------------------------------------------------------- frames
def _scene(case, seed):
    if case["scene"] == "cubes":
        s = L.HostScene(3, seed=seed, width=case["width"], height=case["height"], instances=case["instances"],
                        point_lights=case["points"], ao_samples=case["ao"], light_samples=case["light_samples"],
                        sampler=case["sampler"])
    else:
        s = L.HostScene(2, seed=seed, width=case["width"], height=case["height"], instances=case["instances"],
                        meshes=case["meshes"], subdivisions=case["subdivisions"], point_lights=case["points"],
                        spot_lights=case["spots"], ao_samples=case["ao"], light_samples=case["light_samples"],
                        sampler=case["sampler"])
    return s


def _prepare_frame(case, seed):
    ctx = _context()
    g = L.GPUScene(ctx, _scene(case, seed))
    g.frame.set_shadow_cull(case["cull"])
    st = {"case": case, "ctx": ctx, "scene": g, "n": 0}
    if case["denoise"]:
        st["denoiser"] = D.Denoiser(ctx)
        st["denoiser"].load()
    g.update_resources_gpu()
    st["planes"] = {"light": _plane(g.frame, L.PLANE_LIGHT), "depth": _plane(g.frame, L.PLANE_DEPTH),
                    "normal": _plane(g.frame, L.PLANE_NORMAL), "albedo": _plane(g.frame, L.PLANE_ALBEDO),
                    "material": _plane(g.frame, L.PLANE_MATERIAL), "hit": _plane(g.frame, L.PLANE_PRIMARY_HIT),
                    "shadow_bits": _plane(g.frame, L.PLANE_SHADOW_BITS), "ao_bits": _plane(g.frame, L.PLANE_AO_BITS)}
    if case["denoise"]:
        st["planes"]["signal"] = _plane(g.frame, L.PLANE_SIGNAL)
        st["planes"]["denoised"] = _plane(g.frame, L.PLANE_DENOISED)
    return st


def _run_frame(st):
    case, g = st["case"], st["scene"]
    out = dict(st["planes"])
    if case["denoise"]:
        g.update_resources_gpu()
        g.frame.gbuffer(g.tlas)
        g.frame.trace(g.tlas, 3)
        st["denoiser"].denoise(g.frame)
        g.frame.light_pass(L.LIGHT_PASS_DENOISED)
    else:
        g.render(3)
    if case["post"]:
        g.frame.taa(True)
        g.frame.compose(source_taa=True)
        h = g.frame.luminance_histogram(source_taa=True)
        out["taa"] = _plane(g.frame, L.PLANE_TAA)
        out["compose"] = _plane(g.frame, L.PLANE_COMPOSE)
        out["bins"] = h["bins"].astype(np.int64)
        out["luminance"] = h["average_luminance"]
    return out


def _work_frame(case):
    pixels, slots = case["width"] * case["height"], _slots(case)
    lit = (0.6 if case["scene"] == "cubes" else 0.23) * pixels
    tris = 12 if case["scene"] == "cubes" else 20 * 4 ** case["subdivisions"] * min(case["meshes"], case["instances"])
    # planes out (40 B of G-buffer, 16 B of light), one bit per sample, instances and ModelBlocks
    # in, and of the meshes the triangles that the pixels can show (one node and one triangle each)
    nbytes = pixels * 56 + lit * (slots + case["ao"]) / 8 + case["instances"] * (64 + 128) + min(tris, lit) * 160
    # a ray: set-up and one box and one triangle test; a light of a lit pixel: one BRDF
    flops = pixels * 60 + lit * ((slots + case["ao"]) * 80 + slots / case["light_samples"] * 80)
    if case["denoise"]:
        nbytes += lit * (16 + 16 + 16 + 16)
        flops += lit * (31872 + 49 * 14)
    if case["post"]:
        nbytes += pixels * (52 + 20 + 16)
        flops += pixels * 600
    return {"bytes": float(nbytes), "flops": float(flops)}


# ---------------------------------------------------------------------------- the light pass alone
def _smooth(rng, shape, cells, device="cuda"):
    """A smooth random field in [0, 1] over the image: `cells` random values across, interpolated."""
    n = max(2, cells)
    t = torch.from_numpy(rng.random((1, 1, n, n))).to(device)
    return torch.nn.functional.interpolate(t, size=shape, mode="bicubic", align_corners=True)[0, 0].clamp(0, 1)


def _light_inputs(case, seed):
    """G-buffer planes, lights and camera of a smooth surface seen at 5 to 60 units, the float32 and
    8-bit values that both the entry point and the 64-bit evaluation take."""
    rng = np.random.default_rng(seed)
    w, h = case["width"], case["height"]
    near, far, fov = 0.1, 200.0, math.radians(60.0)
    f = 1.0 / math.tan(fov / 2)
    proj = np.zeros((4, 4))                       # rows; depth in [0, 1], y down
    proj[0, 0], proj[1, 1] = f * h / w, -f
    proj[2, 2], proj[2, 3], proj[3, 2] = far / (near - far), near * far / (near - far), -1.0
    a, b = rng.uniform(0, 2 * math.pi), rng.uniform(-0.5, 0.5)
    rot = np.array([[math.cos(a), 0, math.sin(a)], [0, 1, 0], [-math.sin(a), 0, math.cos(a)]]) @ \
        np.array([[1, 0, 0], [0, math.cos(b), -math.sin(b)], [0, math.sin(b), math.cos(b)]])
    cam = rng.uniform(-10, 10, 3)
    view = np.eye(4)
    view[:3, :3], view[:3, 3] = rot.T, -rot.T @ cam
    out = {"cam": cam.astype(np.float32), "proj": proj.astype(np.float32), "view": view.astype(np.float32),
           "inverse_proj": np.linalg.inv(proj).astype(np.float32),
           "inverse_view": np.linalg.inv(view).astype(np.float32)}
    z = 5.0 + 55.0 * _smooth(rng, (h, w), 6)
    lit = _smooth(rng, (h, w), 9) > 0.4
    depth = torch.where(lit, (proj[2, 2] * -z + proj[2, 3]) / z, torch.ones_like(z)).float()
    n = torch.stack([_smooth(rng, (h, w), 14) * 2 - 1, _smooth(rng, (h, w), 14) * 2 - 1,
                     0.3 + _smooth(rng, (h, w), 14)], -1)
    n = n / n.norm(dim=-1, keepdim=True) @ torch.from_numpy(rot.T.copy()).to(n)
    normal = torch.zeros((h, w, 4), dtype=torch.float32, device="cuda")
    normal[..., :3] = torch.where(lit[..., None], n, torch.zeros_like(n)).float()
    normal[..., 3] = lit.float()

    def packed(lo, hi):
        c = [(lo[k] + (hi[k] - lo[k]) * _smooth(rng, (h, w), 11)).mul(255).round().to(torch.int64) for k in range(4)]
        v = c[0] | c[1] << 8 | c[2] << 16 | c[3] << 24
        return torch.where(lit, v, torch.zeros_like(v))

    out["albedo"] = packed((0, 0, 0, 1), (1, 1, 1, 1))
    out["material"] = packed((0.05, 0, 1, 1), (1, 1, 1, 1))
    out["emission"] = packed((0, 0, 0, 1), (0.02, 0.02, 0.02, 1))
    out["depth"], out["normal"], out["lit"] = depth, normal, lit
    words = (w * h + 31) // 32
    planes = case["lights"] * case["light_samples"] + case["ao"]
    bits = torch.zeros((planes, words * 32), dtype=torch.bool, device="cuda")
    for k in range(planes):
        bits[k, :w * h] = ((_smooth(rng, (h, w), 24) > 0.55) & lit).reshape(-1)
    out["bits"] = bits
    k = case["lights"]
    out["type"] = np.array([(2, 0, 0, 0, 1)[i % 5] for i in range(k)])
    out["color"] = rng.uniform(0.5, 1.0, (k, 3)).astype(np.float32)
    out["intensity"] = np.where(out["type"] == 2, rng.uniform(1, 3, k), rng.uniform(100, 1000, k)).astype(np.float32)
    d = rng.normal(size=(k, 3))
    out["direction"] = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    out["position"] = np.where(out["type"][:, None] == 2, -1e4 * out["direction"],
                               cam + rng.uniform(-40, 40, (k, 3))).astype(np.float32)
    return out


_INNER, _OUTER = np.float32(math.radians(60.0)), np.float32(math.radians(50.0))


def _pack_bits(bits):
    w = (torch.ones(32, dtype=torch.int64, device=bits.device) << torch.arange(32, device=bits.device))
    rows = [(b.view(-1, 32).to(torch.int64) * w).sum(-1).cpu().numpy().astype(np.uint32) for b in bits]
    return np.stack(rows)


def _prepare_light(case, seed):
    ctx = _context()
    x = _light_inputs(case, seed)
    s = _abi.Scene()
    s.ambient_light_color[:] = [1.0, 1.0, 1.0]
    s.ambient_light_intensity = 0.2
    for name in ("proj", "view", "inverse_proj", "inverse_view"):
        getattr(s, name)[:] = x[name].T.reshape(-1).tolist()
    s.cam_pos[:] = x["cam"].tolist()
    s.num_lights, s.ao_min, s.ao_max, s.ao_num_samples = case["lights"], 1e-4, 2.0, case["ao"]
    s.shadow_type, s.sampler = L.SHADOW_RAYTRACING, L.SAMPLER_PARITY
    lights = (_abi.Light * case["lights"])()
    for i, lt in enumerate(lights):
        lt.color[:], lt.position[:] = x["color"][i].tolist(), x["position"][i].tolist()
        lt.direction[:], lt.intensity = x["direction"][i].tolist(), float(x["intensity"][i])
        lt.inner_angle, lt.outer_angle = float(_INNER), float(_OUTER)
        lt.type, lt.num_shadow_samples, lt.radius, lt.shadow_map = int(x["type"][i]), case["light_samples"], 2.0, -1
    f = ctx.frame(case["width"], case["height"])
    f.upload(s, lights, case["lights"], None, 0)
    for plane, name in ((L.PLANE_ALBEDO, "albedo"), (L.PLANE_MATERIAL, "material"), (L.PLANE_EMISSION, "emission")):
        f.write(plane, x[name].cpu().numpy().astype(np.uint32))
    f.write(L.PLANE_NORMAL, x["normal"].cpu().numpy())
    f.write(L.PLANE_DEPTH, x["depth"].cpu().numpy())
    slots = case["lights"] * case["light_samples"]
    bits = _pack_bits(x["bits"])
    f.write(L.PLANE_SHADOW_BITS, bits[:slots])
    if case["ao"]:
        f.write(L.PLANE_AO_BITS, bits[slots:])
    return {"case": case, "ctx": ctx, "frame": f, "light": _plane(f, L.PLANE_LIGHT)}


def _run_light(st):
    st["frame"].light_pass()
    return st["light"]


def _exact_light(case, seed):
    """light.frag's sum over the lights, in 64 bits."""
    x = _light_inputs(case, seed)
    w, h = case["width"], case["height"]
    dev, f64 = "cuda", torch.float64
    pix = torch.nonzero(x["lit"].reshape(-1))[:, 0]
    t = lambda v: torch.as_tensor(np.asarray(v, np.float64), dtype=f64, device=dev)  # noqa: E731
    ux, uy = (pix % w + 0.5) / w, (torch.div(pix, w, rounding_mode="floor") + 0.5) / h
    clip = torch.stack([ux * 2 - 1, uy * 2 - 1, x["depth"].reshape(-1)[pix].double(), torch.ones_like(ux)], -1)
    v = clip @ t(x["inverse_proj"]).T
    p = ((v / v[:, 3:]) @ t(x["inverse_view"]).T)[:, :3]
    N = x["normal"].reshape(-1, 4)[pix, :3].double()

    def u8(name, k):
        return ((x[name].reshape(-1)[pix] >> (8 * k)) & 255).double() / 255.0

    albedo = torch.stack([u8("albedo", k) for k in range(3)], -1) ** 2.2
    rough, metal, occ = (u8("material", k)[:, None] for k in range(3))
    emission = torch.stack([u8("emission", k) for k in range(3)], -1)
    dot = lambda a, b: (a * b).sum(-1, keepdim=True)  # noqa: E731
    unit = lambda a: a / a.norm(dim=-1, keepdim=True)  # noqa: E731
    V = unit(t(x["cam"]) - p)
    F0 = 0.04 * (1 - metal) + albedo * metal
    k1 = (rough + 1) ** 2 / 8
    a2 = rough ** 4
    nv = dot(N, V).clamp_min(0)
    Lo = torch.zeros_like(p)
    ns = case["light_samples"]
    for i in range(case["lights"]):
        pos, direction, typ = t(x["position"][i]), t(x["direction"][i]), int(x["type"][i])
        to = pos - p
        Lv = unit(to) if typ != 2 else unit(-direction).expand_as(p)
        att = torch.ones_like(nv) if typ == 2 else 1 / dot(to, to)
        if typ == 1:
            att = att * ((dot(Lv, unit(-direction)) - float(_OUTER)) / (float(_INNER) - float(_OUTER))).clamp(0, 1)
        shadow = x["bits"][i * ns:(i + 1) * ns][:, pix].double().mean(0)[:, None]
        radiance = t(x["color"][i]) * float(x["intensity"][i]) * att * (1 - shadow)
        H = unit(V + Lv)
        nl, nh = dot(N, Lv).clamp_min(0), dot(N, H).clamp_min(0)
        D_ = a2 / (math.pi * (nh ** 2 * (a2 - 1) + 1) ** 2)
        G = nv / (nv * (1 - k1) + k1) * nl / (nl * (1 - k1) + k1)
        F = F0 + (1 - F0) * (1 - dot(H, V).clamp(0, 1)).clamp(0, 1) ** 5
        spec = D_ * G * F / (4 * nv * nl + 1e-4)
        Lo = Lo + ((1 - F) * (1 - metal) * albedo / math.pi + spec) * radiance * nl
    slots = case["lights"] * ns
    ao = x["bits"][slots:][:, pix].double().mean(0)[:, None] if case["ao"] else torch.ones_like(nv)
    out = torch.full((h * w, 4), 0.2, dtype=f64, device=dev)
    out[:, 3] = 1.0
    out[pix, :3] = 0.2 * albedo * occ * ao + Lo + emission
    return out


def _work_light(case):
    lit = 0.6 * case["width"] * case["height"]
    slots = case["lights"] * case["light_samples"]
    return {"bytes": lit * (32 + 16 + 16 + (slots + case["ao"]) / 8), "flops": lit * (case["lights"] * 100.0 + 60)}


# ---------------------------------------------------------------------------- the denoiser
def _images(case, seed):
    """Feature planes, distances, the noisy split and targets of images with smooth surfaces, a third
    of them background, 1-sample AO and shadow noise."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, h, w = case["images"], case["height"], case["width"]
    rnd = lambda *s: torch.rand(*s, generator=g, device="cuda")  # noqa: E731

    def smooth(c, cells):
        t = rnd(n, c, cells, cells)
        return torch.nn.functional.interpolate(t, size=(h, w), mode="bicubic", align_corners=True).clamp(0, 1)

    valid = smooth(1, 7)[:, 0] > 0.4
    depth = torch.where(valid, 5 + 20 * smooth(1, 6)[:, 0], torch.zeros(n, h, w, device="cuda"))
    ao_t, sh_t = smooth(1, 12)[:, 0], smooth(1, 16)[:, 0]
    ao = (rnd(n, h, w) < ao_t).float()
    frac = (rnd(n, h, w, 5) < sh_t[..., None]).float()
    nrm = smooth(3, 10).permute(0, 2, 3, 1) * 2 - 1
    nrm = nrm / nrm.norm(dim=-1, keepdim=True).clamp_min(1e-3)
    un = smooth(3, 9).permute(0, 2, 3, 1) * 2
    part = rnd(n, h, w, 5)
    part = part / part.sum(-1, keepdim=True)
    lit = (part * frac).sum(-1)
    alb = smooth(1, 20)[:, 0]
    feat = torch.stack([ao, frac.mean(-1), nrm[..., 0], nrm[..., 1], nrm[..., 2], torch.zeros_like(ao),
                        smooth(1, 8)[:, 0], alb], -1) * valid[..., None]
    noisy = torch.cat([un * lit[..., None], ao[..., None]], -1) * valid[..., None]
    uns = torch.cat([un, frac.mean(-1)[..., None]], -1) * valid[..., None]
    target = torch.cat([sh_t[..., None].expand(n, h, w, 3), ao_t[..., None]], -1) * valid[..., None]
    return {"feat": feat.to(torch.bfloat16).contiguous(), "depth": depth.contiguous(), "noisy": noisy.contiguous(),
            "uns": uns.contiguous(), "target": target.contiguous()}


def _prepare_denoiser(case, seed):
    ctx = _context()
    x = _images(case, seed)
    den = D.Denoiser(ctx)
    den.load()
    b = _abi.DenoiseBatch()
    b.features, b.lin_depth = x["feat"].data_ptr(), x["depth"].data_ptr()
    b.noisy, b.unshadowed = x["noisy"].data_ptr(), x["uns"].data_ptr()
    b.target = x["target"].data_ptr() if case["kind"] == "train" else None
    b.weight = None
    b.width, b.height, b.images = case["width"], case["height"], case["images"]
    out = torch.zeros_like(x["noisy"])
    return {"case": case, "ctx": ctx, "den": den, "batch": b, "keep": x, "out": out}


def _run_train(st):
    grad, loss = st["den"].gradient(st["batch"])
    return {"grad": grad, "loss": loss}


def _run_infer(st):
    st["den"].infer(st["batch"], st["out"].data_ptr())
    return st["out"]


def _params():
    p = torch.from_numpy(np.fromfile(WEIGHTS, np.float32)).cuda().double()
    out, o = [], 0
    for n, k in ((64, 72), (64, 64), (64, 64), (49, 64)):
        out += [p[o:o + n * k].view(n, k).clone(), p[o + n * k:o + n * k + n].clone()]
        o += n * k + n
    return out


def _network(x, i, params):
    """The denoiser's forward pass over image i, in 64 bits: (output rows of the valid pixels, their index)."""
    d = x["depth"][i].double()
    h, w = d.shape
    pix = torch.nonzero(d.reshape(-1) > 0)[:, 0]
    py, px = torch.div(pix, w, rounding_mode="floor"), pix % w
    at = lambda t, dy, dx: t[(py + dy).clamp(0, h - 1), (px + dx).clamp(0, w - 1)]  # noqa: E731
    dc = d.reshape(-1)[pix]
    f = x["feat"][i].double()
    cols = []
    for tap in range(9):
        dy, dx = tap // 3 - 1, tap % 3 - 1
        c = at(f, dy, dx).clone()
        dq = at(d, dy, dx)
        c[:, 5] = torch.where(dq > 0, ((dq - dc) / dc).clamp(-1, 1), torch.zeros_like(dc))
        cols.append(c)
    a = torch.cat(cols, 1)
    for l in range(3):
        a = torch.relu(a @ params[2 * l].T + params[2 * l + 1])
    wgt = torch.softmax(a @ params[6].T + params[7], 1)
    s, u = x["noisy"][i].double(), x["uns"][i].double()
    acc, au = 0, 0
    for k in range(49):
        dy, dx = k // 7 - 3, k % 7 - 3
        acc = acc + wgt[:, k:k + 1] * at(s, dy, dx)
        au = au + wgt[:, k:k + 1] * at(u, dy, dx)[:, :3]
    ratio = torch.where(au > 0, (acc[:, :3] / torch.where(au > 0, au, torch.ones_like(au))).clamp(0, 1),
                        torch.ones_like(au))
    return torch.cat([ratio, acc[:, 3:]], 1), pix


def _exact_denoiser(case, seed):
    x = _images(case, seed)
    params = _params()
    if case["kind"] == "infer":
        out = torch.zeros(x["noisy"].shape, dtype=torch.float64, device="cuda")
        with torch.no_grad():
            for i in range(case["images"]):
                y, pix = _network(x, i, params)
                out[i].view(-1, 4)[pix] = y
        return out
    for p in params:
        p.requires_grad_(True)
    total, npx = 0.0, case["images"] * case["width"] * case["height"]
    cw = torch.tensor([1 / 3, 1 / 3, 1 / 3, 1.0], dtype=torch.float64, device="cuda")
    for i in range(case["images"]):
        y, pix = _network(x, i, params)
        loss = (cw * (y - x["target"][i].double().view(-1, 4)[pix]) ** 2).sum() / npx
        loss.backward()
        total += float(loss.detach())
    grad = torch.cat([p.grad.reshape(-1) for p in params])
    return {"grad": grad, "loss": total}


def _work_denoiser(case):
    px = case["images"] * case["width"] * case["height"]
    if case["kind"] == "infer":
        return {"bytes": px * (16 + 4 + 16 + 16 + 16.0), "flops": 0.65 * px * (31872.0 + 49 * 14)}
    return {"bytes": px * (16 + 4 + 16 + 16 + 16.0) + 16177 * 4, "flops": 0.65 * px * (3 * 31872.0 + 49 * 42)}


# ---------------------------------------------------------------------------- BLAS
def _prepare_blas(case, seed):
    v, idx = L.HostScene(2, seed=seed, width=16, height=16, meshes=1, instances=1,
                         subdivisions=max(case["subdivisions"], 1)).meshes()[0]
    n = min(case["keep"], idx.size // 3)
    idx = idx[:3 * n]
    _use_stream()
    dev = lambda *s: torch.zeros(s, dtype=torch.int32, device="cuda")  # noqa: E731
    return {"v": torch.from_numpy(np.ascontiguousarray(v, np.float32)).cuda(),
            "i": torch.from_numpy(idx.view(np.int32).copy()).cuda(), "nodes": dev(max(n - 1, 1), 16),
            "tris": dev(n, 12), "morton": dev(n), "order": dev(n)}


def _run_blas(st):
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    status = L.lib.luz_blas_build_noalloc(p(st["v"]), st["v"].shape[0], p(st["i"]), st["i"].numel(), p(st["nodes"]),
                                          p(st["tris"]), p(st["morton"]), p(st["order"]),
                                          C.c_void_p(_stream.cuda_stream))
    if status != 0:
        raise RuntimeError(f"BLAS build: status {status}")
    return {k: st[k] for k in ("nodes", "tris", "morton", "order")}


def _work_blas(case):
    n = min(case["keep"], 20 * 4 ** max(case["subdivisions"], 1))
    return {"bytes": n * (12 + 24 + 64 + 48 + 8.0), "flops": n * 100.0}


# ---------------------------------------------------------------------------- batches
_SIZES = ((256, 256), (512, 512), (1280, 720), (1920, 1080), (509, 311))


def _batch_scenes(case):
    """(size, triangles) of each scene: of the case alone, the seed makes the scenes' contents."""
    rng = np.random.default_rng(case["scenes"] * 1000003 + case["triangles"])
    for i in range(case["scenes"]):
        tris = int(round(math.exp(rng.uniform(math.log(1000), math.log(case["triangles"])))))
        yield _SIZES[(i * 3 + 1) % len(_SIZES)], tris


def _prepare_batch(case, seed):
    ctx = _context()
    ctx.set_blue_noise(L.blue_noise())
    scenes = [L.HostScene(6, seed=seed * 100 + i, width=w, height=h, triangles=tris, ao_samples=case["ao"])
              for i, ((w, h), tris) in enumerate(_batch_scenes(case))]
    b = L.Batch(ctx, scenes)
    planes = [{"light": _plane(f, L.PLANE_LIGHT, b), "hit": _plane(f, L.PLANE_PRIMARY_HIT, b),
               "shadow_bits": _plane(f, L.PLANE_SHADOW_BITS, b), "ao_bits": _plane(f, L.PLANE_AO_BITS, b)}
              for f in b.frames]
    return {"ctx": ctx, "batch": b, "planes": planes}


def _run_batch(st):
    st["batch"].render(3)
    return st["planes"]


def _work_batch(case):
    pixels = sum(w * h for (w, h), _ in _batch_scenes(case))
    lit = 0.4 * pixels
    slots = 8
    return {"bytes": pixels * 56 + lit * (slots + case["ao"]) / 8, "flops": pixels * 60 + lit * (slots + case["ao"]) * 80 +
            lit * slots * 80.0}


# ---------------------------------------------------------------------------- the interface
_PREPARE = {"frame": _prepare_frame, "light": _prepare_light, "train": _prepare_denoiser, "infer": _prepare_denoiser,
            "blas": _prepare_blas, "batch": _prepare_batch}
_WORK = {"frame": _work_frame, "light": _work_light, "train": _work_denoiser, "infer": _work_denoiser,
         "blas": _work_blas, "batch": _work_batch}


def prepare(case, seed):
    st = _PREPARE[case["kind"]](case, int(seed))
    st["run"] = case["kind"]
    return st


_RUN = {"frame": _run_frame, "light": _run_light, "train": _run_train, "infer": _run_infer, "blas": _run_blas,
        "batch": _run_batch}


def run(state):
    return _RUN[state["run"]](state)


def work(case):
    return _WORK[case["kind"]](case)


def exact(case, seed):
    """The 64-bit values of the light pass and the denoiser. A traced frame has none here: it
    would take a 64-bit ray tracer over millions of rays; BLAS outputs are bytes."""
    if case["kind"] == "light":
        return _exact_light(case, int(seed))
    if case["kind"] in ("train", "infer"):
        return _exact_denoiser(case, int(seed))
    return None
