"""Performance cases of pyvr_gb300: the work a user has the framework do.

Every case goes through a public entry point (``VolumeRenderer``,
``BatchRenderer``, ``DeviceVolume``, ``DeviceLUT``, ``NativeRenderServer``,
``render_views``) on seeded synthetic scenes: value-noise volumes, orbit
cameras, piecewise-linear transfer functions, the ``RenderConfig`` presets.

  listed()             the cases that are always measured
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what a program has in hand before the call
  run(state)           one pass through the entry points, and its outputs
  work(case)           bytes and operations a pass cannot do without
  exact(case, seed)    the float outputs of run() in 64-bit arithmetic

The 64-bit march (``_march64``) is plain torch, written from the renderer's
documented semantics: no code of the package takes part in it.
"""

import math

import numpy as np
import torch

from pyvr_gb300 import (Camera, ColorTransferFunction, Light, OpacityTransferFunction, RenderConfig,
                        Volume, VolumeRenderer)

BOUNDS = (np.full(3, -1.0, np.float32), np.full(3, 1.0, np.float32))
LIGHT_DIRECTION = (1.0, -1.0, 0.0)
AMBIENT, DIFFUSE = 0.2, 0.8
# step, most steps (RenderConfig presets; the reference step is 0.01)
PRESETS = {"preview": (0.05, 50), "fast": (0.02, 100), "balanced": (0.01, 500),
           "high_quality": (0.005, 1000)}
REFERENCE_STEP = 0.01


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # an interactive session on a small volume (64^3, 256^2): the camera
        # moves, one frame comes back as bytes -- the smallest whole call
        dict(name="frame_small", kind="frame", d=64, h=64, w=64, storage="f32", width=256, height=256,
             preset="balanced", arithmetic="fast", floats=False),
        # the plain renderer's frame: 256^3 uint8, 1024^2, high quality
        dict(name="frame_plain_u8", kind="frame", d=256, h=256, w=256, storage="u8", width=1024, height=1024,
             preset="high_quality", arithmetic="fast", floats=False),
        # the exact arithmetic (images equal to the CPU oracle's), with the
        # float image, as regression checks and comparisons ask for it
        dict(name="frame_exact_f16", kind="frame", d=160, h=160, w=160, storage="f16", width=512, height=512,
             preset="balanced", arithmetic="exact", floats=True),
        # one render into device buffers, no normals, odd sizes: a pipeline
        # that keeps its frames on the GPU
        dict(name="device_odd_f32", kind="device", d=201, h=150, w=173, storage="f32", normals="none",
             records="float", brick=3, width=643, height=361, preset="balanced"),
        # many uneven renders in one call: thumbnails, parameter sweeps
        dict(name="batch_uneven", kind="batch", mix=0, jobs=32, min_dim=32, max_dim=320, min_res=128, max_res=768,
             records="half_normals"),
        # an orbit frame of a served volume at 512^2 (16^3 bricks, half
        # records), one render per call: what a server's launch does
        dict(name="serve_orbit", kind="device", d=384, h=384, w=384, storage="u8", normals="device",
             records="half_normals", brick=4, width=512, height=512, preset="balanced"),
        # the render server under a burst of 40 requests over six resident
        # volumes: orbit frames, edited transfer functions, a few captures
        dict(name="serve_burst", kind="serve", mix=0, requests=40, volumes=6, min_dim=128, max_dim=320, res=512),
        # a transfer-function edit in a preview: the table is rebuilt on the
        # device and a small frame rendered
        dict(name="tf_edit_preview", kind="tf_edit", d=128, h=128, w=128, storage="f16", points=8, lut=256,
             width=256, height=256, preset="preview"),
        # a new volume arrives at a server: upload from page-locked memory,
        # device normals, layout, first frame
        dict(name="load_f16_512", kind="load", d=512, h=512, w=512, storage="f16", records="half_normals",
             brick=4, width=512, height=512, preset="balanced", read_normals=False),
        # a new non-cubic float32 volume through the drop-in renderer:
        # load_volume from an ordinary array, compute_normals, render
        dict(name="load_f32_box", kind="reload", d=128, h=200, w=161, storage="f32", width=512, height=512,
             preset="balanced"),
        # one optimisation step of a transfer function: 8 views of 512^2
        # forward, and backward to the table
        dict(name="train_lut", kind="train", n=128, views=8, width=512, height=512, lut=256, normals=True,
             voxels=False),
        # one optimisation step of voxels and table together, few small odd
        # views, no normals
        dict(name="train_voxels", kind="train", n=72, views=3, width=251, height=197, lut=128, normals=False,
             voxels=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "device", "device", "batch", "serve", "tf_edit", "load", "reload", "train"])
    preset = rng.choice(["fast", "balanced", "balanced", "high_quality"])
    storage = rng.choice(["u8", "f16", "f32"])
    if kind == "frame":
        n = _log(rng, 48, 288)
        return dict(kind=kind, d=n, h=n, w=n, storage=storage, width=_log(rng, 128, 1024),
                    height=_log(rng, 128, 1024), preset=preset, arithmetic=rng.choice(["fast", "fast", "exact"]),
                    floats=rng.random() < 0.3)
    if kind == "device":
        dims = [_log(rng, 40, 400)] * 3 if rng.random() < 0.5 else [_log(rng, 40, 320) for _ in range(3)]
        return dict(kind=kind, d=dims[0], h=dims[1], w=dims[2], storage=storage,
                    normals=rng.choice(["none", "device", "device"]),
                    records=rng.choice(["float", "half_exact", "half_normals"]), brick=rng.choice([2, 3, 4]),
                    width=_log(rng, 64, 1024), height=_log(rng, 64, 1024), preset=preset)
    if kind == "batch":
        return dict(kind=kind, mix=rng.randint(1, 10 ** 6), jobs=rng.randint(2, 32), min_dim=32, max_dim=_log(rng, 96, 320),
                    min_res=96, max_res=_log(rng, 192, 768), records=rng.choice(["float", "half_normals"]))
    if kind == "serve":
        return dict(kind=kind, mix=rng.randint(1, 10 ** 6), requests=rng.randint(8, 40), volumes=rng.randint(2, 6),
                    min_dim=96, max_dim=_log(rng, 128, 320), res=_log(rng, 192, 512))
    if kind == "tf_edit":
        n = _log(rng, 48, 200)
        return dict(kind=kind, d=n, h=n, w=n, storage=rng.choice(["u8", "f16"]), points=rng.randint(2, 24),
                    lut=rng.choice([64, 256, 256, 1024]), width=_log(rng, 96, 512), height=_log(rng, 96, 512),
                    preset=rng.choice(["preview", "fast"]))
    if kind == "load":
        n = _log(rng, 64, 440)
        return dict(kind=kind, d=n, h=n, w=n, storage=storage,
                    records="float" if storage == "f32" else "half_normals", brick=rng.choice([3, 4]),
                    width=_log(rng, 128, 512), height=_log(rng, 128, 512), preset="balanced",
                    # small volumes: the normals come back to the host too
                    read_normals=n <= 128 and rng.random() < 0.7)
    if kind == "reload":
        return dict(kind=kind, d=_log(rng, 48, 256), h=_log(rng, 48, 256), w=_log(rng, 48, 256), storage=storage,
                    width=_log(rng, 128, 768), height=_log(rng, 128, 768), preset="balanced")
    return dict(kind="train", n=_log(rng, 32, 128), views=rng.randint(1, 6), width=_log(rng, 96, 448),
                height=_log(rng, 96, 448), lut=rng.choice([64, 256, 256, 777]), normals=rng.random() < 0.5,
                voxels=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# Seeded inputs
# ---------------------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _noise(dims, rng):
    """Value noise in [0, 1] on the (D, H, W) grid: four octaves of uniform
    lattices, trilinearly upsampled, weights 1, 1/2, 1/4, 1/8."""
    acc = torch.zeros(tuple(dims), dtype=torch.float32, device=_device())
    for k, lat in enumerate((8, 16, 32, 64)):
        v = torch.from_numpy(rng.random((lat, lat, lat), dtype=np.float32)).to(acc.device)
        acc += 0.5 ** k * torch.nn.functional.interpolate(v[None, None], size=tuple(dims), mode="trilinear",
                                                          align_corners=True)[0, 0]
    lo, hi = acc.min(), acc.max()
    return (acc - lo) / (hi - lo)


def _stored(noise, storage):
    if storage == "u8":
        return torch.round(noise * 255.0).to(torch.uint8)
    return noise.to(torch.float16 if storage == "f16" else torch.float32)


def _scale(storage):
    return 1.0 / 255.0 if storage == "u8" else 1.0


def _orbit(rng):
    """Orbit parameters (float32 values): azimuth, elevation, distance from
    the volume's centre."""
    return tuple(float(np.float32(rng.uniform(a, b))) for a, b in ((-math.pi, math.pi), (-0.8, 0.8), (2.6, 3.6)))


def _camera(orbit):
    return Camera.from_spherical(target=np.zeros(3, np.float32), azimuth=orbit[0], elevation=orbit[1], roll=0.0,
                                 distance=orbit[2])


def _tf_points(rng, n):
    """n opacity points in [0, 0.3] and 6 colour points."""
    xs = np.sort(rng.random(n))
    otf = [(float(x), float(y)) for x, y in zip(xs, rng.uniform(0.0, 0.3, n))]
    ctf = [(float(x), tuple(map(float, c))) for x, c in zip(np.linspace(0.0, 1.0, 6), rng.random((6, 3)))]
    return ctf, otf


def _tfs(points, lut=256):
    return (ColorTransferFunction(points[0], lut_size=lut), OpacityTransferFunction(points[1], lut_size=lut))


def _light():
    return Light.directional(list(LIGHT_DIRECTION), AMBIENT, DIFFUSE)


def _volume(data):
    return Volume(data=data, min_bounds=BOUNDS[0].copy(), max_bounds=BOUNDS[1].copy())


def _config(preset):
    return getattr(RenderConfig, preset)()


class _records:
    """Volumes laid out inside use this record form; restored afterwards (the
    form is a setting of the whole library)."""

    def __init__(self, mode):
        self.mode = mode

    def __enter__(self):
        from pyvr_gb300.batch import get_compact_records, set_compact_records
        self.prev = get_compact_records()
        set_compact_records(self.mode)

    def __exit__(self, *exc):
        from pyvr_gb300.batch import set_compact_records
        set_compact_records(self.prev)
        return False


def _single(case, seed):
    """The scene of a one-volume case: stored voxels, orbit, TF points."""
    rng = np.random.default_rng(seed)
    data = _stored(_noise((case["d"], case["h"], case["w"]), rng), case["storage"])
    orbit = _orbit(rng)
    return data, orbit, _tf_points(rng, case.get("points", 8))


def _batch_scenes(case, seed):
    """Per job: dims, storage, resolution (from the case's mix), orbit, TF
    points, noise seed (from the seed)."""
    mix, rng = np.random.default_rng(case["mix"]), np.random.default_rng(seed)
    out = []
    for i in range(case["jobs"]):
        dims = tuple(int(round(x)) for x in np.exp(mix.uniform(math.log(case["min_dim"]),
                                                               math.log(case["max_dim"]), 3)))
        res = int(round(math.exp(mix.uniform(math.log(case["min_res"]), math.log(case["max_res"])))))
        out.append(dict(dims=dims, storage=["u8", "f16", "f32"][int(mix.integers(0, 3))], res=res, orbit=_orbit(rng),
                        points=_tf_points(rng, int(mix.integers(4, 13))), noise=int(rng.integers(1 << 31))))
    return out


def _serve_scene(case, seed):
    """Volumes (extent, storage, noise seed) and requests (volume, orbit, TF
    points, side, preset): sizes and kinds from the case's mix, the rest from
    the seed."""
    mix, rng = np.random.default_rng(case["mix"]), np.random.default_rng(seed)
    vols = [(int(round(math.exp(mix.uniform(math.log(case["min_dim"]), math.log(case["max_dim"]))))),
             "u8" if mix.random() < 0.5 else "f16", int(rng.integers(1 << 31))) for _ in range(case["volumes"])]
    sessions = [(list(_orbit(rng)), _tf_points(rng, 6)) for _ in vols]
    reqs = []
    for _ in range(case["requests"]):
        v, u = int(mix.integers(len(vols))), mix.random()
        orbit, points = sessions[v]
        side, preset = case["res"], "balanced"
        if u < 0.75:
            orbit = [orbit[0] + float(rng.normal(0, 0.05)),
                     float(np.clip(orbit[1] + rng.normal(0, 0.05), -1.5, 1.5)), orbit[2]]
        elif u < 0.95:
            points = (points[0], sorted((float(np.clip(x + rng.normal(0, 0.05), 0, 1)), y) for x, y in points[1]))
        else:
            side, preset = 2 * case["res"], "high_quality"
        sessions[v] = (orbit, points)
        reqs.append((v, tuple(orbit), points, side, preset))
    return vols, reqs


def _train_scene(case, seed):
    """Volume, normals or None, table, target image and orbits of a training
    step, on the device."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    vol = _noise((n, n, n), rng)
    normals = None
    if case["normals"]:
        g = torch.stack(torch.gradient(vol), -1)
        normals = (g / (g.norm(dim=-1, keepdim=True) + 1e-8)).contiguous()
    lut = torch.from_numpy(np.concatenate([rng.random((case["lut"], 3)),
                                           rng.uniform(0.0, 0.3, (case["lut"], 1))], 1).astype(np.float32))
    target = torch.from_numpy(rng.random((case["views"], case["height"], case["width"], 4), dtype=np.float32))
    orbits = [_orbit(rng) for _ in range(case["views"])]
    return vol, normals, lut.to(vol.device), target.to(vol.device), orbits


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------

class _ServerSession:
    """A render server that closes when the last reference to it goes."""

    def __init__(self, server):
        self.server = server

    def __del__(self):
        try:
            self.server.close()
        except Exception:
            pass


def _frame_renderer(case, seed, load):
    data, orbit, points = _single(case, seed)
    r = VolumeRenderer(case["width"], case["height"], config=_config(case["preset"]), light=_light())
    r.set_transfer_functions(*_tfs(points))
    vol = _volume(data.cpu().numpy())
    if load:
        r.load_volume(vol, value_scale=_scale(case["storage"]))
        r.compute_normals()
        r.set_camera(_camera(orbit))
        r.render()  # the first frame lays the volume out
    return r, vol, _camera(orbit)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        r, _, cam = _frame_renderer(case, seed, True)
        return dict(case=case, renderer=r, camera=cam)
    if kind == "reload":
        r, vol, cam = _frame_renderer(case, seed, False)
        return dict(case=case, renderer=r, camera=cam, volume=vol)
    if kind == "train":
        from pyvr_gb300.diff import DiffScene
        vol, normals, lut, target, orbits = _train_scene(case, seed)
        scene = DiffScene([_camera(o) for o in orbits], _light(), RenderConfig.balanced(), case["width"],
                          case["height"])
        return dict(case=case, volume=vol.requires_grad_(case["voxels"]), lut=lut.requires_grad_(True),
                    normals=normals, target=target, scene=scene)

    from pyvr_gb300.batch import BatchRenderer, DeviceLUT, DeviceVolume, RenderJob, Tuning, page_locked_copy
    if kind == "device":
        data, orbit, points = _single(case, seed)
        with _records(case["records"]):
            dv = DeviceVolume(_volume(data.cpu().numpy()), value_scale=_scale(case["storage"]),
                              normals=case["normals"], brick_log2=case["brick"])
        npx = case["width"] * case["height"] * 4
        job = RenderJob(dv, DeviceLUT(*_tfs(points)), _camera(orbit), _light(), _config(case["preset"]),
                        case["width"], case["height"], torch.empty(npx, dtype=torch.uint8, device="cuda"),
                        torch.empty(npx, dtype=torch.float32, device="cuda") if case["normals"] == "none" else None)
        return dict(case=case, batch=BatchRenderer(capacity=1, slots=2), job=job)
    if kind == "batch":
        jobs = []
        with _records(case["records"]):
            for s in _batch_scenes(case, seed):
                data = _stored(_noise(s["dims"], np.random.default_rng(s["noise"])), s["storage"])
                dv = DeviceVolume(_volume(data.cpu().numpy()), value_scale=_scale(s["storage"]), normals="device")
                jobs.append(RenderJob(dv, DeviceLUT(*_tfs(s["points"])), _camera(s["orbit"]), _light(),
                                      RenderConfig.balanced(), s["res"], s["res"],
                                      torch.empty(s["res"] * s["res"] * 4, dtype=torch.uint8, device="cuda")))
        return dict(case=case, batch=BatchRenderer(capacity=len(jobs), slots=2), jobs=jobs)
    if kind == "tf_edit":
        data, orbit, points = _single(case, seed)
        with _records("half_normals"):
            dv = DeviceVolume(_volume(data.cpu().numpy()), value_scale=_scale(case["storage"]), normals="device")
        ctf, otf = _tfs(points, case["lut"])
        npx = case["width"] * case["height"] * 4
        job = RenderJob(dv, DeviceLUT.on_device(ctf, otf), _camera(orbit), _light(), _config(case["preset"]),
                        case["width"], case["height"], torch.empty(npx, dtype=torch.uint8, device="cuda"))
        return dict(case=case, batch=BatchRenderer(capacity=1, slots=2), job=job, ctf=ctf, otf=otf)
    if kind == "load":
        data, orbit, points = _single(case, seed)
        npx = case["width"] * case["height"] * 4
        return dict(case=case, volume=_volume(page_locked_copy(data.cpu().numpy())), camera=_camera(orbit),
                    light=_light(), config=_config(case["preset"]), lut=DeviceLUT(*_tfs(points)),
                    batch=BatchRenderer(capacity=1, slots=2),
                    out=torch.empty(npx, dtype=torch.uint8, device="cuda"))
    if kind == "serve":
        from pyvr_gb300.server import NativeRenderServer
        vols, reqs = _serve_scene(case, seed)
        server = NativeRenderServer(budget_bytes=4 << 30, brick_log2=4, tuning=Tuning(), lut_reserve=128)
        with _records("half_normals"):
            for i, (n, storage, noise) in enumerate(vols):
                data = _stored(_noise((n, n, n), np.random.default_rng(noise)), storage)
                server.cache.insert(i, _volume(data.cpu().numpy()), _scale(storage), server._free_volume)
        torch.cuda.synchronize()
        requests = [dict(kind="render", volume_id=v, camera=_camera(o), light=_light(), config=_config(preset),
                         color_tf=_tfs(p)[0], opacity_tf=_tfs(p)[1], width=side, height=side)
                    for v, o, p, side, preset in reqs]
        return dict(case=case, session=_ServerSession(server), requests=requests)
    raise ValueError(f"unknown kind {kind!r}")


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "frame":
        from pyvr_gb300.batch import arithmetic
        r = state["renderer"]
        with arithmetic(case["arithmetic"]):
            r.set_camera(state["camera"])
            if case["floats"]:
                return r.render_float()
            return np.frombuffer(r.render(), np.uint8)
    if kind == "reload":
        r = state["renderer"]
        r.load_volume(state["volume"], value_scale=_scale(case["storage"]))
        r.compute_normals()
        r.set_camera(state["camera"])
        return np.frombuffer(r.render(), np.uint8)
    if kind == "train":
        from pyvr_gb300.diff import render_views
        vol, lut = state["volume"], state["lut"]
        vol.grad = lut.grad = None
        image = render_views(vol, lut, state["scene"], normals=state["normals"])
        loss = ((image - state["target"]) ** 2).mean()
        loss.backward()
        out = [image.detach(), lut.grad]
        return out + [vol.grad] if case["voxels"] else out
    stream = torch.cuda.current_stream()
    if kind in ("device", "tf_edit"):
        job = state["job"]
        if kind == "tf_edit":
            job.lut.build(state["ctf"], state["otf"], stream=stream)
        state["batch"].render([job], stream=stream)
        return [job.out_rgba8] if job.out_rgba32f is None else [job.out_rgba8, job.out_rgba32f]
    if kind == "batch":
        state["batch"].render(state["jobs"], stream=stream)
        return [j.out_rgba8 for j in state["jobs"]]
    if kind == "load":
        from pyvr_gb300.batch import DeviceVolume, RenderJob
        with _records(case["records"]):
            dv = DeviceVolume(state["volume"], value_scale=_scale(case["storage"]), normals="device",
                              brick_log2=case["brick"])
        state["batch"].render([RenderJob(dv, state["lut"], state["camera"], state["light"], state["config"],
                                         case["width"], case["height"], state["out"])], stream=stream)
        normals = [dv.read_normals()] if case["read_normals"] else []
        dv.close()
        return [state["out"]] + normals
    from pyvr_gb300.server import RenderRequest
    futures = [state["session"].server.submit(RenderRequest(**kw)) for kw in state["requests"]]
    return [f.result(timeout=60) for f in futures]


# ---------------------------------------------------------------------------
# The march in 64 bits (plain torch)
# ---------------------------------------------------------------------------

def _rays(orbit, width, height, step, device):
    """Start points, steps and hits of all pixels, bottom row first.  The
    positions of the samples are part of the renderer's definition (float32
    matrices, float32 ray setup, repeated float32 additions of one step), so
    they are float32 here too; all that is computed at them is float64."""
    az, el, dist = orbit
    eye = dist * np.array([math.cos(el) * math.cos(az), math.cos(el) * math.sin(az), math.sin(el)])
    up = np.array([-math.sin(el) * math.cos(az), -math.sin(el) * math.sin(az), math.cos(el)])
    fwd = -eye / np.linalg.norm(eye)
    right = np.cross(fwd, up)
    right /= np.linalg.norm(right)
    up = np.cross(right, fwd)
    view = np.eye(4)
    view[0, :3], view[1, :3], view[2, :3] = right, up, -fwd
    view[:3, 3] = -view[:3, :3] @ eye
    iv = np.linalg.inv(view.astype(np.float32).astype(np.float64)).astype(np.float32)
    cot = 1.0 / math.tan(math.pi / 8)  # field of view pi / 4
    ip = [np.float32(1.0 / np.float64(np.float32(v))) for v in (cot / (width / height), cot)]
    f32 = lambda v: torch.tensor(np.asarray(v, np.float32), device=device)
    iv, cam = f32(iv), f32(eye)
    x = (torch.arange(width, dtype=torch.float32, device=device) + 0.5) / f32(width) * 2.0 - 1.0
    y = (torch.arange(height, dtype=torch.float32, device=device) + 0.5) / f32(height) * 2.0 - 1.0
    ex, ey = (x * f32(ip[0])).repeat(height), (y * f32(ip[1])).repeat_interleave(width)
    w = [(iv[r, 0] * ex + iv[r, 1] * ey) - iv[r, 2] for r in range(3)]
    d = torch.stack(w, 1) * (1.0 / torch.sqrt((w[0] * w[0] + w[1] * w[1]) + w[2] * w[2]))[:, None]
    inv = 1.0 / d
    t0, t1 = (-1.0 - cam) * inv, (1.0 - cam) * inv
    near, far = torch.minimum(t0, t1).amax(1), torch.maximum(t0, t1).amin(1)
    hit = (near <= far) & (far > 0)
    return cam + d * near.clamp(min=0.0)[:, None], d * f32(step), hit


class _March64:
    """The march of several views over one volume, in float64 at the
    renderer's sample positions.  voxels and normals are (D, H, W[, 3]) tensors; texel (x, y, z) of the world axes is
    element z + D * (y + H * x) of the flat array."""

    def __init__(self, voxels, scale, normals, lut, orbits, width, height, preset):
        self.dev = voxels.device
        self.dims = tuple(voxels.shape)
        self.flat = voxels.reshape(-1).double()
        self.nflat = None if normals is None else normals.reshape(-1, 3).double()
        self.scale, self.lut = scale, lut.double()
        self.step, self.most = PRESETS[preset]
        self.k = float(np.float32(self.step) / np.float32(REFERENCE_STEP))
        rays = [_rays(o, width, height, self.step, self.dev) for o in orbits]
        self.pos, self.delta, self.hit = (torch.cat(x) for x in zip(*rays))
        light = torch.tensor(LIGHT_DIRECTION, dtype=torch.float64, device=self.dev)
        self.light = light / light.norm()

    def _trilinear(self, corners, f):
        c = corners
        fx, fy, fz = f
        lerp = lambda a, b, t: a + t * (b - a)
        z = [lerp(c[2 * i], c[2 * i + 1], fz) for i in range(4)]
        return lerp(lerp(z[0], z[1], fy), lerp(z[2], z[3], fy), fx)

    def samples(self, pos):
        """What the samples at pos (n, 3) compute, and which are in the box."""
        t = (pos + 1.0) * 0.5
        inside = ((t >= 0) & (t <= 1)).all(1)
        t = t[inside].double()
        D, H, W = self.dims
        ext = (W, H, D)
        u = [t[:, a] * ext[a] - 0.5 for a in range(3)]
        lo = [x.floor() for x in u]
        f = [x - l for x, l in zip(u, lo)]
        idx = [(l.long().clamp(0, e - 1), (l.long() + 1).clamp(0, e - 1)) for l, e in zip(lo, ext)]
        at = [idx[2][c] + D * (idx[1][b] + H * idx[0][a]) for a in (0, 1) for b in (0, 1) for c in (0, 1)]
        density = self._trilinear([self.flat[i] for i in at], f) * self.scale
        n = self.lut.shape[0]
        lu = density * n - 0.5
        l0 = lu.floor()
        w = lu - l0
        i0, i1 = l0.clamp(0, n - 1).long(), (l0 + 1).clamp(0, n - 1).long()
        rgba = self.lut[i0] + w[:, None] * (self.lut[i1] - self.lut[i0])
        if self.nflat is None:
            nrm = torch.stack([density, torch.zeros_like(density), torch.zeros_like(density)], 1)
        else:
            nrm = self._trilinear([self.nflat[i] for i in at], [x[:, None] for x in f])
        n2 = (nrm * nrm).sum(1)
        di = torch.where(n2 > 0, (nrm @ self.light) / n2.clamp(min=1e-300).sqrt(), torch.zeros_like(n2))
        e = torch.exp(-rgba[:, 3] * self.k)
        return inside, dict(at=at, f=f, w=w, i0=i0, i1=i1, e=e, alpha=1.0 - e, rgb=rgba[:, :3],
                            light=AMBIENT + DIFFUSE * di.clamp(min=0.0))

    def walk(self, visit):
        """visit(rays, sample) step by step while the accumulated alpha is
        below 0.99; returns the image (n, 4) and the number of samples."""
        acc = torch.zeros((self.pos.shape[0], 4), dtype=torch.float64, device=self.dev)
        alive = self.hit.nonzero()[:, 0]
        pos, d = self.pos[alive], self.delta[alive]
        entered = torch.zeros_like(alive, dtype=torch.bool)
        count = 0
        for i in range(self.most):
            if not alive.numel():
                break
            inside, s = self.samples(pos)
            rays = alive[inside]
            count += rays.numel()
            if visit is not None:
                visit(rays, s, acc)
            tr = 1.0 - acc[rays, 3]
            acc[rays, :3] += (tr * s["alpha"] * s["light"])[:, None] * s["rgb"]
            acc[rays, 3] += tr * s["alpha"]
            pos = pos + d
            # a ray ends once it has left the box; the first steps may still lie outside it
            keep = (acc[alive, 3] < 0.99) & (inside | (~entered & (i < 8)))
            entered = (entered | inside)[keep]
            alive, pos, d = alive[keep], pos[keep], d[keep]
        return acc, count

    def gradients(self, image, gimage, voxels):
        """dL/dlut (and dL/dvoxels) for dL/dimage, from a second walk: the
        radiance behind a sample is what the image holds beyond it."""
        n = self.lut.shape[0]
        ways = 4096  # private copies of the table: few additions meet in one entry
        glut = torch.zeros((ways * n, 4), dtype=torch.float64, device=self.dev)
        gvol = torch.zeros_like(self.flat) if voxels else None

        def visit(rays, s, acc):
            g, tr = gimage[rays], 1.0 - acc[rays, 3]
            alpha, color = s["alpha"], s["light"][:, None] * s["rgb"]
            add = (tr * alpha)[:, None] * color
            behind = image[rays, :3] - acc[rays, :3] - add
            left = (tr * (1.0 - alpha)).clamp(min=1e-300)[:, None]
            dalpha = tr * ((g[:, :3] * (color - behind / left)).sum(1) + g[:, 3] *
                           (1.0 - image[rays, 3]) / left[:, 0])
            drgb = g[:, :3] * (tr * s["light"] * alpha)[:, None]
            d = torch.cat([drgb, (dalpha * self.k * s["e"])[:, None]], 1)
            copy = (rays % ways) * n
            glut.index_add_(0, copy + s["i0"], (1.0 - s["w"])[:, None] * d)
            glut.index_add_(0, copy + s["i1"], s["w"][:, None] * d)
            if gvol is not None:
                gd = (d * (self.lut[s["i1"]] - self.lut[s["i0"]])).sum(1) * n * self.scale
                fx, fy, fz = s["f"]
                weights = [a * b * c for a in (1 - fx, fx) for b in (1 - fy, fy) for c in (1 - fz, fz)]
                for at, w in zip(s["at"], weights):
                    gvol.index_add_(0, at, gd * w)

        self.walk(visit)
        out = [glut.view(ways, n, 4).sum(0)]
        return out + [gvol.view(self.dims)] if voxels else out


def _table(points, n=256):
    x = np.linspace(0.0, 1.0, n)
    ctf, otf = points
    cols = [np.interp(x, [p[0] for p in ctf], [p[1][c] for p in ctf]) for c in range(3)]
    cols.append(np.interp(x, [p[0] for p in otf], [p[1] for p in otf]))
    return torch.from_numpy(np.stack(cols, 1).astype(np.float32)).to(_device())


def _normals64(data):
    g = torch.stack(torch.gradient(data.double()), -1)
    return g / (g.norm(dim=-1, keepdim=True) + 1e-8)


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        vol, normals, lut, target, orbits = _train_scene(case, seed)
        m = _March64(vol, 1.0, normals, lut, orbits, case["width"], case["height"], "balanced")
        image, _ = m.walk(None)
        g = 2.0 * (image - target.reshape(-1, 4).double()) / target.numel()
        return [image.view(target.shape)] + m.gradients(image, g, case["voxels"])
    if kind == "frame" and case["floats"] or kind == "device" and case["normals"] == "none":
        data, orbit, points = _single(case, seed)
        normals = None if kind == "device" else _normals64(data)
        m = _March64(data, _scale(case["storage"]), normals, _table(points), [orbit], case["width"], case["height"],
                     case["preset"])
        image = m.walk(None)[0]
        return [None, image.view(case["height"], case["width"], 4) if kind == "frame" else image.view(-1)]
    if kind == "load" and case["read_normals"]:
        return [None, _normals64(_single(case, seed)[0])]
    return None  # RGBA8 images


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------

# operations of one sample: position and texel coordinates (30), trilinear
# filters (7 lerps of 3 per channel), table lerp (12), opacity, shading and
# compositing (30)
SAMPLE_FLOPS = {False: 30 + 21 + 12 + 30, True: 30 + 84 + 12 + 30}
ITEM = {"u8": 1, "f16": 2, "f32": 4}


def _count(data, scale, points, orbits, width, height, preset):
    """In-box samples of a frame, from a march at an eighth of its size."""
    lut = points if isinstance(points, torch.Tensor) else _table(points)
    w, h = max(8, width // 8), max(8, height // 8)
    m = _March64(data, scale, None, lut, orbits, w, h, preset)
    return m.walk(None)[1] * (width * height) / (w * h)


def work(case):
    kind = case["kind"]
    if kind == "train":
        vol, normals, lut, target, orbits = _train_scene(case, 1)
        samples = _count(vol, 1.0, lut, orbits, case["width"], case["height"], "balanced")
        px = case["views"] * case["width"] * case["height"]
        # image written and read, target and gradient read; volume, normals and
        # table read by either direction, gradients written
        nbytes = px * 16 * 4 + vol.numel() * (4 + (12 if case["normals"] else 0)) * 2 + lut.numel() * 12
        per = SAMPLE_FLOPS[case["normals"]]
        # the backward needs the sample again, the reverse recurrences and two
        # table entries (60), and eight voxel contributions (24)
        flops = samples * (2 * per + 60 + (24 if case["voxels"] else 0))
        return dict(bytes=nbytes + (vol.numel() * 4 if case["voxels"] else 0), flops=flops)
    if kind == "batch":
        nbytes = flops = 0.0
        for s in _batch_scenes(case, 1):
            data = _stored(_noise(s["dims"], np.random.default_rng(s["noise"])), s["storage"])
            flops += SAMPLE_FLOPS[True] * _count(data, _scale(s["storage"]), s["points"], [s["orbit"]], s["res"],
                                                 s["res"], "balanced")
            nbytes += data.numel() * ITEM[s["storage"]] + s["res"] ** 2 * 4
        return dict(bytes=nbytes, flops=flops)
    if kind == "serve":
        vols, reqs = _serve_scene(case, 1)
        data = [_stored(_noise((n,) * 3, np.random.default_rng(noise)), st) for n, st, noise in vols]
        nbytes = sum(float(x.numel() * x.element_size()) for x in data)
        flops = 0.0
        for v, orbit, points, side, preset in reqs:
            flops += SAMPLE_FLOPS[True] * _count(data[v], _scale(vols[v][1]), points, [orbit], side, side, preset)
            nbytes += side * side * 4
        return dict(bytes=nbytes, flops=flops)
    data, orbit, points = _single(case, 1)
    normals = case.get("normals") != "none"
    samples = _count(data, _scale(case["storage"]), points, [orbit], case["width"], case["height"], case["preset"])
    nbytes = data.numel() * ITEM[case["storage"]] + case["width"] * case["height"] * 4
    flops = samples * SAMPLE_FLOPS[normals]
    if kind in ("frame", "device") and (case.get("floats") or case.get("normals") == "none"):
        nbytes += case["width"] * case["height"] * 16
    if kind in ("load", "reload"):
        # differences, norm and quotients of every voxel; the layout written once
        flops += data.numel() * 16
        nbytes += data.numel() * (8 if case.get("records") == "half_normals" else 16)
        if case.get("read_normals"):
            nbytes += data.numel() * 12
    return dict(bytes=float(nbytes), flops=float(flops))
