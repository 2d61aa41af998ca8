"""Small single renders with 2 or 4 lanes per ray: images, float images and
sample counts equal the oracle's (exact arithmetic, bit for bit) and those of
the persistent batch kernel, which marches one lane per ray (both
arithmetics)."""

import numpy as np
import pytest

import oracle
from pyvr_gb300 import Camera, Light, RenderConfig, Volume
from pyvr_gb300 import workloads as W

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# 4 lanes up to about 197^2 (220^2 with half records) pixels on 152 SMs, 2 up to
# 279^2 (312^2)
SIZES = [(1, 1), (9, 5), (61, 37), (192, 200), (224, 224), (301, 233)]


def _render(dv, lut, cam, cfg, w, h, alone):
    from pyvr_gb300.batch import BatchRenderer, RenderJob
    o8 = [torch.zeros(w * h * 4, dtype=torch.uint8, device="cuda") for _ in range(2)]
    of = [torch.zeros(w * h * 4, dtype=torch.float32, device="cuda") for _ in range(2)]
    n = torch.zeros((2, 2), dtype=torch.int64, device="cuda")
    jobs = [RenderJob(dv, lut, cam, Light.directional([1, -1, 0], 0.2, 0.8), cfg, w, h, o8[k], of[k], n[k])
            for k in range(1 if alone else 2)]
    br = BatchRenderer(capacity=2, slots=1)
    torch.cuda.synchronize()
    br.render(jobs)
    br.synchronize()
    br.close()
    return o8[0].cpu().numpy(), of[0].cpu().numpy(), n[0].tolist()


@pytest.mark.parametrize("normals", ["device", "none"])
@pytest.mark.parametrize("records,dtype", [("float", "f32"), ("half_normals", "u8")])
@pytest.mark.parametrize("lut_size", [256, 4096])
def test_split_march(normals, records, dtype, lut_size):
    from pyvr_gb300.batch import DeviceLUT, DeviceVolume, arithmetic, get_compact_records, set_compact_records
    from pyvr_gb300.renderer import rgba_lut
    noise = W.value_noise((24, 24, 24), 4)
    noise[noise < 0.4] = 0.0  # clear bricks and flat places
    data = W.to_storage(noise, dtype)
    vol = Volume(data=data, min_bounds=np.full(3, -1.0, np.float32), max_bounds=np.full(3, 1.0, np.float32))
    vs = 1.0 / 255.0 if dtype == "u8" else 1.0
    prev = get_compact_records()
    set_compact_records(records)
    try:
        dv = DeviceVolume(vol, value_scale=vs, normals=normals, brick_log2=2)
    finally:
        set_compact_records(prev)
    if normals == "device":
        vol.normals = dv.read_normals()
    from pyvr_gb300 import OpacityTransferFunction
    otf = OpacityTransferFunction([(0.0, 0.0), (0.1, 0.0), (0.5, 0.3), (1.0, 0.9)])
    ctf = W.standin_colormap(5)
    lut, table = DeviceLUT(ctf, otf, lut_size), rgba_lut(ctf, otf, lut_size)
    outside = Camera.from_spherical(np.zeros(3, np.float32), 0.7, 0.3, 0.0, 3.0)
    inside = Camera.from_spherical(np.zeros(3, np.float32), 2.0, -0.2, 0.0, 0.4)
    configs = [(RenderConfig.balanced(), s) for s in SIZES]
    # step limits inside a group of samples, and steps so long that a ray has few samples
    configs += [(RenderConfig.custom(0.02, m), (31, 17)) for m in (1, 2, 3, 4, 5, 7)]
    configs += [(RenderConfig.custom(0.7, 9), (31, 17))]
    for cfg, (w, h) in configs:
        for cam in (outside, inside):
            for mode in ("exact", "fast"):
                with arithmetic(mode):
                    a8, af, an = _render(dv, lut, cam, cfg, w, h, True)
                    b8, bf, bn = _render(dv, lut, cam, cfg, w, h, False)
                assert np.array_equal(a8, b8) and np.array_equal(af.view(np.uint32), bf.view(np.uint32)), (w, h, mode)
                assert an == bn, (w, h, mode)
                if mode == "exact" and w <= 61:
                    s = W.frame_inputs(vol, cam, Light.directional([1, -1, 0], 0.2, 0.8), cfg, table, w, h, vs,
                                       batch_camera=True)
                    o8, of, on = oracle.render(s)
                    assert np.array_equal(a8.reshape(o8.shape), o8) and an[0] == on
                    assert np.array_equal(af.reshape(of.shape).view(np.uint32), of.view(np.uint32))
    dv.close()


# half a tile per block for half records, with tables that are staged (to 512
# entries), staged with whole tiles (to 2048) and read from global memory
@pytest.mark.parametrize("lut_size", [1, 512, 513, 2048, 2049])
@pytest.mark.parametrize("tile_w,tile_h", [(16, 16), (64, 4), (8, 32)])
def test_half_tiles(lut_size, tile_w, tile_h):
    from pyvr_gb300 import OpacityTransferFunction
    from pyvr_gb300.batch import (BatchRenderer, DeviceLUT, DeviceVolume, RenderJob, Tuning, arithmetic,
                                  get_compact_records, set_compact_records)
    vol = Volume(data=W.to_storage(W.value_noise((40, 40, 40), 6), "u8"), min_bounds=np.full(3, -1.0, np.float32),
                 max_bounds=np.full(3, 1.0, np.float32))
    prev = get_compact_records()
    set_compact_records("half_normals")
    try:
        dv = DeviceVolume(vol, value_scale=1.0 / 255.0, normals="device", brick_log2=3)
    finally:
        set_compact_records(prev)
    rgba = np.random.default_rng(lut_size).random((lut_size, 4)).astype(np.float32) * np.float32(0.4)
    lut = DeviceLUT(rgba=rgba)
    cam, light = Camera.from_spherical(np.zeros(3, np.float32), 0.7, 0.3, 0.0, 3.0), Light.directional([1, -1, 0], 0.2, 0.8)
    for w, h in ((417, 331), (1029, 129)):  # more pixels than several lanes per ray take
        for mode in ("exact", "fast"):
            out = []
            for n in (1, 2):  # alone, and as a job of the batch kernel
                o8 = [torch.zeros(w * h * 4, dtype=torch.uint8, device="cuda") for _ in range(n)]
                of = [torch.zeros(w * h * 4, dtype=torch.float32, device="cuda") for _ in range(n)]
                c = torch.zeros((n, 2), dtype=torch.int64, device="cuda")
                br = BatchRenderer(capacity=2, slots=1, tuning=Tuning(tile_w=tile_w, tile_h=tile_h, brick_log2=3))
                torch.cuda.synchronize()
                with arithmetic(mode):
                    br.render([RenderJob(dv, lut, cam, light, RenderConfig.fast(), w, h, o8[k], of[k], c[k])
                               for k in range(n)])
                br.synchronize()
                br.close()
                out.append((o8[0].cpu().numpy(), of[0].cpu().numpy().view(np.uint32), c[0].tolist()))
            assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1]), (w, h, mode)
            assert out[0][2] == out[1][2] and out[0][2][1] > 0, (w, h, mode)
    dv.close()
