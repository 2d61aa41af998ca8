"""Uploads in slabs (32 MB and more) of every kind of source and record: uint8
normals and quads over many bricks along x, page-locked and ordinary arrays.
Normals read back equal numpy's; frames equal the oracle's bit for bit."""

import numpy as np
import pytest

import oracle
from pyvr_gb300 import RenderConfig, Volume, compute_normal_volume
from pyvr_gb300 import workloads as W

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dims,dtype,normals,brick,locked", [
    ((331, 331, 331), "u8", "device", 3, True), ((330, 330, 330), "u8", "device", 4, False),
    ((101, 300, 1200), "u8", "none", 2, False), ((65, 210, 1301), "f16", "none", 4, True),
    ((211, 211, 211), "f32", "device", 3, False)])
def test_slabs(dims, dtype, normals, brick, locked):
    from pyvr_gb300.batch import (BatchRenderer, DeviceLUT, DeviceVolume, RenderJob, arithmetic,
                                  get_compact_records, page_locked_copy, set_compact_records)
    from pyvr_gb300.renderer import rgba_lut
    a = np.random.default_rng(11).random(dims, dtype=np.float32)
    a[a < 0.3] = 0.0
    data = W.to_storage(a, dtype)
    assert data.nbytes >= 32 << 20
    vs = 1.0 / 255.0 if dtype == "u8" else 1.0
    with np.errstate(all="ignore"):
        nrm = compute_normal_volume(data) if normals == "device" else None
    vol = Volume(data=page_locked_copy(data) if locked else data, min_bounds=np.full(3, -1.0, np.float32),
                 max_bounds=np.full(3, 1.0, np.float32))
    prev = get_compact_records()
    set_compact_records("half_normals")
    try:
        dv = DeviceVolume(vol, value_scale=vs, normals=normals, brick_log2=brick, wait=False)
    finally:
        set_compact_records(prev)
    cam, light, cfg = W.config_small()["camera"], W.config_small()["light"], RenderConfig.fast()
    ctf, otf = W.standin_colormap(2), W.random_opacity(np.random.default_rng(5), 6, 0.1)
    w, h = 61, 52
    outf = torch.empty(w * h * 4, dtype=torch.float32, device="cuda")
    br = BatchRenderer(capacity=1, slots=1)
    with arithmetic("exact"):
        br.render([RenderJob(dv, DeviceLUT(ctf, otf), cam, light, cfg, w, h, None, outf)])
        br.synchronize()
    br.close()
    if nrm is not None:
        want = nrm.astype(np.float32)
        if dtype != "f32":
            want = want.astype(np.float16).astype(np.float32)
        assert np.array_equal(dv.read_normals(), want, equal_nan=True)
        vol.normals = want
    dv.close()
    _, of, _ = oracle.render(W.frame_inputs(vol, cam, light, cfg, rgba_lut(ctf, otf), w, h, vs, batch_camera=True))
    got = outf.cpu().numpy().reshape(h, w, 4)
    assert np.array_equal(got.view(np.uint32), of.view(np.uint32)) and of.any()
