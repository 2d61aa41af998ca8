"""The brick layout at its edges: every storage type, record form and brick
size over extents around the brick size, cubic and not, with normals from the
device, given and none.  Normals read back equal numpy's (rounded to half in
half records, where they are not halves already); frames equal the oracle's
bit for bit, which covers values, slots and clamped aprons."""

import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle
from pyvr_gb300 import RenderConfig, Volume, compute_normal_volume
from pyvr_gb300 import workloads as W

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pyvr_gb300", "csrc")


def _data(dims, dtype, seed):
    rng = np.random.default_rng(seed)
    a = rng.random(dims, dtype=np.float32)
    a[a < 0.3] = 0.0  # flat places: zero gradients
    if dtype == "u8":
        return np.rint(a * 255).astype(np.uint8)
    return a.astype(np.float16 if dtype == "f16" else np.float32)


@pytest.mark.parametrize("brick", [2, 3, 4])
@pytest.mark.parametrize("dtype", ["u8", "f16", "f32"])
@pytest.mark.parametrize("records", ["float", "half_normals"])
def test_layout_edges(brick, dtype, records):
    from pyvr_gb300.batch import (BatchRenderer, DeviceLUT, DeviceVolume, RenderJob, arithmetic,
                                  get_compact_records, set_compact_records)
    from pyvr_gb300.renderer import rgba_lut
    b = 1 << brick
    cam, light = W.config_small()["camera"], W.config_small()["light"]
    ctf, otf = W.standin_colormap(2), W.random_opacity(np.random.default_rng(5), 6, 0.3)
    lut, dl = rgba_lut(ctf, otf), DeviceLUT(ctf, otf)
    cfg = RenderConfig.fast()
    w, h = 45, 38
    br = BatchRenderer(capacity=1, slots=1)
    prev = get_compact_records()
    set_compact_records(records)
    try:
        cases = [((n, n, n), "device") for n in (2, b - 1, b, b + 1, 2 * b, 3 * b + 2)]
        cases += [((b, 2 * b + 1, 3), "device"), ((b + 2, 3, 2 * b), "given"), ((2 * b,) * 3, "none"),
                  ((1, b + 1, 2 * b - 1), "none")]
        for k, (dims, mode) in enumerate(cases):
            data = _data(dims, dtype, 31 * k + brick)
            with np.errstate(all="ignore"):
                nrm = compute_normal_volume(data) if mode != "none" else None
            vol = Volume(data=data, normals=nrm, min_bounds=np.full(3, -1.0, np.float32),
                         max_bounds=np.full(3, 1.0, np.float32))
            vs = 1.0 / 255.0 if dtype == "u8" else 1.0
            dv = DeviceVolume(vol, value_scale=vs, normals=mode, brick_log2=brick)
            half = records == "half_normals" and dtype != "f32"
            if nrm is not None:
                want = nrm.astype(np.float32)
                if half:
                    want = want.astype(np.float16).astype(np.float32)
                assert np.array_equal(dv.read_normals(), want, equal_nan=True), (dims, mode)
                vol.normals = want
            out8 = torch.empty(w * h * 4, dtype=torch.uint8, device="cuda")
            outf = torch.empty(w * h * 4, dtype=torch.float32, device="cuda")
            with arithmetic("exact"):
                br.render([RenderJob(dv, dl, cam, light, cfg, w, h, out8, outf)])
                br.synchronize()
            o8, of, _ = oracle.render(W.frame_inputs(vol, cam, light, cfg, lut, w, h, vs, batch_camera=True))
            finite = np.isfinite(of).all(axis=2)
            got = outf.cpu().numpy().reshape(h, w, 4)
            assert np.array_equal(got[finite].view(np.uint32), of[finite].view(np.uint32)), (dims, mode)
            assert np.array_equal(np.isfinite(got).all(axis=2), finite), (dims, mode)
            assert np.array_equal(out8.cpu().numpy().reshape(h, w, 4)[finite], o8[finite]), (dims, mode)
            dv.close()
    finally:
        set_compact_records(prev)
        br.close()


def test_half_normals_exhaustive(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "half_normals_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-std=c++17",
                    f"-I{CSRC}", os.path.join(HERE, "cuda", "half_normals_check.cu"), "-o", exe],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout.split()
    triples, u8_bad, undecided, pairs, f16_bad = (int(x) for x in out)
    assert triples == 767 ** 3 and pairs == 0x7bff * (0x10000 - 0x800)
    assert u8_bad == 0, f"{u8_bad} of {triples} uint8 components differ"
    assert undecided < 0.01 * triples, undecided
    assert f16_bad == 0, f"{f16_bad} of {pairs} float16 quotients differ"


@pytest.mark.parametrize("dims,dtype,normals,brick", [((257,) * 3, "f16", "device", 3), ((262,) * 3, "f16", "device", 4),
                                                      ((300, 41, 700), "f32", "none", 3), ((3000, 4000, 3), "u8", "none", 4)])
def test_upload_in_slabs(dims, dtype, normals, brick):
    # 32 MB and more arrive in slabs, each laid out while the next is copied:
    # normals and frames as for a volume that arrived whole
    from pyvr_gb300.batch import (BatchRenderer, DeviceLUT, DeviceVolume, RenderJob, arithmetic,
                                  get_compact_records, page_locked_copy, set_compact_records)
    from pyvr_gb300.renderer import rgba_lut
    data = page_locked_copy(_data(dims, dtype, 77))
    with np.errstate(all="ignore"):
        nrm = compute_normal_volume(data) if normals == "device" else None
    vol = Volume(data=data, min_bounds=np.full(3, -1.0, np.float32), max_bounds=np.full(3, 1.0, np.float32))
    prev = get_compact_records()
    set_compact_records("half_normals")
    try:
        dv = DeviceVolume(vol, normals=normals, brick_log2=brick, wait=False)
    finally:
        set_compact_records(prev)
    cam, light, cfg = W.config_small()["camera"], W.config_small()["light"], RenderConfig.fast()
    ctf, otf = W.standin_colormap(2), W.random_opacity(np.random.default_rng(5), 6, 0.3)
    w, h = 61, 52
    outf = torch.empty(w * h * 4, dtype=torch.float32, device="cuda")
    br = BatchRenderer(capacity=1, slots=1)
    with arithmetic("exact"):
        br.render([RenderJob(dv, DeviceLUT(ctf, otf), cam, light, cfg, w, h, None, outf)])
        br.synchronize()
    if nrm is not None:
        assert np.array_equal(dv.read_normals(), nrm.astype(np.float32), equal_nan=True)
        vol.normals = nrm.astype(np.float32)
    _, of, _ = oracle.render(W.frame_inputs(vol, cam, light, cfg, rgba_lut(ctf, otf), w, h, 1.0, batch_camera=True))
    got = outf.cpu().numpy().reshape(h, w, 4)
    finite = np.isfinite(of).all(axis=2)
    assert np.array_equal(got[finite].view(np.uint32), of[finite].view(np.uint32))
    assert np.array_equal(np.isfinite(got).all(axis=2), finite)
    br.close()
    dv.close()
