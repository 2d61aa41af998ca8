"""The differentiable march from the scene's own arrays (no workspace) against
the packed one: images and loop lengths equal bit for bit; gradients up to the
order of their float sums."""

import ctypes

import numpy as np
import pytest

from pyvr_gb300 import Camera, Light, RenderConfig, _native
from pyvr_gb300.diff import DiffScene

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# thin and odd volumes; few voxels under many rays, whose gradients are summed
# per warp; tables on both sides of the per-warp gradient table's limit
@pytest.mark.parametrize("dims,size,lut_size", [
    ((1, 1, 1), (40, 33), 1), ((2, 17, 3), (61, 47), 512), ((1, 5, 8), (33, 70), 513),
    ((13, 2, 1), (17, 16), 2048), ((33, 16, 31), (96, 65), 256), ((5, 5, 5), (128, 128), 64)])
@pytest.mark.parametrize("normals", [True, False])
def test_arrays_equal_packed_texels(dims, size, lut_size, normals):
    lib, rng = _native.load(), np.random.default_rng(lut_size)
    w, h = size
    vol = torch.tensor(rng.random(dims, dtype=np.float32) * 1.2 - 0.1, device="cuda")
    nrm = torch.tensor(rng.normal(size=dims + (3,)).astype(np.float32), device="cuda") if normals else None
    lut = np.concatenate([rng.random((lut_size, 3)), rng.uniform(0.0, 0.2, (lut_size, 1))], 1).astype(np.float32)
    lut = torch.tensor(lut, device="cuda")
    cams = [Camera.from_spherical(np.zeros(3, np.float32), a, 0.4, 0.0, 3.0) for a in (0.3, 2.1)]
    scene = DiffScene(cams, Light.directional([1, -1, 0], 0.2, 0.8), RenderConfig.fast(), w, h)
    c = scene.c_scene(vol, lut, nrm)
    stream = torch.cuda.current_stream().cuda_stream
    bytes_, bytes_volume = ctypes.c_longlong(), ctypes.c_longlong()
    _native.check(lib.pvr_diff_workspace(ctypes.byref(c), ctypes.byref(bytes_), ctypes.byref(bytes_volume)))
    assert bytes_.value > 0
    ws = torch.empty(bytes_volume.value, dtype=torch.uint8, device="cuda")
    grad = torch.tensor(rng.random((2, h, w, 4), dtype=np.float32), device="cuda")
    out = []
    for p, n in ((None, 0), (ws.data_ptr(), bytes_volume.value)):
        image = torch.empty((2, h, w, 4), device="cuda")
        steps = torch.empty((2, h, w), dtype=torch.int32, device="cuda")
        _native.check(lib.pvr_diff_forward_ws(ctypes.byref(c), image.data_ptr(), steps.data_ptr(), p, n, stream))
        # gradients are added: to 1 here
        glut, gvol = torch.ones_like(lut), torch.ones_like(vol)
        _native.check(lib.pvr_diff_backward_ws(ctypes.byref(c), image.data_ptr(), steps.data_ptr(), grad.data_ptr(),
                                               glut.data_ptr(), gvol.data_ptr(), 0, p, n, stream))
        one = torch.full_like(lut, 7.0)  # the LUT gradient alone, written
        _native.check(lib.pvr_diff_backward_ws(ctypes.byref(c), image.data_ptr(), steps.data_ptr(), grad.data_ptr(),
                                               one.data_ptr(), None, 1, p, n, stream))
        out.append((image, steps, glut - 1, gvol - 1, one))
    a, b = out
    assert torch.equal(a[0].view(torch.int32), b[0].view(torch.int32)) and torch.equal(a[1], b[1])
    assert bool(a[1].any())
    # up to 2 x 100 samples of 128^2 rays fall on one entry: 3e6 roundings of
    # 2^-24 in random order leave 1e-4 of the sum
    for x, y in zip(a[2:], b[2:]):
        assert float((x - y).norm()) <= 1e-3 * float(y.norm()) + 1e-5
