"""The differentiable march called from several threads at once: the C entry
points take no handle, so calls with different table sizes may overlap."""

import ctypes
import threading

import numpy as np
import pytest

from pyvr_gb300 import Camera, Light, RenderConfig, _native
from pyvr_gb300.diff import DiffScene

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _scene():
    cam = Camera.from_spherical(np.zeros(3, np.float32), 0.3, 0.4, 0.0, 3.0)
    return DiffScene([cam], Light.directional([1, -1, 0], 0.2, 0.8), RenderConfig.fast(), 16, 16)


# two per-warp tables of more than 48 KB, and two per-block ones
@pytest.mark.parametrize("sizes", [(512, 400), (2048, 1600)])
def test_backward_calls_of_different_table_sizes(sizes):
    lib, scene, errors = _native.load(), _scene(), []

    def work(n):
        torch.cuda.set_device(0)
        vol, lut = torch.rand(8, 8, 8, device="cuda"), torch.rand(n, 4, device="cuda") * 0.1
        image = torch.empty((1, 16, 16, 4), device="cuda")
        steps = torch.empty((1, 16, 16), dtype=torch.int32, device="cuda")
        g, glut = torch.ones_like(image), torch.zeros_like(lut)
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()
        c = scene.c_scene(vol, lut)
        rc = lib.pvr_diff_forward(ctypes.byref(c), image.data_ptr(), steps.data_ptr(), stream.cuda_stream)
        for k in range(4000):
            if rc:
                errors.append((n, lib.pvr_last_error()))
                break
            rc = lib.pvr_diff_backward(ctypes.byref(c), image.data_ptr(), steps.data_ptr(), g.data_ptr(),
                                       glut.data_ptr(), None, stream.cuda_stream)
            if k % 64 == 0:
                stream.synchronize()
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(n,)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


def test_backward_leaves_the_saved_scene_alone():
    # saved-tensor hooks give every backward tensors of its own; their
    # addresses must not reach another backward of the same graph
    from pyvr_gb300.diff import render_views
    vol = torch.rand(8, 8, 8, device="cuda").requires_grad_()
    lut = (torch.rand(64, 4, device="cuda") * 0.1).requires_grad_()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.clone(), lambda t: t.clone()):
        image = render_views(vol, lut, _scene())
    saved = bytes(image.grad_fn.c)
    image.backward(torch.ones_like(image), retain_graph=True)
    first = lut.grad.clone(), vol.grad.clone()
    assert bytes(image.grad_fn.c) == saved
    image.backward(torch.ones_like(image))
    # up to the order of the float sums
    for got, one in ((lut.grad, first[0]), (vol.grad, first[1])):
        assert float((got - 2 * one).abs().max()) <= 1e-4 * float(one.abs().max())
