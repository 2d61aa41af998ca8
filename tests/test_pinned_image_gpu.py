"""pvr_render_pinned: the handle's page-locked image, one per handle,
overwritten by the next call."""

import ctypes

import numpy as np
import pytest

from pyvr_gb300 import Camera, VolumeRenderer, _native
from pyvr_gb300 import workloads as W

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_pinned_image():
    c = W.config_small()
    w, h = 61, 44
    lib = _native.load()

    def pinned(r):
        p = ctypes.c_void_p()
        _native.check(lib.pvr_render_pinned(r._h, ctypes.byref(p)))
        return p.value, ctypes.string_at(p.value, w * h * 4)

    with VolumeRenderer(w, h, config=c["config"], light=c["light"]) as r:
        r.load_volume(c["volume"])
        r.set_transfer_functions(c["ctf"], c["otf"])
        images, addresses = [], set()
        for azimuth in (0.3, 2.1):
            r.set_camera(Camera.from_spherical(np.zeros(3, np.float32), azimuth, 0.4, 0.0, 3.0))
            p, image = pinned(r)
            assert image == r.render() and any(image)
            images.append(image)
            addresses.add(p)
        assert len(addresses) == 1 and images[0] != images[1]
        # the handle keeps no image of render()'s: the pinned one is the last pinned render
        assert ctypes.string_at(addresses.pop(), w * h * 4) == images[1]
