"""What a launch tuning says and does: the one a launcher reports is the one it
runs."""

import ctypes

import pytest

from pyvr_gb300 import _native

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_reported_default_is_what_runs():
    # as many persistent blocks as fit, which is blocks_per_sm 0: setting the
    # reported tuning again changes nothing
    from pyvr_gb300.batch import BatchRenderer, Tuning
    br = BatchRenderer(capacity=1, slots=1)
    t = _native.PvrTuning()
    _native.check(_native.load().pvr_batch_get_tuning(br.handle, ctypes.byref(t)))
    br.close()
    default = Tuning()
    assert (t.tile_w, t.tile_h, t.steps_per_iter, t.blocks_per_sm) == (
        default.tile_w, default.tile_h, default.steps_per_iter, default.blocks_per_sm) == (16, 16, 1, 0)


def test_tiles_and_steps_of_the_caller_keep_one_lane_per_ray():
    import numpy as np

    from pyvr_gb300 import Camera, Light, RenderConfig, Volume
    from pyvr_gb300.batch import BatchRenderer, DeviceLUT, DeviceVolume, RenderJob, Tuning, make_job_struct
    lanes = getattr(_native.load(), "_ZN3pvr12render_lanesEPK9pvr_batchRK7pvr_job")
    lanes.argtypes, lanes.restype = [ctypes.c_void_p, ctypes.c_void_p], ctypes.c_int
    dv = DeviceVolume(Volume(data=np.ones((9, 9, 9), np.float32)), normals="none")
    lut = DeviceLUT(rgba=np.full((4, 4), 0.1, np.float32))
    cam = Camera.from_spherical(np.zeros(3, np.float32), 0.7, 0.3, 0.0, 3.0)
    job = make_job_struct(RenderJob(dv, lut, cam, Light.directional([1, -1, 0], 0.2, 0.8), RenderConfig.fast(), 64, 48))
    br = BatchRenderer(capacity=1, slots=1)
    assert lanes(br.handle, ctypes.byref(job)) == 4
    # blocks per SM are a batch's
    for t, want in ((Tuning(), 4), (Tuning(8, 32, 1, 0), 1), (Tuning(16, 16, 4, 0), 1), (Tuning(64, 4, 1, 0), 1),
                    (Tuning(16, 16, 1, 5), 4), (Tuning(), 4)):
        br.set_tuning(t)
        assert lanes(br.handle, ctypes.byref(job)) == want, t
    br.close()
    dv.close()
